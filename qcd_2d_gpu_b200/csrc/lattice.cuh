// Checkerboard geometry and the SoA link store in HBM.
//
// Sites are split by parity p = (t + x + y) mod 2 into two sublattices of
// Vh = V/2 sites.  A sublattice index is id = y' + Lyh*(x + Lx*t) with
// Lyh = Ly/2 (the reference's half-lattice index, mc_updates.h:130-134);
// the physical y of the site is 2y' + q with q = ((t + x) mod 2) xor p.
// Stream id of the random-number generator is this id for both parities
// (lattice_setup.h:15-21; even and odd kernels share state + id).
//
// Link store: one plane per (direction mu, parity p), plane index mu*2 + p,
// mu = 0 (y), 1 (x), 2 (t); inside a plane the links are contiguous in id.
//   FP64: one plane of 32-byte records (w, x, y, z) -> one 256-bit load per link.
//   FP32: one float4 plane -> one 16-B load per link.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "su2.cuh"

namespace qcd {

enum { DIR_Y = 0, DIR_X = 1, DIR_T = 2 };
enum { BC_PER = 0, BC_PCC = 1, BC_PMC = 2 };

struct Geo {
  int lt, lx, ly;  // physical extents (all even)
  int lyh;         // Ly / 2
  int slice;       // Lyh * Lx : sublattice sites per t-slice
  int vh;          // Lyh * Lx * Lt
  // s / lyh for 0 <= s < slice as (s * lyh_magic) >> 32, lyh_magic = ceil(2^32 / lyh):
  // exact when lyh^2 * lx < 2^32 (fastdiv = 1), otherwise a hardware division is used
  unsigned long long lyh_magic;
  int fastdiv;
  // n / slice for any 32-bit n as the high word of n * slice_m (0: slice = 1)
  unsigned long long slice_m;
};

// m = ceil(2^64 / d) for 2 <= d < 2^32 (0 for d = 1): floor(n * m / 2^64) =
// floor(n / d) for every n < 2^32, because m * d - 2^64 < d
__host__ __forceinline__ unsigned long long div_magic(unsigned long long d) { return ~0ull / d + 1; }
__device__ __forceinline__ int div_by(unsigned int n, unsigned long long m) {
  return m ? (int)__umul64hi((unsigned long long)n, m) : (int)n;
}

__host__ __forceinline__ Geo make_geo(int lt, int lx, int ly) {
  Geo g;
  g.lt = lt;
  g.lx = lx;
  g.ly = ly;
  g.lyh = ly / 2;
  g.slice = g.lyh * lx;
  g.vh = g.slice * lt;
  g.lyh_magic = ((1ull << 32) + (unsigned long long)g.lyh - 1) / (unsigned long long)g.lyh;
  g.fastdiv = (unsigned long long)g.lyh * (unsigned long long)g.lyh * (unsigned long long)lx < (1ull << 32);
  g.slice_m = div_magic((unsigned long long)g.slice);
  return g;
}

// Decoded sublattice site plus the offsets (in sublattice index units) of its
// six neighbours, which all lie on the other sublattice.  Offsets add: the
// site x + mu - nu is id + off_plus(mu) + off_minus(nu) on the same
// sublattice, because moving in x or t does not change q and moving in y does
// not change x or t.
struct Nbr {
  int id, yq, x, t, q;
  int yp, ym, xp, xm, tp, tm;
};

__device__ __forceinline__ void finish_nbr(const Geo& g, int parity, Nbr& n);

// From the sublattice index (two divisions).
__device__ __forceinline__ Nbr make_nbr(const Geo& g, int id, int parity) {
  Nbr n;
  n.id = id;
  n.yq = id % g.lyh;
  int r = id / g.lyh;
  n.x = r % g.lx;
  n.t = r / g.lx;
  finish_nbr(g, parity, n);
  return n;
}

// From the position s inside t-slice t (launch grid (slice, Lt)): one
// multiply-high instead of two divisions.
__device__ __forceinline__ Nbr make_nbr_slice(const Geo& g, int s, int t, int parity) {
  Nbr n;
  n.t = t;
  n.x = g.fastdiv ? (int)(((unsigned long long)(unsigned)s * g.lyh_magic) >> 32) : s / g.lyh;
  n.yq = s - n.x * g.lyh;
  n.id = s + t * g.slice;
  finish_nbr(g, parity, n);
  return n;
}

// From the sublattice index: the t-slice by a multiply-high, the rest as in
// make_nbr_slice; the same offsets as make_nbr.
__device__ __forceinline__ Nbr make_nbr_fast(const Geo& g, int id, int parity) {
  const int t = div_by((unsigned int)id, g.slice_m);
  return make_nbr_slice(g, id - t * g.slice, t, parity);
}

__device__ __forceinline__ void finish_nbr(const Geo& g, int parity, Nbr& n) {
  n.q = ((n.t + n.x) & 1) ^ parity;
  // +y: a site with odd physical y moves to the next y' (wrapping), an even
  // one stays at the same y' (mc_updates.h:139-141, 195-197)
  n.yp = n.q ? (n.yq == g.lyh - 1 ? -(g.lyh - 1) : 1) : 0;
  // -y: the mirror image (mc_updates.h:252-254, 309-311)
  n.ym = n.q ? 0 : (n.yq == 0 ? g.lyh - 1 : -1);
  n.xp = n.x == g.lx - 1 ? -(g.lx - 1) * g.lyh : g.lyh;
  n.xm = n.x == 0 ? (g.lx - 1) * g.lyh : -g.lyh;
  n.tp = n.t == g.lt - 1 ? -(g.lt - 1) * g.slice : g.slice;
  n.tm = n.t == 0 ? (g.lt - 1) * g.slice : -g.slice;
}

// ------------------------------------------------- sites of a phase launch --
// A phase launch gives each CTA a tile of 2 t-slices x 2 x-rows x 32 y', a warp
// per row, with the x-row pairs of a slice pair laid end to end (so a short or
// ragged row leaves no lane idle but in the last CTA of a slice pair).  A link is
// read for the staples of sites on both sides of it in the two directions
// across it: a tile two wide in x and in t finds half of those reads in L1, a run
// of 256 sites of one slice hardly any.  384^3 site pairs: over-relaxation phase
// 504 -> 488 us, heat-bath 610 -> 590 us; tiles 4 wide, or of 64 or 256
// threads, gain less.
//
// Launches on the odd sites (each follows one on the even sites) walk the
// slices from the last to the first, so a launch begins with the links its
// predecessor touched last, while they are in L2: 128^3 (100 MB of FP32 links)
// over-relaxation 19.1 -> 17.5 us, 192^3 62 -> 59 us, 384^3 1%.
constexpr int kTileY = 32, kTileThreads = 4 * kTileY;

__host__ __forceinline__ dim3 tile_grid(const Geo& g) {  // Lt and Lx are even
  return dim3((unsigned int)((g.lyh * (g.lx / 2) + kTileY - 1) / kTileY), (unsigned int)(g.lt / 2));
}

// Launches follow one another by programmatic dependence (launch_chained): the
// CTAs of a launch are set up while its predecessor drains, and wait here until
// the predecessor has completed and its writes are visible.  A kernel launched
// so reads and writes global memory only after chain_wait, through a value that
// went through it (an asm operand, so that no load can be moved above), and
// calls chain_ready when its CTA has little left to do.  Calling chain_ready
// just before the store is best over all sizes; as the first thing, the CTAs of
// launches to come take up slots (54x62x70 heat-bath pass 35.7 us against 29.8),
// never, the set-up is exposed again at the large sizes.  Passes without and
// with the chain: 16^3 FP64 40 -> 25 us, 24x20x28 28 -> 17, 54x62x70 39 -> 30,
// 128^3 FP32 over-relaxation 103 -> 90, heat-bath 149 -> 133.
__device__ __forceinline__ void chain_wait(unsigned int& x) {
  asm volatile("griddepcontrol.wait;" : "+r"(x)::"memory");
}
__device__ __forceinline__ void chain_wait(int& x) { asm volatile("griddepcontrol.wait;" : "+r"(x)::"memory"); }
__device__ __forceinline__ void chain_ready() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
__host__ inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int block, cudaStream_t stream,
                                           A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned int)block);
  c.stream = stream;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// The site of this thread, after the wait for the preceding launch; false
// beyond the end of the slice pair.
template <int PAR>
__device__ __forceinline__ bool tile_nbr(const Geo& g, Nbr& n) {
  const int u = blockIdx.x * kTileY + threadIdx.x % kTileY, w = threadIdx.x / kTileY;
  if (u >= g.lyh * (g.lx / 2)) return false;
  const int xp = g.fastdiv ? (int)(((unsigned long long)(unsigned)u * g.lyh_magic) >> 32) : u / g.lyh;
  n.t = 2 * (PAR ? gridDim.y - 1 - blockIdx.y : blockIdx.y) + w / 2;
  n.x = 2 * xp + w % 2;
  n.yq = u - xp * g.lyh;
  n.id = n.yq + g.lyh * n.x + g.slice * n.t;
  finish_nbr(g, PAR, n);
  chain_wait(n.id);
  return true;
}

__device__ __forceinline__ int off_plus(const Nbr& n, int dir) {
  return dir == DIR_Y ? n.yp : dir == DIR_X ? n.xp : n.tp;
}
__device__ __forceinline__ int off_minus(const Nbr& n, int dir) {
  return dir == DIR_Y ? n.ym : dir == DIR_X ? n.xm : n.tm;
}

// physical y of the site is 0 / Ly-1
__device__ __forceinline__ bool at_y0(const Geo& g, const Nbr& n) { return n.yq == 0 && n.q == 0; }
__device__ __forceinline__ bool at_ytop(const Geo& g, const Nbr& n) {
  return n.yq == g.lyh - 1 && n.q == 1;
}

__host__ __device__ __forceinline__ size_t plane_of(int dir, int parity) { return (size_t)(dir * 2 + parity); }

// Load/store policy: CG = false reads neighbour links by ordinary loads, which may
// hit in L1: no link that a phase reads so is written in that launch.  Not by the
// non-coherent path (ld.global.nc, __ldg): that one asks for data that nothing writes
// while the kernel lives, and a chained launch is alive while its predecessor still
// writes.  Ordinary loads after chain_wait see the predecessor's writes by the memory
// model; both go through L1, and the passes take the same time to 1%.
// CG = true (the wavefront kernel) reads and writes at L2 (.cg): there, other CTAs of
// the same launch rewrite links, and a line left in this SM's L1 by an earlier task
// could be stale.  The link a thread rewrites is read at L2 in either case: its sector
// may hold a link that another SM rewrites in the same launch, and the next launch's
// CTAs may already be set up on this SM.
//
// ld_float4, ld_link and ld_pair are not volatile, so they can be scheduled among other
// loads: nothing that a kernel reads through them is written by that kernel.
__device__ __forceinline__ float4 ld_float4(const float4* p) {
  float4 v;
  asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
template <class T, bool CG>
__device__ __forceinline__ void st_rw(T* p, const T& v) {
  if (CG)
    __stcg(p, v);
  else
    *p = v;
}

// ---------------------------------------------------------------- FP64 ----
// A link is one 32-byte record (w, x, y, z), read and written in one access: half
// the load instructions and addresses of two double2 planes (passes: heat-bath 128^3
// 285 -> 275 us, 256^3 2.57 -> 2.49 ms, over-relaxation 128^3 210 -> 201 us; measurement
// 256^3 306 -> 290 us).
__device__ __forceinline__ Quat<double> ld_link(const double* p) {
  Quat<double> u;
  asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(u.w), "=d"(u.x), "=d"(u.y), "=d"(u.z) : "l"(p));
  return u;
}
__device__ __forceinline__ Quat<double> ld_link_cg(const double* p) {
  Quat<double> u;
  asm volatile("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(u.w), "=d"(u.x), "=d"(u.y), "=d"(u.z)
               : "l"(p)
               : "memory");
  return u;
}
template <bool CG>
struct Links64T {
  double* q;  // six planes (plane_of(dir, parity)) of vh records
  int vh;
  __device__ __forceinline__ double* at(int dir, int parity, int id) const {
    return q + (plane_of(dir, parity) * vh + id) * 4;
  }
  __device__ __forceinline__ Quat<double> ld(int dir, int parity, int id) const {
    return CG ? ld_link_cg(at(dir, parity, id)) : ld_link(at(dir, parity, id));
  }
  // the link this thread rewrites
  __device__ __forceinline__ Quat<double> ld_own(int dir, int parity, int id) const {
    return ld_link_cg(at(dir, parity, id));
  }
  __device__ __forceinline__ void st(int dir, int parity, int id, const Quat<double>& u) const {
    if (CG)
      asm volatile("st.global.cg.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(at(dir, parity, id)), "d"(u.w), "d"(u.x),
                   "d"(u.y), "d"(u.z)
                   : "memory");
    else
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(at(dir, parity, id)), "d"(u.w), "d"(u.x),
                   "d"(u.y), "d"(u.z)
                   : "memory");
  }
};
typedef Links64T<false> Links64;

// ---------------------------------------------------------------- FP32 ----
template <bool CG>
struct Links32T {
  float4* q;
  int vh;
  __device__ __forceinline__ Quat<float> ld(int dir, int parity, int id) const {
    const float4* p = q + plane_of(dir, parity) * vh + id;
    const float4 a = CG ? __ldcg(p) : ld_float4(p);
    return Quat<float>{a.x, a.y, a.z, a.w};
  }
  __device__ __forceinline__ Quat<float> ld_own(int dir, int parity, int id) const {
    float4 a = __ldcg(q + plane_of(dir, parity) * vh + id);
    return Quat<float>{a.x, a.y, a.z, a.w};
  }
  __device__ __forceinline__ void st(int dir, int parity, int id, const Quat<float>& u) const {
    st_rw<float4, CG>(q + plane_of(dir, parity) * vh + id, make_float4(u.w, u.x, u.y, u.z));
  }
};
typedef Links32T<false> Links32;

}  // namespace qcd
