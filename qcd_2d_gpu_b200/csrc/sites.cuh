// Device building blocks shared by the single-lattice kernels (kernels.cuh)
// and the batched-replica kernels (batch.cu): the per-link update of one
// checkerboard phase and the deterministic FP64 block reductions.  Templates
// and inline functions only, so several translation units can include it.
#pragma once
#include "lattice.cuh"
#include "rng.cuh"
#include "su2.cuh"
#include "updates.cuh"

namespace qcd {

constexpr int kBlock = 256;

struct PhaseArgs {
  float beta;
  float eps;
  int upd;
  int* err;     // device error word
  int* accept;  // V ints, reference site order; only for Metropolis
  int renorm;   // FP32: re-project each updated link (in double) before it is stored
  // FP32 draws (counter-based): the key, a device word that counts drawing
  // phases (advanced on the device, so a captured graph draws fresh numbers on
  // every replay), this phase's offset from it, and the offset added to the
  // site index (a replica's stream offset in a batch)
  unsigned long long seed;
  const unsigned long long* phase_ptr;  // null: phase_off is the number itself
  long long phase_off;
  unsigned int site_off;
  PhiloxKeys keys;  // round keys of `seed` (philox_keys), set by whoever fills the arguments
  // where this launch writes the count for later launches (count_draws), or null
  unsigned long long* count_out = nullptr;
  unsigned int count_add = 0;
};

// The drawing-phase counter lives on the device as word 0, with word 1 as scratch that
// holds nothing between passes (starts, checkpoints, the other schedules and the cluster
// set word 0 alone).  A drawing pass advances it without a launch of its own (2 us each
// before): phases 0-2 read word 0 while phase 0 writes the advanced count to word 1,
// phases 3-5 read word 1 while phase 3 copies it back, so no launch writes the word it
// reads.
template <class Args>
__host__ inline void count_slots(Args& a, unsigned long long* word0, unsigned long long* word1, int k, bool draws) {
  a.phase_ptr = k < 3 ? word0 : word1;
  a.phase_off = k < 3 ? k : k - 6;
  a.count_out = !draws ? nullptr : k == 0 ? word1 : k == 3 ? word0 : nullptr;
  a.count_add = k == 0 ? 6 : 0;
}
__device__ __forceinline__ unsigned long long draw_count(const PhaseArgs& a) {
  const unsigned long long* p = a.phase_ptr;
  asm volatile("" : "+l"(p));  // after chain_wait
  return *p;
}
// Called after the update: a store that waits for a load would hold back the links asked
// for after it (FP64 Metropolis 32x32x64: 82.8 us, 84.8 with this first).
__device__ __forceinline__ void count_draws(const PhaseArgs& a) {
  if (a.count_out && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    __stcg(a.count_out, draw_count(a) + a.count_add);
}
// the drawing-phase number of this launch
__device__ __forceinline__ unsigned long long draw_phase(const PhaseArgs& a) {
  return (a.phase_ptr ? draw_count(a) : 0) + a.phase_off;
}

// The wavefront and the fused pairs, which read word 0 alone, advance it by this
// one-thread launch (inside a captured graph too).  Internal linkage: each
// translation unit that includes this header has its own copy.
static __global__ void advance_counter(unsigned long long* c, unsigned long long n) { *c += n; }

// ------------------------------------------------------- one link update --
// Update U_MU at site n of sublattice PAR: the body of the six launches of
// mc_up_per/pcc/pmc (mc_updates.h:129-465, mc_updates_pcc.h:4-214,
// mc_updates_pmc.h:4-247).  Shared by the per-phase kernels (CG = false) and
// the wavefront kernel (CG = true).
template <int MU, int PAR, int BC, int KIND, bool CG>
__device__ __forceinline__ void site64(const Links64T<CG>& L, const RngStore& R, const Geo& g,
                                       const PhaseArgs& a, const Nbr& n) {
  if (BC == BC_PCC && MU != DIR_Y && at_y0(g, n)) return;
  const int id = n.id;
  Quat<double> A = staple_sum<MU, BC, Links64T<CG>, double>(L, g, n, PAR);
  if (KIND == KIND_HB) {
    MrgStream st = R.load(id);
    Quat<double> U = heatbath_ref(A, (double)a.beta, st, a.err);
    if (!CG) chain_ready();
    L.st(MU, PAR, id, U);
    R.store(id, st);
  } else if (KIND == KIND_METRO) {
    MrgStream st = R.load(id);
    Quat<double> U = L.ld_own(MU, PAR, id);
    int acc = metropolis_ref(U, A, (double)a.beta, (double)a.eps, a.upd, st);
    if (!CG) chain_ready();
    L.st(MU, PAR, id, U);
    R.store(id, st);
    atomicAdd(a.accept + PAR * g.vh + id, acc);
  } else {
    Quat<double> U = overrelax_ref(A, L.ld_own(MU, PAR, id));
    if (!CG) chain_ready();
    L.st(MU, PAR, id, U);
  }
}

// FP32: the same updates with FP32 links and FP64 fix-ups; the heat-bath and
// Metropolis draw from the counter-based Philox stream of (site, phase), so
// no generator state is read or written.
// The new value of FP32 link U_mu of site `id` of sublattice `par` from its staple
// sum; gid is the site's global sublattice index (the Philox site counter and
// the accept slot), `links` and `id` address the link's store.  Metropolis
// accept counts are added only when count_accept is set.
template <int KIND, class L>
__device__ __forceinline__ Quat<float> link_new32(const L& links, const Quat<float>& A, const Geo& g,
                                                  const PhaseArgs& a, int mu, int par, int id, int gid, int renorm,
                                                  bool count_accept) {
  Quat<float> U;
  if (KIND == KIND_HB) {
    PhiloxStream st(a.keys, a.site_off + (unsigned int)gid, draw_phase(a));
    U = heatbath_fast(A, a.beta, st, a.err);
  } else if (KIND == KIND_METRO) {
    PhiloxStream st(a.keys, a.site_off + (unsigned int)gid, draw_phase(a));
    U = links.ld_own(mu, par, id);
    int acc = metropolis_fast(U, A, a.beta, a.eps, a.upd, st);
    if (count_accept) atomicAdd(a.accept + par * g.vh + gid, acc);
  } else {
    U = overrelax_fast(A, links.ld_own(mu, par, id));
  }
  return renorm ? renorm_fast(U) : U;
}
// the same with the staples gathered at n (a shared-memory tile in the fused-pair kernel)
template <int MU, int PAR, int BC, int KIND, class L>
__device__ __forceinline__ Quat<float> link_update32(const L& links, const Geo& g, const PhaseArgs& a, const Nbr& n,
                                                     int gid, int renorm, bool count_accept) {
  const Quat<float> A = staple_sum<MU, BC, L, float>(links, g, n, PAR);
  return link_new32<KIND>(links, A, g, a, MU, PAR, n.id, gid, renorm, count_accept);
}

template <int MU, int PAR, int BC, int KIND, bool CG>
__device__ __forceinline__ void site32(const Links32T<CG>& L, const RngStore& R, const Geo& g,
                                       const PhaseArgs& a, const Nbr& n, int renorm) {
  if (BC == BC_PCC && MU != DIR_Y && at_y0(g, n)) return;
  const Quat<float> U = link_update32<MU, PAR, BC, KIND>(L, g, a, n, n.id, renorm, true);
  if (!CG) chain_ready();
  L.st(MU, PAR, n.id, U);
}

// ---------------------------------------------------------- reductions --
// Deterministic FP64 sums: each CTA writes its partial (fixed tree order),
// the last CTA to finish adds the partials in index order and resets the
// arrival counter.  No floating-point atomics, so the result does not depend
// on CTA scheduling (the reference's en_av uses atomicAdd, observables.h:137-140).
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sums two values over the CTA into out2 (valid in thread 0).
__device__ __forceinline__ void block_sum2(double v0, double v1, double* out0, double* out1) {
  __shared__ double sh[2][kBlock / 32];
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = v0;
    sh[1][w] = v1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int i = 0; i < kBlock / 32; i++) {
      a += sh[0][i];
      b += sh[1][i];
    }
    *out0 = a;
    *out1 = b;
  }
}

// After thread 0 of every CTA stored its partial pair: the last CTA adds all
// partials in order, scales them and writes out[0..1]; with `err` also the
// device error word, as the int at out[2] (`out` is then the caller's pinned
// host memory, and one kernel brings the whole answer).
__device__ __forceinline__ void finish_sum2(double2* partials, unsigned int* counter, double scale,
                                            double* out, const int* err = nullptr) {
  __shared__ bool last;
  const unsigned int ctas = gridDim.x;
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned int prev = atomicAdd(counter, 1u);
    last = (prev == ctas - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // fixed-order sum over partials: per-thread strided chunks, then the CTA tree
  double a = 0, b = 0;
  for (unsigned int i = threadIdx.x; i < ctas; i += kBlock) {
    double2 v = __ldcg(partials + i);  // L2: written by other CTAs
    a += v.x;
    b += v.y;
  }
  __syncthreads();
  double sa, sb;
  block_sum2(a, b, &sa, &sb);
  if (threadIdx.x == 0) {
    out[0] = sa * scale;
    out[1] = sb * scale;
    if (err) *reinterpret_cast<int*>(out + 2) = __ldcg(err);
    *counter = 0u;
  }
}

// 1 - 1/2 Re tr of the plaquettes at one site, in the reference's product
// order (plaquette_yx/yt/xt, observables.h:1-21):
//   P_yx = U_y(x) U_x(x+y) U_y(x+x)^+ U_x(x)^+  and alike.
template <class L>
__device__ __forceinline__ Quat<double> ld64(const L& links, int d, int p, int id);
template <>
__device__ __forceinline__ Quat<double> ld64<Links64>(const Links64& links, int d, int p, int id) {
  return links.ld(d, p, id);
}
template <>
__device__ __forceinline__ Quat<double> ld64<Links32>(const Links32& links, int d, int p, int id) {
  Quat<float> u = links.ld(d, p, id);
  return Quat<double>{u.w, u.x, u.y, u.z};
}

// FP32 links: the three products in FP32 (the link's own precision), the
// result handed to the FP64 sums
__device__ __forceinline__ double plaq(const Links32& links, int mu, int nu, int p, int id, int omu, int onu) {
  Quat<float> A = q_mul(links.ld(mu, p, id), links.ld(nu, p ^ 1, id + omu));
  Quat<float> B = q_mul_bd(A, links.ld(mu, p ^ 1, id + onu));
  A = q_mul_bd(B, links.ld(nu, p, id));
  return 1.0 - (double)A.w;
}

template <class L>
__device__ __forceinline__ double plaq(const L& links, int mu, int nu, int p, int id, int omu,
                                       int onu) {
  // U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
  Quat<double> A = q_mul(ld64(links, mu, p, id), ld64(links, nu, p ^ 1, id + omu));
  Quat<double> B = q_mul_bd(A, ld64(links, mu, p ^ 1, id + onu));
  A = q_mul_bd(B, ld64(links, nu, p, id));
  return 1 - A.w;
}

// A measurement covers kMeasureIds sublattice indices of both parities per CTA
// and turn: warps 0-3 take the even sites, warps 4-7 the odd sites of the same
// indices.  The two need the same six link classes (a site's own links are the
// other's neighbours), so each link leaves HBM once; taking all even sites
// before all odd ones read the store twice.
//
// Bound by HBM on a large lattice, by the latency of one turn on a small one.
// A small lattice gets a CTA per 128 indices, one turn each, as long as that
// leaves SMs idle (16^3: 5 us; with eight sites in series per thread 14 us);
// above, four turns per CTA, which amortise its reduction where other launches
// fill the GPU (a batch of 96 replicas: 3% of its run).  A large one gets the CTAs that are
// resident at once on 148 SMs at the kernel's register count, which then walk
// the lattice side by side, so neighbours meet in L1 and L2 and no last wave
// runs half empty.  384^3, thermalised links: FP64 0.95 ms at 2 CTAs per SM (1.26 ms
// with twice as many CTAs, 1.7 ms with a CTA per 1024 indices and one parity after the
// other), FP32 0.55 ms at 4, site pairs 0.50-0.60 ms at 3 (0.89 ms before).
constexpr int kMeasureIds = kBlock / 2;
constexpr int kMeasureSMs = 148;
constexpr int kMeasurePerSM64 = 2, kMeasurePerSM32 = 4, kMeasurePerSMPair = 3;
// CTAs of a measurement over `ids` sublattice indices (pairs of them in the
// site-pair store).  The count depends on the lattice only, so the summation
// order is the same on every device and for a lattice measured alone or in a batch.
__host__ __device__ __forceinline__ unsigned int measure_blocks(long long ids, int per_sm) {
  const long long one = (ids + kMeasureIds - 1) / kMeasureIds, four = (one + 3) / 4;
  const long long most = one < kMeasureSMs ? one : four > kMeasureSMs ? four : kMeasureSMs;
  return (unsigned int)(most < kMeasureSMs * per_sm ? most : kMeasureSMs * per_sm);
}

// Energy and plaquette sums of CTA c of nb: -(1 - P_xt) and 3 - the sum of the
// three 1 - P of each site.  One site per thread and turn keeps few links live.
template <class L, bool PMC>
__device__ __forceinline__ void measure_sites(const L& links, const Geo& g, int c, int nb, double& e, double& pl) {
  const int p = threadIdx.x >= kMeasureIds;
  const unsigned int ids = (unsigned int)g.vh;
  unsigned int k = (unsigned int)c * kMeasureIds + threadIdx.x % kMeasureIds;
  for (chain_wait(k); k < ids; k += (unsigned int)nb * kMeasureIds) {
    const int id = (int)k;
    const int t = div_by(k, g.slice_m);
    const int s = id - t * g.slice;
    const Nbr n = make_nbr_slice(g, s, t, p);
    double a = plaq(links, DIR_Y, DIR_X, p, id, n.yp, n.xp);
    double b = plaq(links, DIR_Y, DIR_T, p, id, n.yp, n.tp);
    double cc = plaq(links, DIR_X, DIR_T, p, id, n.xp, n.tp);
    if (PMC && at_ytop(g, n)) {
      a = 0;
      b = 0;
    }
    e += -cc;
    pl += 3 - a - b - cc;  // the 1/3 of the plaquette average is applied once per thread
  }
  chain_ready();
}

}  // namespace qcd
