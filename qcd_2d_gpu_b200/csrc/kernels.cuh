// Device kernels of the sweep, the starts, re-projection, measurement and the
// layout conversions.  Launch geometry: one thread per sublattice site,
// 256 threads per CTA, ragged tail masked (the reference instead requires the
// CTA size to divide V/2, kernel.cu:66-70).
#pragma once
#include <curand_kernel.h>
#include "lattice.cuh"
#include "rng.cuh"
#include "su2.cuh"
#include "updates.cuh"
#include "sites.cuh"

namespace qcd {

// ------------------------------------------------------------ one phase --
// Launch grid tile_grid(g), kTileThreads threads.  FP64 CTAs per SM, measured: seven (72
// registers) for every kind; over-relaxation passes 48x64x80 22.9 us and 128^3 197 us
// (24.9 and 201 at nine), heat-bath 64^3 40.1 and 128^3 283 us (40.6 and 288 at nine, 45.0
// and 294 at six), Metropolis 64^3 63.2 us (64.5 at eight, 69.9 at six).
template <int MU, int PAR, int BC, int KIND>
__global__ void __launch_bounds__(kTileThreads, 7) phase64(Links64 L, RngStore R, Geo g, PhaseArgs a) {
  Nbr n;
  if (!tile_nbr<PAR>(g, n)) return;
  site64<MU, PAR, BC, KIND, false>(L, R, g, a, n);
  if (KIND != KIND_OR) count_draws(a);
}

// FP32 planes: eight CTAs per SM, which leaves registers to ask for several links at
// once (heat-bath pass 126x128x130 149 -> 145 us, 54x62x70 27.4 -> 25.7 us against the
// compiler's 32-36 registers; the same at six, 148 at ten).
template <int MU, int PAR, int BC, int KIND>
__global__ void __launch_bounds__(kTileThreads, 8) phase32(Links32 L, RngStore R, Geo g, PhaseArgs a) {
  Nbr n;
  if (!tile_nbr<PAR>(g, n)) return;
  site32<MU, PAR, BC, KIND, false>(L, R, g, a, n, a.renorm);
  if (KIND != KIND_OR) count_draws(a);
}

// ------------------------------------------------------------ RNG setup --
// curand_init(seed, id, 0) per half-lattice site (lattice_setup.h:15-21),
// by jumps from curand_init(seed, 0, 0) (mrg_cta_base, mrg_jump_from;
// `jumps` holds mrg_jump_table).
static_assert(kBlock == kMrgJumps, "one jump matrix per thread of a CTA");
__global__ void __launch_bounds__(kBlock) rng_setup(RngStore R, unsigned long long seed, int vh,
                                                    const uint32_t* __restrict__ jumps) {
  __shared__ unsigned int base[6];
  const int id0 = blockIdx.x * kBlock;
  if (threadIdx.x == 0) mrg_cta_base(base, jumps, seed, (unsigned long long)id0);
  __syncthreads();
  const int id = id0 + threadIdx.x;
  if (id >= vh) return;
  R.store(id, mrg_jump_from(base, jumps, threadIdx.x));
}

// ------------------------------------------------------------ starts -----
__device__ __forceinline__ void put(const Links64& L, int d, int p, int id, const Quat<double>& u) {
  L.st(d, p, id, u);
}
__device__ __forceinline__ void put(const Links32& L, int d, int p, int id, const Quat<double>& u) {
  L.st(d, p, id, Quat<float>{(float)u.w, (float)u.x, (float)u.y, (float)u.z});
}

// Cold start (id_init2, lattice_setup.h:38-51).
template <class L>
__global__ void __launch_bounds__(kBlock) init_cold(L links, int vh) {
  const int id = blockIdx.x * kBlock + threadIdx.x;
  if (id >= vh) return;
  for (int p = 0; p < 2; p++)
    for (int d = 0; d < 3; d++) put(links, d, p, id, q_one<double>());
}

// uniform cube (-0.5, 0.5]^4, normalised (su2_rand, su2.h:29-34)
__device__ __forceinline__ Quat<double> random_link(MrgStream& st) {
  Quat<double> a;
  a.w = st.uniform_double() - 0.5;
  a.x = st.uniform_double() - 0.5;
  a.y = st.uniform_double() - 0.5;
  a.z = st.uniform_double() - 0.5;
  return q_normalize(a);
}

// Hot start (rand_init2 lattice_setup.h:24-37; rand_init2_pcc :52-81): stream id
// fills even y, x, t then odd y, x, t; with PCC the x and t links at y = 0 are
// the identity and consume no draws.

template <class L>
__global__ void __launch_bounds__(kBlock) init_hot(L links, RngStore R, Geo g, int pcc) {
  const int id = blockIdx.x * kBlock + threadIdx.x;
  if (id >= g.vh) return;
  MrgStream st = R.load(id);
  for (int p = 0; p < 2; p++) {
    const Nbr n = make_nbr(g, id, p);
    const bool frozen = pcc && at_y0(g, n);
    for (int d = 0; d < 3; d++) {
      if (d != DIR_Y && frozen)
        put(links, d, p, id, q_one<double>());
      else
        put(links, d, p, id, random_link(st));
    }
  }
  R.store(id, st);
}

// ------------------------------------------------------- re-projection --
// normalize (lattice_setup.h:202-207): every link divided by its norm.
__global__ void __launch_bounds__(kBlock) normalize64(Links64 L, int vh) {
  const int id = blockIdx.x * kBlock + threadIdx.x;
  if (id >= vh) return;
  for (int p = 0; p < 2; p++)
    for (int d = 0; d < 3; d++) L.st(d, p, id, q_normalize(L.ld_own(d, p, id)));
}
__global__ void __launch_bounds__(kBlock) normalize32(Links32 L, int vh) {
  const int id = blockIdx.x * kBlock + threadIdx.x;
  if (id >= vh) return;
  for (int p = 0; p < 2; p++)
    for (int d = 0; d < 3; d++) L.st(d, p, id, renorm_fast(L.ld_own(d, p, id)));
}

// ----------------------------------------------------- layout changes ---
// reference AoS: phi[(p*Vh + id)*12 + d*4 + c].  A CTA moves 256 consecutive
// sites of one parity through shared memory, so that both sides are read and
// written in whole lines: HBM-bound, 256^3 FP64 0.54 ms for 3.2 GB (1.05 ms with
// a thread reading or writing its own 96 B).  The AoS side is accessed in
// 8-byte words, because a caller's buffer need not be aligned further.
// A staged site takes 14 doubles: at that stride the 16-byte accesses of eight
// neighbouring threads fall in different banks.
constexpr int kAosPad = 14;
constexpr int kAosShared = kBlock * kAosPad;  // doubles

// n sites from AoS site `first` on, staged from slot `slot` on (n <= kBlock,
// every thread of the CTA takes part)
template <int N>
__device__ __forceinline__ void aos_stage(double* sh, int slot, const double* __restrict__ aos, size_t first, int n) {
  constexpr int per = N * 12 / kBlock;
  double v[per];
#pragma unroll
  for (int k = 0; k < per; k++) {
    const int i = k * kBlock + threadIdx.x;
    if (i < n * 12) v[k] = __ldcs(aos + first * 12 + i);
  }
#pragma unroll
  for (int k = 0; k < per; k++) {
    const int i = k * kBlock + threadIdx.x;
    if (i < n * 12) sh[(slot + i / 12) * kAosPad + i % 12] = v[k];
  }
}
template <int N>
__device__ __forceinline__ void aos_unstage(const double* sh, int slot, double* __restrict__ aos, size_t first,
                                            int n) {
#pragma unroll
  for (int k = 0; k < N * 12 / kBlock; k++) {
    const int i = k * kBlock + threadIdx.x;
    if (i < n * 12) aos[first * 12 + i] = sh[(slot + i / 12) * kAosPad + i % 12];
  }
}
// link d of the site in a slot
__device__ __forceinline__ Quat<double> aos_get(const double* sh, int slot, int d) {
  const double2* s = reinterpret_cast<const double2*>(sh + slot * kAosPad + d * 4);
  const double2 a = s[0], b = s[1];
  return Quat<double>{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void aos_set(double* sh, int slot, int d, const Quat<double>& u) {
  double2* s = reinterpret_cast<double2*>(sh + slot * kAosPad + d * 4);
  s[0] = make_double2(u.w, u.x);
  s[1] = make_double2(u.y, u.z);
}
__device__ __forceinline__ Quat<float> narrow(const Quat<double>& u) {
  return Quat<float>{(float)u.w, (float)u.x, (float)u.y, (float)u.z};
}
__device__ __forceinline__ Quat<double> widen(const Quat<double>& u) { return u; }
__device__ __forceinline__ Quat<double> widen(const Quat<float>& u) { return Quat<double>{u.w, u.x, u.y, u.z}; }

// Launch grid (ceil(V/2 / kBlock), 2): blockIdx.y is the parity.
template <class L>
__global__ void __launch_bounds__(kBlock) aos_to_soa(const double* __restrict__ aos, L links, int vh) {
  __shared__ __align__(16) double sh[kAosShared];
  const int id0 = blockIdx.x * kBlock, p = blockIdx.y;
  const int n = vh - id0 < kBlock ? vh - id0 : kBlock;
  aos_stage<kBlock>(sh, 0, aos, (size_t)p * vh + id0, n);
  __syncthreads();
  if (threadIdx.x < n)
    for (int d = 0; d < 3; d++) put(links, d, p, id0 + threadIdx.x, aos_get(sh, threadIdx.x, d));
}
template <class L>
__global__ void __launch_bounds__(kBlock) soa_to_aos(L links, double* __restrict__ aos, int vh) {
  __shared__ __align__(16) double sh[kAosShared];
  const int id0 = blockIdx.x * kBlock, p = blockIdx.y;
  const int n = vh - id0 < kBlock ? vh - id0 : kBlock;
  if (threadIdx.x < n)
    for (int d = 0; d < 3; d++) aos_set(sh, threadIdx.x, d, widen(links.ld_own(d, p, id0 + threadIdx.x)));
  __syncthreads();
  aos_unstage<kBlock>(sh, 0, aos, (size_t)p * vh + id0, n);
}

// en_av<PMC> (observables.h:99-141): energy = mean of -(1 - P_xt), plaquette
// = mean of (P_yx + P_yt + P_xt)/3; with PMC the y plaquettes at y = Ly-1 count
// as 1.  out[0] = energy, out[1] = plaquette.
template <class L, int PMC, int PER_SM>
__global__ void __launch_bounds__(kBlock, PER_SM) measure(L links, Geo g, double2* partials, unsigned int* counter,
                                                          double* out, const int* err) {
  double e = 0, pl = 0;
  measure_sites<L, PMC != 0>(links, g, blockIdx.x, gridDim.x, e, pl);  // grid: measure_blocks(V/2, PER_SM)
  double se, sp;
  block_sum2(e, pl * (1.0 / 3.0), &se, &sp);
  if (threadIdx.x == 0) partials[blockIdx.x] = make_double2(se, sp);
  finish_sum2(partials, counter, 1.0 / (2.0 * (double)g.vh), out, err);
}

// Unitarity: out[0] = mean det, out[1] = number of links with |det-1| > tol
// or not finite (print_det, lattice_setup.h:176-183, plus a NaN/Inf check).
template <class L>
__global__ void __launch_bounds__(kBlock) unitarity(L links, int vh, double tol, double2* partials,
                                                    unsigned int* counter, double* out, const int* err) {
  const int id = blockIdx.x * kBlock + threadIdx.x;
  double s = 0, bad = 0;
  if (id < vh) {
    for (int p = 0; p < 2; p++)
      for (int d = 0; d < 3; d++) {
        double det = q_det(ld64(links, d, p, id));
        s += det;
        if (!(fabs(det - 1.0) <= tol)) bad += 1;
      }
  }
  double ss, sb;
  block_sum2(s, bad, &ss, &sb);
  if (threadIdx.x == 0) partials[blockIdx.x] = make_double2(ss, sb);
  finish_sum2(partials, counter, 1.0, out, err);
}

// ----------------------------------------------------------- RNG tape ----
struct TapeRec {
  double ud;
  float uf, log_uf, cospi_2uf, sc_sin, sc_cos;
  unsigned int same_step;
};

__global__ void __launch_bounds__(kBlock) rng_tape(unsigned long long seed, long long first, int n_streams,
                                                   int n_draws, TapeRec* out) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n_streams) return;
  curandStateMRG32k3a_t st;
  curand_init(seed, (unsigned long long)(first + i), 0ull, &st);
  for (int k = 0; k < n_draws; k++) {
    curandStateMRG32k3a_t cp = st;
    float f = curand_uniform(&cp);
    double d = curand_uniform_double(&st);
    unsigned int same = 1;
    for (int j = 0; j < 3; j++) same &= (cp.s1[j] == st.s1[j]) & (cp.s2[j] == st.s2[j]);
    TapeRec r;
    r.ud = d;
    r.uf = f;
    r.log_uf = logf(f);
    r.cospi_2uf = cospif(2 * f);
    float s, c;
    sincospif(2 * f, &s, &c);
    r.sc_sin = s;
    r.sc_cos = c;
    r.same_step = same;
    out[(size_t)i * n_draws + k] = r;
  }
}

}  // namespace qcd
