// Small lattices: all phases of a run of passes in one launch, the links in the
// shared memory of one cluster.
//
// A phase of a small lattice is a chain of latencies: the launch, links from L2, the
// update, the store's way back to L2.  One cluster of 16 CTAs holds the links in
// its distributed shared memory and walks through the passes by itself: links are
// copied in, each phase updates the CTA's own sites reading neighbours from the
// other CTAs' shared memory, the cluster's hardware barrier separates the phases,
// and the links are copied out.  Index j of a parity belongs to CTA j >> lg, slot
// j mod 2^lg.  The updates are the phase kernels' own code on another store, in the
// same order, so the results are theirs.  No wait on memory needs a bound: the
// CTAs of a cluster run together by construction.
//
// What is left is the latency of one update (8^3 takes 1.9 us a phase in FP64, 16^3
// 2.4) and, as the CTAs fill, the rate of remote shared-memory reads, so the whole
// GPU wins early (kResidentItems).  Phase launches -> cluster, back to back: five FP64
// heat-bath sweeps of 16^3 88-93 -> 73 us, of 8^3 75 -> 57 us; two FP32 sweeps with three
// over-relaxation passes of 16^3 110 -> 70 us, of 18x20x22 112 -> 80 us.
#pragma once
#include "paired.cuh"

namespace qcd {

constexpr int kResidentCtas = 16;
constexpr int kResidentLog = 8;  // most slots of a CTA: 2^8, one thread each
constexpr int kResidentPasses = 64;
// Largest work of a phase (sites; pairs) that one cluster takes instead of launches on
// the whole GPU.  Heat-bath and over-relaxation 4096, phase launches against cluster, us:
//   2048 pairs   one heat-bath sweep 20.4 / 18.3, two sweeps with three OR passes 123 / 86
//   2400 pairs                       21.0 / 24.0                                 128 / 122
//   3360 pairs                       21.5 / 24.8                                 134 / 127
//   4080 pairs                       21.4 / 25.8                                 132 / 135
//   2048 FP64    one heat-bath sweep 18.9 / 17.2, five 93 / 75, two with one OR pass 61 / 49
//   2560 FP64                        20.1 / 21.5       99 / 94                       67 / 61
//   4000 FP64                        19.8 / 23.1       97 / 101                      66 / 67
//   4000 planes  one heat-bath sweep 16.1 / 15.8, two with three OR passes 112 / 79
// so from 2048 to 4096 pairs or FP64 sites the cluster gains where over-relaxation passes
// or several sweeps share a call, and a call of one sweep is up to a fifth longer.
// Metropolis, whose hits are longer, 2048 (two sweeps, 2048 FP64 sites 36 / 31, 2048 pairs
// 46 / 37; 3360 pairs, more hits, 205 / 218) but on single-precision planes, whose sites
// have half the bytes to fetch (4000 sites 34 / 31).
constexpr int kResidentItems = 4096, kResidentItemsMetro = 2048;
static_assert(kResidentItems <= kResidentCtas << kResidentLog, "slots for every site");

struct ResidentProgram {
  int n;  // passes
  unsigned char kind[kResidentPasses], renorm[kResidentPasses];
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// (volatile: not to be moved across the cluster barrier)
__device__ __forceinline__ float4 ld_cluster(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ double2 as_double2(const float4& v) {
  return make_double2(__hiloint2double(__float_as_int(v.y), __float_as_int(v.x)),
                      __hiloint2double(__float_as_int(v.w), __float_as_int(v.z)));
}
__device__ __forceinline__ void st_local_d2(uint32_t a, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void st_local_f4(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// 16-byte slots in the cluster's shared memory: row r of 2^lg slots per CTA
struct ClusterRows {
  uint32_t base;  // address of the rows in this CTA's shared memory
  int lg;
  __device__ __forceinline__ uint32_t local(int row, int j) const {
    return base + (uint32_t)((row << lg) + (j & ((1 << lg) - 1))) * 16u;
  }
  // rows `row`.. of index j, wherever they are (a branch to the plain path for the
  // CTA's own slots measured 5-30% slower)
  template <int N>
  __device__ __forceinline__ void get(int row, int j, float4 out[N]) const {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local(row, j)), "r"(j >> lg));
    for (int i = 0; i < N; i++) out[i] = ld_cluster(a + i * stride());
  }
  __device__ __forceinline__ uint32_t stride() const { return 16u << lg; }  // from row to row
};

// The three stores in the cluster: ld reads any site or pair, st writes one of
// this CTA's.  kRows 16-byte rows per index.
struct Cluster64 {
  static constexpr int kRows = 12;
  static constexpr bool kStored = true;  // draws from the stored generator
  typedef Quat<double> Link;
  typedef Links64 Global;
  ClusterRows m;
  __device__ __forceinline__ Link ld(int d, int p, int j) const {
    float4 r[2];
    m.get<2>(2 * (int)plane_of(d, p), j, r);
    const double2 u = as_double2(r[0]), v = as_double2(r[1]);
    return Link{u.x, u.y, v.x, v.y};
  }
  __device__ __forceinline__ Link ld_own(int d, int p, int j) const { return ld(d, p, j); }
  __device__ __forceinline__ void st(int d, int p, int j, const Link& u) const {
    const uint32_t a = m.local(2 * (int)plane_of(d, p), j);
    st_local_d2(a, u.w, u.x);
    st_local_d2(a + m.stride(), u.y, u.z);
  }
};
struct Cluster32 {
  static constexpr int kRows = 6;
  static constexpr bool kStored = false;
  typedef Quat<float> Link;
  typedef Links32 Global;
  ClusterRows m;
  __device__ __forceinline__ Link ld(int d, int p, int j) const {
    float4 r[1];
    m.get<1>((int)plane_of(d, p), j, r);
    return Link{r[0].x, r[0].y, r[0].z, r[0].w};
  }
  __device__ __forceinline__ Link ld_own(int d, int p, int j) const { return ld(d, p, j); }
  __device__ __forceinline__ void st(int d, int p, int j, const Link& u) const {
    st_local_f4(m.local((int)plane_of(d, p), j), u.w, u.x, u.y, u.z);
  }
};
struct ClusterPair {
  static constexpr int kRows = 12;
  static constexpr bool kStored = false;
  typedef Q2 Link;
  typedef Pair32 Global;
  ClusterRows m;
  int vhp;
  __device__ __forceinline__ Link ld(int d, int p, int j) const {
    float4 r[2];
    m.get<2>(2 * (int)plane_of(d, p), j, r);
    return Link{f2(r[0].x, r[0].y), f2(r[0].z, r[0].w), f2(r[1].x, r[1].y), f2(r[1].z, r[1].w)};
  }
  __device__ __forceinline__ Link ld_own(int d, int p, int j) const { return ld(d, p, j); }
  __device__ __forceinline__ void st(int d, int p, int j, const Link& q) const {
    const uint32_t a = m.local(2 * (int)plane_of(d, p), j);
    st_local_f4(a, q.w.x, q.w.y, q.x.x, q.x.y);
    st_local_f4(a + m.stride(), q.y.x, q.y.y, q.z.x, q.z.y);
  }
};

// One staple added to the sum, forward or backward (add_staples, add_staples2)
template <class R>
__device__ __forceinline__ Quat<R> add_forward(const Quat<R>& A, const Quat<R>& a, const Quat<R>& b,
                                               const Quat<R>& c) {
  return q_acc_mul_bd(A, q_mul_bd(a, b), c);
}
template <class R>
__device__ __forceinline__ Quat<R> add_backward(const Quat<R>& A, const Quat<R>& a, const Quat<R>& b,
                                                const Quat<R>& c) {
  return q_acc_mul(A, q_mul_adbd(a, b), c);
}
__device__ __forceinline__ Q2 add_forward(const Q2& A, const Q2& a, const Q2& b, const Q2& c) {
  return p2_acc_mul_bd(A, p2_mul_bd(a, b), c);
}
__device__ __forceinline__ Q2 add_backward(const Q2& A, const Q2& a, const Q2& b, const Q2& c) {
  return p2_acc_mul_ad(A, p2_mul(b, a), c);
}
template <class R>
__device__ __forceinline__ Quat<R> swapped_if(bool swap, const Quat<R>& q) {
  return q;
}
__device__ __forceinline__ Q2 swapped_if(bool swap, const Q2& q) { return swap ? swap_lanes(q) : q; }

// Direction, parity and boundary are run-time values here, so that the phases
// share one piece of code: with a copy for each, every phase of a small lattice
// begins by fetching its instructions.  All twelve links are asked for before the
// first product.  pair: lanes trade places across the row seam.
template <class S>
__device__ __forceinline__ typename S::Link resident_staples(const S& L, const Geo& g, const Nbr& n, int mu, int par,
                                                             int bc, bool pair) {
  const int o = par ^ 1, om = off_plus(n, mu);
  const bool sp = pair && n.t == g.lt - 1, sm = pair && n.t == 0;
  typename S::Link a[4], b[4], c[4];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int nu = i == 0 ? (mu == DIR_Y ? DIR_X : DIR_Y) : (mu == DIR_T ? DIR_X : DIR_T);
    const int f = n.id + off_plus(n, nu), m = n.id + off_minus(n, nu);
    const bool seam_p = nu == DIR_T && sp, seam_m = nu == DIR_T && sm, mu_p = mu == DIR_T && sp;
    a[2 * i] = swapped_if(mu_p, L.ld(nu, o, n.id + om));
    b[2 * i] = swapped_if(seam_p, L.ld(mu, o, f));
    c[2 * i] = L.ld(nu, par, n.id);
    a[2 * i + 1] = swapped_if(mu_p || seam_m, L.ld(nu, par, m + om));
    b[2 * i + 1] = swapped_if(seam_m, L.ld(mu, o, m));
    c[2 * i + 1] = swapped_if(seam_m, L.ld(nu, o, m));
  }
  typename S::Link A{};
  const bool masked = bc == BC_PMC && mu != DIR_Y;  // the first plane is then the y plane
  if (!(masked && at_ytop(g, n))) A = add_forward(A, a[0], b[0], c[0]);
  if (!(masked && at_y0(g, n))) A = add_backward(A, a[1], b[1], c[1]);
  A = add_forward(A, a[2], b[2], c[2]);
  return add_backward(A, a[3], b[3], c[3]);
}

// One update of site or pair n; the generator words of FP64 in `rng` (this CTA's
// shared memory, six rows of 2^lg words).
template <int KIND>
__device__ __forceinline__ void resident_update(const Cluster64& L, uint32_t* rng, const Geo& g, const PhaseArgs& a,
                                                const Nbr& n, int mu, int par, int bc, int rn) {
  const int l = n.id & ((1 << L.m.lg) - 1), step = 1 << L.m.lg;
  const Quat<double> A = resident_staples(L, g, n, mu, par, bc, false);
  if (KIND == KIND_OR) {
    L.st(mu, par, n.id, overrelax_ref(A, L.ld_own(mu, par, n.id)));
  } else {
    MrgStream st;
    for (int i = 0; i < 3; i++) {
      st.s1[i] = rng[i * step + l];
      st.s2[i] = rng[(3 + i) * step + l];
    }
    if (KIND == KIND_HB) {
      L.st(mu, par, n.id, heatbath_ref(A, (double)a.beta, st, a.err));
    } else {
      Quat<double> U = L.ld_own(mu, par, n.id);
      const int acc = metropolis_ref(U, A, (double)a.beta, (double)a.eps, a.upd, st);
      L.st(mu, par, n.id, U);
      atomicAdd(a.accept + par * g.vh + n.id, acc);
    }
    for (int i = 0; i < 3; i++) {
      rng[i * step + l] = st.s1[i];
      rng[(3 + i) * step + l] = st.s2[i];
    }
  }
}
template <int KIND>
__device__ __forceinline__ void resident_update(const Cluster32& L, uint32_t* rng, const Geo& g, const PhaseArgs& a,
                                                const Nbr& n, int mu, int par, int bc, int rn) {
  const Quat<float> A = resident_staples(L, g, n, mu, par, bc, false);
  L.st(mu, par, n.id, link_new32<KIND>(L, A, g, a, mu, par, n.id, n.id, rn, true));
}
template <int KIND>
__device__ __forceinline__ void resident_update(const ClusterPair& L, uint32_t* rng, const Geo& gh,
                                                const PhaseArgs& a, const Nbr& n, int mu, int par, int bc, int rn) {
  const Q2 A = resident_staples(L, gh, n, mu, par, bc, true);
  L.st(mu, par, n.id, pair_new<KIND>(L, A, a, mu, par, n.id, rn));
}

// bytes of shared memory of a CTA
template <class S>
__host__ __device__ constexpr int resident_bytes(int lg) {
  return (S::kRows * 16 + (S::kStored ? 24 : 0)) << lg;
}

// Grid: one cluster of kResidentCtas CTAs; g: the half geometry for pairs.  `count`:
// the drawing-phase counter's word.
template <class S, int SK>
__global__ void __launch_bounds__(1 << kResidentLog, 1)
    resident(S L, typename S::Global global, RngStore R, Geo g, PhaseArgs a, ResidentProgram p, int bc,
             unsigned long long* count) {
  extern __shared__ __align__(16) unsigned char smem[];
  L.m.base = (uint32_t)__cvta_generic_to_shared(smem);
  uint32_t* rng = reinterpret_cast<uint32_t*>(smem + (size_t)(S::kRows * 16 << L.m.lg));
  const int j0 = blockIdx.x << L.m.lg, n = min(g.vh - j0, 1 << L.m.lg);
  int l = threadIdx.x;  // this thread's slot
  chain_wait(l);
  const int t = div_by((unsigned int)(j0 + l), g.slice_m), s = j0 + l - t * g.slice;
  if (l < n) {
    for (int c = 0; c < 6; c++) L.st(c >> 1, c & 1, j0 + l, global.ld_own(c >> 1, c & 1, j0 + l));
#pragma unroll
    for (int i = 0; i < (S::kStored ? 6 : 0); i++) rng[(i << L.m.lg) + l] = R.get(i, j0 + l);
  }
  const unsigned long long drawn0 = draw_count(a);
  cluster_barrier();
  int drawn = 0;
  a.phase_ptr = nullptr;
  for (int i = 0; i < p.n; i++) {
    const int kind = p.kind[i], rn = p.renorm[i];
#pragma unroll 1
    for (int k = 0; k < 6; k++) {
      const int mu = k >> 1, par = k & 1;
      a.phase_off = (long long)drawn0 + drawn + k;
      if (l < n) {
        const Nbr nb = make_nbr_slice(g, s, t, par);
        if (!(bc == BC_PCC && mu != DIR_Y && at_y0(g, nb))) {
          if (kind == KIND_OR)
            resident_update<KIND_OR>(L, rng, g, a, nb, mu, par, bc, rn);
          else
            resident_update<SK>(L, rng, g, a, nb, mu, par, bc, rn);
        }
      }
      cluster_barrier();
    }
    if (kind != KIND_OR) drawn += 6;
  }
  chain_ready();
  if (l < n) {
    for (int c = 0; c < 6; c++) global.st(c >> 1, c & 1, j0 + l, L.ld_own(c >> 1, c & 1, j0 + l));
#pragma unroll
    for (int i = 0; i < (S::kStored ? 6 : 0); i++) R.put(i, j0 + l, rng[(i << L.m.lg) + l]);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && drawn) *count = drawn0 + drawn;
}

}  // namespace qcd
