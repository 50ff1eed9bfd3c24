// Staple gather and the three link updates.
//
// Staple of U_mu(x) in the plane (mu, nu), with the reference's product order
// (mc_updates.h:158-176 and the five sibling kernels):
//   forward   U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
//   backward  U_nu(x+mu-nu)^+ U_mu(x-nu)^+ U_nu(x-nu)
// nu runs over (x, t) for mu = y, (y, t) for mu = x, (y, x) for mu = t, forward
// before backward, accumulated into a zero quaternion.  The boundary
// conditions are folded into the gather:
//   PCC  x and t links on the plane y = 0 are never updated
//        (mc_updates_pcc.h:29,83,134,189);
//   PMC  for mu = x, t the y staple that crosses y = Ly-1 <-> 0 is left out
//        (mc_updates_pmc.h:33,40,96,103,156,163,219,225); the y links
//        themselves use the periodic gather (mc_updates_pmc.h:250-251).
#pragma once
#include "lattice.cuh"
#include "rng.cuh"
#include "su2.cuh"

namespace qcd {

enum { KIND_METRO = 0, KIND_HB = 1, KIND_OR = 2 };

// device error word bits
// (DEVERR_TIMEOUT: a bounded wait of the wavefront or the fused-pair kernels ran out)
enum { DEVERR_HB_LOOP = 1, DEVERR_NONUNITARY = 2, DEVERR_TIMEOUT = 4 };

// The Kennedy-Pendleton rejection loop accepts a try with probability > 1/2 where
// beta |A| exceeds 1 (|A|: norm of the staple sum, up to 4) and with 0.443 (2 beta
// |A|)^1.5 where that is small.  This bound is reached when the staple sum is zero or not
// finite, or with couplings of a few hundredths and less; the update then stops and
// flags the error instead of spinning.
#define QCD_HB_MAX_TRIES 4096

template <int MU>
struct Planes {
  static constexpr int NU1 = MU == DIR_Y ? DIR_X : DIR_Y;
  static constexpr int NU2 = MU == DIR_T ? DIR_X : DIR_T;
};

// FP32 staples add their second product straight into the sum with
// multiply-adds (A + X Y^+, A + X Y); FP64 keeps the reference's separate
// product and sum, whose rounding the bit-parity tests pin.
__device__ __forceinline__ Quat<float> q_acc_mul_bd(const Quat<float>& A, const Quat<float>& a,
                                                    const Quat<float>& b) {
  Quat<float> c;
  c.w = A.w + a.w * b.w + a.x * b.x + a.y * b.y + a.z * b.z;
  c.x = A.x + a.x * b.w - a.w * b.x - a.y * b.z + a.z * b.y;
  c.y = A.y + a.y * b.w - a.z * b.x - a.w * b.y + a.x * b.z;
  c.z = A.z + a.z * b.w + a.y * b.x - a.w * b.z - a.x * b.y;
  return c;
}
__device__ __forceinline__ Quat<float> q_acc_mul(const Quat<float>& A, const Quat<float>& a, const Quat<float>& b) {
  Quat<float> c;
  c.w = A.w + a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z;
  c.x = A.x + a.x * b.w + a.w * b.x + a.y * b.z - a.z * b.y;
  c.y = A.y + a.y * b.w + a.z * b.x + a.w * b.y - a.x * b.z;
  c.z = A.z + a.z * b.w - a.y * b.x + a.w * b.z + a.x * b.y;
  return c;
}
__device__ __forceinline__ Quat<double> q_acc_mul_bd(const Quat<double>& A, const Quat<double>& a,
                                                     const Quat<double>& b) {
  return q_add(A, q_mul_bd(a, b));
}
__device__ __forceinline__ Quat<double> q_acc_mul(const Quat<double>& A, const Quat<double>& a,
                                                  const Quat<double>& b) {
  return q_add(A, q_mul(a, b));
}

template <int MU, int NU, int BC, class L, class R>
__device__ __forceinline__ void add_staples(const L& links, const Geo& g, const Nbr& n, int par,
                                            Quat<R>& A) {
  const int o = par ^ 1;
  const bool drop_fwd = BC == BC_PMC && NU == DIR_Y && at_ytop(g, n);
  const bool drop_bwd = BC == BC_PMC && NU == DIR_Y && at_y0(g, n);
  if (!drop_fwd) {
    Quat<R> a = links.ld(NU, o, n.id + off_plus(n, MU));
    Quat<R> b = links.ld(MU, o, n.id + off_plus(n, NU));
    Quat<R> c = links.ld(NU, par, n.id);
    A = q_acc_mul_bd(A, q_mul_bd(a, b), c);
  }
  if (!drop_bwd) {
    const int m = n.id + off_minus(n, NU);
    Quat<R> a = links.ld(NU, par, m + off_plus(n, MU));
    Quat<R> b = links.ld(MU, o, m);
    Quat<R> c = links.ld(NU, o, m);
    A = q_acc_mul(A, q_mul_adbd(a, b), c);
  }
}

template <int MU, int BC, class L, class R>
__device__ __forceinline__ Quat<R> staple_sum(const L& links, const Geo& g, const Nbr& n, int par) {
  Quat<R> A = q_zero<R>();
  add_staples<MU, Planes<MU>::NU1, BC>(links, g, n, par, A);
  add_staples<MU, Planes<MU>::NU2, BC>(links, g, n, par, A);
  return A;
}

// ------------------------------------------------ FP64 (reference parity) --

// Kennedy-Pendleton heat-bath exactly as the reference draws and rounds it
// (mc_updates.h:43-64): float uniforms and float logf/cospif/sincospif for the
// distribution, the new link built in double and normalised with rsqrt.
// Returns the new link X A^+ with A the normalised staple.
__device__ __forceinline__ Quat<double> heatbath_ref(Quat<double> A, double beta,
                                                     MrgStream& st, int* err) {
  double a;
  A = q_normalize_norm(A, &a);
  float inv = (float)(0.5 / (a * beta)), lf, aux;
  for (int tries = 1;; tries++) {
    float r0 = st.uniform(), r1 = st.uniform(), r2 = st.uniform();
    float c = cospif(2 * r1);
    lf = -(logf(r0) + c * c * logf(r2)) * inv;
    aux = 1 - st.uniform();
    if (!(aux * aux > 1 - lf)) break;
    if (tries >= QCD_HB_MAX_TRIES) {
      atomicOr(err, DEVERR_HB_LOOP);
      break;
    }
  }
  Quat<double> X;
  X.w = 1 - 2 * (double)lf;
  double nrm = sqrt(1 - X.w * X.w);
  float ct = 2 * st.uniform() - 1, sp, cp;
  sincospif(2 * st.uniform(), &sp, &cp);
  float stt = sqrtf(fmaxf(0.f, 1 - ct * ct));
  double v1 = ct, v2 = (double)stt * cp, v3 = (double)stt * sp;
  double s = nrm * rsqrt(v1 * v1 + v2 * v2 + v3 * v3);
  X.x = v1 * s;
  X.y = v2 * s;
  X.z = v3 * s;
  return q_mul_bd(X, A);
}

// exp(-s) > u decided in float unless u lies within 1e-4 (relative) of the
// float estimate, then in double (mc_updates.h:7-15).  Same decision as the
// double test.
__device__ __forceinline__ bool metropolis_accept(double s, double u) {
  const double tol = 1e-4;
  double ef = expf(-(float)s);
  if (u < ef * (1 - tol)) return true;
  if (u > ef * (1 + tol)) return false;
  return exp(-s) > u;
}

// `upd` Metropolis hits with proposals r U, r within eps of 1 (su2.h:87-97,
// mc_updates.h:16-36, 119-128); A (not normalised) is reused by every hit.
__device__ __forceinline__ int metropolis_ref(Quat<double>& U, const Quat<double>& A, double beta,
                                              double eps, int upd, MrgStream& st) {
  int acc = 0;
  for (int h = 0; h < upd; h++) {
    double r1 = st.uniform_double() - 0.5;
    double r2 = st.uniform_double() - 0.5;
    double r3 = st.uniform_double() - 0.5;
    double nrm = sqrt(r1 * r1 + r2 * r2 + r3 * r3);
    Quat<double> r;
    r.x = eps * r1 / nrm;
    r.y = eps * r2 / nrm;
    r.z = eps * r3 / nrm;
    r.w = sqrt(1 - eps * eps);
    Quat<double> Un = q_mul(r, U);
    Quat<double> dU{Un.w - U.w, Un.x - U.x, Un.y - U.y, Un.z - U.z};
    double s = -beta * q_retr_mul(dU, A);
    bool ok = s < 0 ? true : metropolis_accept(s, st.uniform_double());
    if (ok) {
      U = Un;
      acc++;
    }
  }
  return acc;
}

// U -> A^+ U^+ A^+ with A the normalised staple (mc_updates.h:109-115):
// leaves Re tr(U A) unchanged.
__device__ __forceinline__ Quat<double> overrelax_ref(Quat<double> A, const Quat<double>& U) {
  double a;
  A = q_normalize_norm(A, &a);
  Quat<double> B = q_mul_adbd(U, A);
  return q_mul_ad(A, B);
}

// ------------------------------------------- FP32 links + FP64 fix-ups ----
// The FP32 updates draw from a generator G with uniform() (float in (0, 1])
// and uniform_double() (double in (0, 1]): the counter-based PhiloxStream.

// Kennedy-Pendleton in FP32.  The accept test, which loses accuracy in single
// precision (1 - lf is within an ulp of 1 for large beta*|A|), is done in
// double.  The length of the spatial part is taken as n = 2 sqrt(lf (1 - lf))
// instead of sqrt(1 - X0^2): no cancellation as X0 -> 1, so float suffices.
// The draws come from the counter-based stream a whole block at a time: each
// try of the rejection loop takes one block (r0, r1, r2 and the accept
// uniform), the direction the first two words of the next one, the same
// words in the same order as drawing them one by one.
//
// The phase is bound by instruction issue, so the steps are written out short:
// exact one-step forms of the draws (PhiloxStream::u24), hardware log, sin and
// cos without the handling of denormals that their arguments never are, and the
// accept test in double only where single precision cannot decide it.
__device__ __forceinline__ float log2_normal(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float cos_normal(float x) {
  float y;
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sin_normal(float x) {
  float y;
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// one block of a try: t = log r0 + cos^2(2 pi r1) log r2 and 1 - the accept uniform
// (hardware approximations, absolute error ~2^-21: the cosine is taken of
// 2 pi (r1 - 1/2), which keeps the argument in [-pi, pi] and only flips the sign)
__device__ __forceinline__ void heatbath_try(const uint32_t w[4], float& t, float& aux) {
  const float c = cos_normal(6.2831853f * PhiloxStream::u24(w[1], 1.f, -0.5f));
  const float ln2 = 0.693147182464599609375f;
  t = __fmaf_rn(log2_normal(PhiloxStream::u24(w[0])), ln2,
                __fmul_rn(__fmul_rn(c, c), __fmul_rn(log2_normal(PhiloxStream::u24(w[2])), ln2)));
  aux = PhiloxStream::u24(w[3], -1.f, 1.f);
}
// aux^2 > 1 - lf in double.  The single-precision estimate of aux^2 + lf - 1 is
// off by less than 4e-7 for lf < 2, and above it the sign is plain; a NaN
// goes to the test in double.
__device__ __forceinline__ bool heatbath_reject(float aux, float lf) {
  const float v = __fmaf_rn(aux, aux, lf - 1.f);
  if (fabsf(v) > 1e-6f) return v > 0.f;
  return (double)aux * aux > 1.0 - (double)lf;
}
// direction of the spatial part from the first two words of a block
__device__ __forceinline__ void heatbath_direction(const uint32_t w[4], float& ct, float& stt, float& cp, float& sp) {
  ct = PhiloxStream::u24(w[0], 2.f, -1.f);
  const float angle = 6.2831853f * PhiloxStream::u24(w[1], 1.f, -0.5f);  // angle + pi
  sp = sin_normal(angle);
  cp = cos_normal(angle);
  stt = sqrtf(fmaxf(0.f, __fmaf_rn(-ct, ct, 1.f)));
}

template <class G>
__device__ __forceinline__ Quat<float> heatbath_fast(Quat<float> A, float beta, G& st, int* err) {
  float det = q_det(A);
  float rinv = rsqrtf(det);
  float a = det * rinv;
  A = Quat<float>{A.w * rinv, A.x * rinv, A.y * rinv, A.z * rinv};
  float inv = 0.5f / (a * beta);
  float lf, t, aux;
  uint32_t w[4];
  for (int tries = 1;; tries++) {
    st.block(w);
    heatbath_try(w, t, aux);
    lf = -t * inv;
    if (!heatbath_reject(aux, lf)) break;
    if (tries >= QCD_HB_MAX_TRIES) {
      atomicOr(err, DEVERR_HB_LOOP);
      break;
    }
  }
  const float x0 = 1.f - 2.f * lf;
  const float nrm = 2.f * sqrtf(lf * (1.f - lf));
  float ct, stt, cp, sp;
  st.block(w);
  heatbath_direction(w, ct, stt, cp, sp);
  Quat<float> X{x0, nrm * ct, -nrm * stt * cp, -nrm * stt * sp};
  return q_mul_bd(X, A);
}

// Over-relaxation U -> (Ahat U Ahat)^+, Ahat = A/|A| (mc_updates.h:109-115),
// written with the quaternion identity q p q = 2 <q, pbar> q - |q|^2 pbar:
//   U' = 2 (<A, Ubar> / |A|^2) Abar - U,   <A, Ubar> = 1/2 Re tr(U A),
// the same map as the reference's two products with ~16 operations instead of
// ~41; it keeps <A, Ubar> (the local action) and |U'| = |U| exactly in exact
// arithmetic.  FP32 only: the FP64 path keeps the reference's products.
__device__ __forceinline__ Quat<float> overrelax_fast(const Quat<float>& A, const Quat<float>& U) {
  const float c = __fdividef(2.f * q_retr_mul(A, U), q_det(A));
  return Quat<float>{c * A.w - U.w, -c * A.x - U.x, -c * A.y - U.y, -c * A.z - U.z};
}

// Metropolis with FP32 links: proposal and action change in float, the
// accept decision with the same single-then-double test as the reference.
template <class G>
__device__ __forceinline__ int metropolis_fast(Quat<float>& U, const Quat<float>& A, float beta,
                                               float eps, int upd, G& st) {
  int acc = 0;
  const float r0 = sqrtf(1.f - eps * eps);
  for (int h = 0; h < upd; h++) {
    float r1 = st.uniform(1.f, -0.5f);
    float r2 = st.uniform(1.f, -0.5f);
    float r3 = st.uniform(1.f, -0.5f);
    float sc = eps * rsqrtf(r1 * r1 + r2 * r2 + r3 * r3);
    Quat<float> r{r0, sc * r1, sc * r2, sc * r3};
    Quat<float> Un = q_mul(r, U);
    Quat<float> dU{Un.w - U.w, Un.x - U.x, Un.y - U.y, Un.z - U.z};
    double s = -(double)beta * (double)q_retr_mul(dU, A);
    bool ok = s < 0 ? true : metropolis_accept(s, st.uniform_double());
    if (ok) {
      U = Un;
      acc++;
    }
  }
  return acc;
}

// Re-projection of an FP32 link with the norm taken in double.  (A series for
// 1/sqrt near 1 saves about 20 instructions, but rounds one component in 10^9 to
// the other neighbouring float, and a long chain does not forget that.)
__device__ __forceinline__ Quat<float> renorm_fast(const Quat<float>& u) {
  double d = (double)u.w * u.w + (double)u.x * u.x + (double)u.y * u.y + (double)u.z * u.z;
  double inv = rsqrt(d);
  return Quat<float>{(float)(u.w * inv), (float)(u.x * inv), (float)(u.y * inv),
                     (float)(u.z * inv)};
}

}  // namespace qcd
