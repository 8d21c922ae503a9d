// cp_dual.cuh -- forward-mode dual numbers and the integrand written over them, for the adjoint
// (gradient) kernel and the flow's training.  A dual number carries a value and tangents in FP32;
// every operation applies the chain rule exactly, so the tangents are the derivatives of the FP32
// evaluation.
//
// The integrand below is the plain form of the same formulas as cp_had_eval (cp_integrand.cuh): it
// skips the compensated-FP32 refinements, which matter for the value at 1e-6 but not for gradients
// checked at 1e-4.  Parameters that the gradient is taken against enter as duals: ln tauMin (the
// pT_hat cut), k_ren, and ln Lambda_nf^2 (alpha_s(mZ)).
//
// Callers hold CpDual<N> with tangents 0..2 for x0, x1, x2 and, for N = 6, 3..5 for alpha_s(mZ),
// k_ren and the pT_hat cut.  Inside, a number's type names the tangents it can have (CpSp<mask>):
// the kinematics depend on x0, x2 and the cut only, a beam's x on x0, x1 and the cut, alpha_s alone
// on alpha_s(mZ) and k_ren.  The others are never formed: with every tangent carried through every
// operation, the zeros took 12% of the three-tangent pass's instructions and 23% of the six-tangent
// one's (2^20 points: 313 -> 279 and 460 -> 345 us).  A product with a single non-zero term is rounded on its own (cp_mul_rn),
// as the FMA with a zero term would round it, so tangents and values keep their last bits.
#pragma once
#include <type_traits>
#include "cp_integrand.cuh"

template <int N>
struct CpDual {
  float v;
  float d[N];
};

template <int N>
CP_HD CpDual<N> cp_dconst(float v)
{
  CpDual<N> r;
  r.v = v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = 0.f;
  return r;
}
template <int N>
CP_HD CpDual<N> cp_dvar(float v, int k)
{
  CpDual<N> r = cp_dconst<N>(v);
  r.d[k] = 1.f;
  return r;
}

// a product that no later addition is contracted with
CP_HD float cp_mul_rn(float a, float b)
{
#if defined(__CUDA_ARCH__)
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}

CP_HD constexpr int cp_bits_in(unsigned m) { return m ? (int)(m & 1u) + cp_bits_in(m >> 1) : 0; }

#if defined(__CUDACC__)
#define CP_HD_MEMBER __host__ __device__ __forceinline__
#else
#define CP_HD_MEMBER inline
#endif

// a dual number with the tangents of the mask M (bit k: tangent k), stored packed
template <unsigned M>
struct CpSp {
  static constexpr unsigned mask = M;
  float v;
  float d[M ? cp_bits_in(M) : 1];
  template <int K>
  static constexpr bool has() { return (M >> K) & 1u; }
  template <int K>
  CP_HD_MEMBER float& at() { return d[cp_bits_in(M & ((1u << K) - 1u))]; }
  template <int K>
  CP_HD_MEMBER float at() const { return d[cp_bits_in(M & ((1u << K) - 1u))]; }
};

// f(integral_constant<K>) for every tangent K of the mask
template <unsigned M, int K = 0, class F>
CP_HD void cp_tangents(const F& f)
{
  if constexpr ((M >> K) != 0u) {
    if constexpr ((M >> K) & 1u) f(std::integral_constant<int, K>{});
    cp_tangents<M, K + 1>(f);
  }
}
#define CP_TANGENTS(M) cp_tangents<M>([&](auto k_) { constexpr int K = decltype(k_)::value;
#define CP_TANGENTS_END })

template <unsigned M, int N>
CP_HD CpSp<M> cp_sp(const CpDual<N>& a)
{
  static_assert((M >> N) == 0u, "tangents of the mask exist");
  CpSp<M> r;
  r.v = a.v;
  CP_TANGENTS(M) r.template at<K>() = a.d[K]; CP_TANGENTS_END;
  return r;
}
// the same number with more tangents (zero)
template <unsigned R, unsigned M>
CP_HD CpSp<R> cp_widen(const CpSp<M>& a)
{
  static_assert((M & ~R) == 0u, "no tangent is dropped");
  CpSp<R> r;
  r.v = a.v;
  CP_TANGENTS(R)
    if constexpr (CpSp<M>::template has<K>()) r.template at<K>() = a.template at<K>();
    else r.template at<K>() = 0.f;
  CP_TANGENTS_END;
  return r;
}

// r.v = val; tangents of both operands, of the first alone, of the second alone
#define CP_SP_BIN(op, val, both, first, second)                                              \
  template <unsigned A, unsigned B>                                                          \
  CP_HD CpSp<(A | B)> operator op(const CpSp<A>& a, const CpSp<B>& b)                        \
  {                                                                                          \
    CpSp<(A | B)> r;                                                                         \
    r.v = val;                                                                               \
    CP_TANGENTS((A | B))                                                                     \
      if constexpr (CpSp<A>::template has<K>() && CpSp<B>::template has<K>())                \
        r.template at<K>() = both;                                                           \
      else if constexpr (CpSp<A>::template has<K>()) r.template at<K>() = first;             \
      else r.template at<K>() = second;                                                      \
    CP_TANGENTS_END;                                                                         \
    return r;                                                                                \
  }
#define CP_DA a.template at<K>()
#define CP_DB b.template at<K>()
CP_SP_BIN(+, a.v + b.v, CP_DA + CP_DB, CP_DA, CP_DB)
CP_SP_BIN(-, a.v - b.v, CP_DA - CP_DB, CP_DA, -CP_DB)
CP_SP_BIN(*, a.v * b.v, fmaf(CP_DA, b.v, a.v * CP_DB), cp_mul_rn(CP_DA, b.v), cp_mul_rn(a.v, CP_DB))
#undef CP_SP_BIN

template <unsigned A, unsigned B>
CP_HD CpSp<(A | B)> operator/(const CpSp<A>& a, const CpSp<B>& b)
{
  CpSp<(A | B)> r;
  const float ib = 1.f / b.v;
  r.v = a.v * ib;
  CP_TANGENTS((A | B))
    if constexpr (CpSp<A>::template has<K>() && CpSp<B>::template has<K>())
      r.template at<K>() = (CP_DA - r.v * CP_DB) * ib;
    else if constexpr (CpSp<A>::template has<K>()) r.template at<K>() = CP_DA * ib;
    else r.template at<K>() = -cp_mul_rn(r.v, CP_DB) * ib;
  CP_TANGENTS_END;
  return r;
}
#undef CP_DB
template <unsigned M> CP_HD CpSp<M> operator+(const CpSp<M>& a, float b) { CpSp<M> r = a; r.v += b; return r; }
template <unsigned M> CP_HD CpSp<M> operator+(float b, const CpSp<M>& a) { return a + b; }
template <unsigned M> CP_HD CpSp<M> operator-(const CpSp<M>& a, float b) { CpSp<M> r = a; r.v -= b; return r; }
template <unsigned M>
CP_HD CpSp<M> operator-(float b, const CpSp<M>& a)
{
  CpSp<M> r;
  r.v = b - a.v;
  CP_TANGENTS(M) r.template at<K>() = -CP_DA; CP_TANGENTS_END;
  return r;
}
template <unsigned M> CP_HD CpSp<M> operator-(const CpSp<M>& a) { return 0.f - a; }
template <unsigned M>
CP_HD CpSp<M> operator*(const CpSp<M>& a, float b)
{
  CpSp<M> r;
  r.v = a.v * b;
  CP_TANGENTS(M) r.template at<K>() = CP_DA * b; CP_TANGENTS_END;
  return r;
}
template <unsigned M> CP_HD CpSp<M> operator*(float b, const CpSp<M>& a) { return a * b; }
template <unsigned M>
CP_HD CpSp<M> operator/(float a, const CpSp<M>& b)
{
  CpSp<0u> c;
  c.v = a;
  return c / b;
}

// f(a) with derivative fp: r = (f(a), fp * a')
template <unsigned M>
CP_HD CpSp<M> cp_dchain(const CpSp<M>& a, float f, float fp)
{
  CpSp<M> r;
  r.v = f;
  CP_TANGENTS(M) r.template at<K>() = fp * CP_DA; CP_TANGENTS_END;
  return r;
}
#undef CP_DA
#undef CP_TANGENTS
#undef CP_TANGENTS_END

template <unsigned M> CP_HD CpSp<M> cp_exp_t(const CpSp<M>& a) { float e = cp_expf(a.v); return cp_dchain(a, e, e); }
template <unsigned M> CP_HD CpSp<M> cp_log_t(const CpSp<M>& a) { return cp_dchain(a, cp_logf(a.v), 1.f / a.v); }
template <unsigned M> CP_HD CpSp<M> cp_expm1_t(const CpSp<M>& a) { return cp_dchain(a, cp_expm1f(a.v), cp_expf(a.v)); }
template <unsigned M>
CP_HD CpSp<M> cp_sqrt_t(const CpSp<M>& a)
{
  float s = cp_sqrtf(a.v);
  return cp_dchain(a, s, s > 0.f ? 0.5f / s : 0.f);
}
template <unsigned M> CP_HD CpSp<M> cp_max0(const CpSp<M>& a) { return a.v > 0.f ? a : a * 0.f; }

// ------------------------------------------------------------------------------------------
// Integrand over dual numbers.
// ------------------------------------------------------------------------------------------
template <class T>
struct CpHadParamsT {
  T lnTauMin;   // ln(4 pTmin^2 / s)
  T kR;         // renormalisation scale factor
  T lnL2[4];    // ln Lambda_nf^2, nf = 3..6
};

// the tangents of the callers' numbers: x0, x1, x2, then alpha_s(mZ), k_ren, the pT_hat cut
template <class T> struct CpTangents;
template <> struct CpTangents<CpDual<3>> { static constexpr unsigned A = 0u, K = 0u, PT = 0u; };
template <> struct CpTangents<CpDual<6>> { static constexpr unsigned A = 8u, K = 16u, PT = 32u; };
#define CP_X0 1u
#define CP_X1 2u
#define CP_X2 4u

template <class T, unsigned M>
CP_HD auto cp_alphas_t(const CpHadParams& P, const CpHadParamsT<T>& Q, const CpSp<M>& Q2in)
{
  CpSp<M> Q2 = Q2in;
  if (Q2.v < P.scale2Min) Q2 = Q2 * 0.f + P.scale2Min;
  const CpSp<M> lnQ2 = cp_log_t(Q2);
  float b0;
  CpSp<CpTangents<T>::A> lnL2;
  if (Q2.v > P.thr2[2] && P.nfmax6) { b0 = 21.f; lnL2 = cp_sp<CpTangents<T>::A>(Q.lnL2[3]); }
  else if (Q2.v > P.thr2[1]) { b0 = 23.f; lnL2 = cp_sp<CpTangents<T>::A>(Q.lnL2[2]); }
  else if (Q2.v > P.thr2[0]) { b0 = 25.f; lnL2 = cp_sp<CpTangents<T>::A>(Q.lnL2[1]); }
  else { b0 = 27.f; lnL2 = cp_sp<CpTangents<T>::A>(Q.lnL2[0]); }
  return (12.f * CP_PI_F / b0) / (lnQ2 - lnL2);
}

template <unsigned M>
CP_HD CpSp<M> cp_poly_t(const CpCteqPoly& c, int f, const CpSp<M>& t)
{
  return (c.co[2][f] * t + c.co[1][f]) * t + c.co[0][f];
}

// the x-dependent quantities of one beam, shared by the 8 parametrisations
template <unsigned M>
struct CpBeamT {
  CpSp<M> x, omx, y, u, x1L, lny;
};

template <unsigned M>
CP_HD CpBeamT<M> cp_beam_t(const CpSp<M>& lnxIn)
{
  // x <= 1 - 1e-10 clamp of PartonDistributions.cc:926 (constant beyond it)
  const CpSp<M> lnx = lnxIn.v > -1e-10f ? lnxIn * 0.f - 1e-10f : lnxIn;
  CpBeamT<M> b;
  b.x = cp_exp_t(lnx);
  b.omx = -cp_expm1_t(lnx);
  b.y = -lnx;
  b.u = lnx + 11.512925465f;
  b.x1L = cp_log_t(b.omx);
  b.lny = cp_log_t(b.y);
  return b;
}

template <unsigned MQ, unsigned MX>
CP_HD CpSp<(MQ | MX)> cp_cteq_answer_t(const CpCteqPoly& c, const CpSp<MQ>& sb1, const CpSp<MQ>& invQ,
                                       const CpBeamT<MX>& b)
{
  const auto& x = b.x;
  const auto& omx = b.omx;
  const auto& u = b.u;
  const auto& x1L = b.x1L;
  const auto A = cp_poly_t(c, CP_CQ_A, sb1), B = cp_poly_t(c, CP_CQ_B, sb1), af1 = cp_poly_t(c, CP_CQ_AF1, sb1);
  const auto af2 = cp_poly_t(c, CP_CQ_AF2, sb1), p = cp_poly_t(c, CP_CQ_P, sb1), af5 = cp_poly_t(c, CP_CQ_AF5, sb1);
  const auto af6 = cp_poly_t(c, CP_CQ_AF6, sb1), af7 = cp_poly_t(c, CP_CQ_AF7, sb1), af8 = cp_poly_t(c, CP_CQ_AF8, sb1);
  const auto ym1 = cp_expm1_t(p * b.lny);
  const auto U = af8 * u + 1.f;
  const auto part3 = x * omx * (af5 + af6 * omx + af7 * x * omx);
  const auto L = c.useX1L ? x1L : cp_log_t(omx + c.eut2);
  const auto e = A + B * x + af1 * af8 * u + af1 * ym1 * U + part3 + c.ut1 * x1L + af2 * L;
  const auto qfac = 1.f - c.qmin * invQ;
  return x * cp_exp_t(e) * qfac;
}

template <unsigned MQ, unsigned MX>
CP_HD void cp_cteq_pair_t(const CpCteqPoly* cteq, CpSp<MQ> Q2, CpSp<MX> lnxA, CpSp<MX> lnxB, CpSp<(MQ | MX)> fa[8],
                          CpSp<(MQ | MX)> fb[8])
{
  if (Q2.v > 1e8f) Q2 = Q2 * 0.f + 1e8f;
  if (Q2.v < 1.f) Q2 = Q2 * 0.f + 1.f;
  const float lnxMin = -13.815510558f;
  if (lnxA.v < lnxMin) lnxA = lnxA * 0.f + lnxMin;
  if (lnxB.v < lnxMin) lnxB = lnxB * 0.f + lnxMin;
  const auto Q = cp_sqrt_t(Q2);
  const auto lnQ = 0.5f * cp_log_t(Q2);
  const auto invQ = 1.f / Q;
  // once per beam rather than once per parametrisation and beam: the same operations on the same
  // values (the host build gives bit-identical results; on the device the compiler may contract a
  // different product into an FMA, a last-bit difference).  12 adjoint passes of 2^22 points:
  // 38.1 -> 33.6 ms
  const auto bA = cp_beam_t(lnxA), bB = cp_beam_t(lnxB);
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const CpCteqPoly& c = cteq[i];
    const auto sb1 = cp_log_t(lnQ - c.lnAlpha) - 1.2f;
    CpSp<(MQ | MX)> ra, rb;
    if (Q.v > c.qlim) {
      ra = cp_cteq_answer_t(c, sb1, invQ, bA);
      rb = cp_cteq_answer_t(c, sb1, invQ, bB);
      if (i != 4) {
        ra = ra * bA.x;
        rb = rb * bB.x;
      }
    } else {
      ra = cp_widen<(MQ | MX)>(sb1 * 0.f);
      rb = cp_widen<(MQ | MX)>(sb1 * 0.f);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k == i) { fa[k] = ra; fb[k] = rb; }
  }
  const auto sa = fa[3], sb = fb[3], ia = 1.f / (fa[4] + 1.f), ib = 1.f / (fb[4] + 1.f);
  const auto ra = fa[4], rb = fb[4];
  fa[3] = sa * ia; fa[4] = sa * ra * ia;
  fb[3] = sb * ib; fb[4] = sb * rb * ib;
#pragma unroll
  for (int k = 0; k < 8; ++k) { fa[k] = cp_max0(fa[k]); fb[k] = cp_max0(fb[k]); }
}

template <unsigned MK, unsigned MF>
CP_HD CpSp<(MK | MF)> cp_channel_sum_t(const CpHadParams& P, const CpSp<MK>& tp, const CpSp<MK>& up,
                                       const CpSp<MF>* A, const CpSp<MF>* Bq)
{
  const auto rt = 1.f / tp, ru = 1.f / up, tu = tp * ru, ut = up * rt;
  const auto sTS = (tp + 1.f) * (tp + 1.f) + (rt + 1.f) * (rt + 1.f) + 1.f;
  const auto sUS = (up + 1.f) * (up + 1.f) + (ru + 1.f) * (ru + 1.f) + 1.f;
  const auto sTU = (tu + 1.f) * (tu + 1.f) + (ut + 1.f) * (ut + 1.f) + 1.f;
  const auto gg2gg = 1.125f * (sTS + sUS + sTU);
  const auto gg2qq = P.nQuarkNew * ((1.f / 6.f) * (ut + tu) - (3.f / 8.f) * (up * up + tp * tp));
  const auto qg2qg = (up * up + 1.f) * (rt * rt) - (4.f / 9.f) * (up + ru);
  const auto qqbar2gg = 0.5f * ((32.f / 27.f) * (ut + tu) - (8.f / 3.f) * (up * up + tp * tp));
  const auto qqT = (4.f / 9.f) * (up * up + 1.f) * (rt * rt);
  const auto qqU = (4.f / 9.f) * (tp * tp + 1.f) * (ru * ru);
  const auto qqTU = -(8.f / 27.f) * (rt * ru);
  const auto qqST = -(8.f / 27.f) * (up * up) * rt;
  const auto QA = A[0] + A[1] + A[3] + A[4] + 2.f * (A[5] + A[6] + A[7]);
  const auto QB = Bq[0] + Bq[1] + Bq[3] + Bq[4] + 2.f * (Bq[5] + Bq[6] + Bq[7]);
  const auto Dsame = A[0] * Bq[0] + A[1] * Bq[1] + A[3] * Bq[3] + A[4] * Bq[4] +
                     2.f * (A[5] * Bq[5] + A[6] * Bq[6] + A[7] * Bq[7]);
  const auto Dopp = A[0] * Bq[4] + A[4] * Bq[0] + A[1] * Bq[3] + A[3] * Bq[1] +
                    2.f * (A[5] * Bq[5] + A[6] * Bq[6] + A[7] * Bq[7]);
  const auto G = A[2] * Bq[2];
  CpSp<(MK | MF)> sum = G * (P.mask[0] * gg2gg + P.mask[1] * gg2qq);
  sum = sum + P.mask[2] * qg2qg * (QA * Bq[2] + A[2] * QB);
  sum = sum + P.mask[3] * (QA * QB * qqT + Dsame * (0.5f * (qqU + qqTU - qqT)) + Dopp * qqST);
  sum = sum + P.mask[4] * Dopp * qqbar2gg;
  return sum;
}

// f * J_base at x, as a function of (x, ln tauMin, k_ren, ln Lambda^2): the plain form of
// cp_had_eval.  Each x_i carries tangent i alone, ln tauMin, k_ren and ln Lambda^2 theirs.
template <class T>
CP_HD T cp_had_weight_t(const CpHadParams& P, const CpHadParamsT<T>& Q, const CpCteqPoly* cteq,
                        const T& x0d, const T& x1d, const T& x2d)
{
  constexpr unsigned PT = CpTangents<T>::PT;
  const auto x0 = cp_sp<CP_X0>(x0d);
  const auto x1 = cp_sp<CP_X1>(x1d);
  const auto x2 = cp_sp<CP_X2>(x2d);
  const auto lnTauMin = cp_sp<PT>(Q.lnTauMin);
  const auto kR = cp_sp<CpTangents<T>::K>(Q.kR);
  const auto lnTau = (1.f - x0) * lnTauMin;
  const auto invTau = cp_exp_t(-lnTau);
  const auto tau = cp_exp_t(lnTau);
  const auto yMax = -0.5f * lnTau;
  const auto a0 = x0 * lnTauMin;
  const auto r = cp_exp_t(a0);
  const auto zMax = cp_sqrt_t(-cp_expm1_t(a0));
  const auto omzMax = r / (zMax + 1.f);
  const auto omz = omzMax + 2.f * zMax * (1.f - x2);
  const auto opz = omzMax + 2.f * zMax * x2;
  const auto tp = -0.5f * omz, up = -0.5f * opz;
  const auto sH = tau * P.s;
  const auto pT2 = 0.25f * sH * omz * opz;
  const auto lnx1 = lnTau * (1.f - x1), lnx2 = lnTau * x1;
  const auto alphaS = cp_alphas_t(P, Q, kR * pT2);
  CpSp<(CP_X0 | CP_X1 | CP_X2 | PT)> fa[8], fb[8];
  cp_cteq_pair_t(cteq, P.kF * pT2, lnx1, lnx2, fa, fb);
  const auto B = cp_channel_sum_t(P, tp, up, fa, fb);
  const auto K0 = (2.f * CP_PI_F * P.conv / P.s) * (-lnTauMin);
  const auto w = K0 * (alphaS * alphaS) * B * yMax * zMax * invTau;
  T out;
  if (!(zMax.v > 0.f)) {
    const auto zero = cp_widen<w.mask>(B * 0.f);
    out.v = zero.v;
    cp_tangents<w.mask>([&](auto k) { out.d[decltype(k)::value] = zero.template at<decltype(k)::value>(); });
    return out;
  }
  out.v = w.v;
  cp_tangents<w.mask>([&](auto k) { out.d[decltype(k)::value] = w.template at<decltype(k)::value>(); });
  return out;
}
#undef CP_X0
#undef CP_X1
#undef CP_X2
