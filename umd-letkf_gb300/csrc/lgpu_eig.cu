// lgpu_eig.cu -- the LETKF transform of every (column, group) unit: FP32 (the
// reference's ssyev precision), with an FP64 form for the units flagged by
// the eigenvalue-gap test or for every unit.
//
// Replaces src/letkf_core.F90:100-141: with A = G + (k-1)/infl I (G from the
// Gram stage, upper triangle as ssyev('V','U') reads it),
//   W    = sqrt(k-1) A^(-1/2)
//   wbar = A^(-1) b           (b = Yb^T R^-1 rho dep, computed in the Gram stage)
//   T    = W + wbar 1^T
// The reference forms both through the eigendecomposition of A.  T is a
// function of the matrix alone, so no eigenvectors are needed:
//   1. Householder tridiagonalisation A = Q S Q^T (Golub & Van Loan, Matrix
//      Computations, 4th ed., Alg. 8.3.1), the reflectors kept in the lower
//      triangle; y = Q^T b along with it.
//   2. S^(-1/2) by partial fractions, x^(-1/2) = sum_p w_p / (x + s_p) with
//      s_p, w_p > 0: the elliptic-function rule of Hale, Higham & Trefethen,
//      "Computing A^alpha, log(A), and related matrix functions by contour
//      integrals" (SIAM J. Numer. Anal. 46(5), 2008, method 3), which is
//      Zolotarev's best approximation on [l0, lmax].  The number of terms
//      follows the condition (4 to 16 in FP32).  Every (S + s_p I)^(-1) comes
//      from one backward pivot recurrence: with eta_j its pivots and
//      rho_j = -e_j / eta_(j+1), the inverse has
//        g_00 = 1/eta_0,  g_(i+1)(i+1) = 1/eta_(i+1) + rho_i^2 g_ii,
//        g_i(j+1) = g_ij rho_j  (j >= i),
//      all terms of the diagonal positive.  One lane runs one shift; a further
//      lane solves S z = y (shift 0), and one checks that S - l0 I is
//      positive definite.
//   3. W = Q S^(-1/2) Q^T and wbar = Q z, the reflectors applied to both
//      sides from the last to the first.
// The three-kernel form before it (reduction, QL on one thread per unit with
// the rotations logged, their replay on Q) spent two thirds of its time in
// the QL's serial recurrence and the replay.
//
// The work matrix lives in registers over a grid of LA x LB lanes: lane
// (a, b) holds rows a + LA r and columns b + LB i.  A reduction step costs
// 3 m^2 multiply-adds for a trailing block of m and a back-transformation
// step K m + K m + m^2; in one row per lane every multiply-add also read a
// quarter of a 16-byte shared-memory vector, and the shared-memory return
// path bounded the reduction.  The 2-D grid reads R + C values per R x C
// multiply-adds.  The steps are unrolled in phases of LA rows so that the
// blocks left of and above the trailing one are dropped at compile time.
#include <type_traits>
#include "lgpu_internal.cuh"
#include <algorithm>
#include <cmath>

namespace lgpu {

namespace {

constexpr int kLevels = 16;   // condition levels 4^1 .. 4^16

// Shifts and weights of the partial fractions on [1, 4^(level + 1)].
template <class R, int NP>
struct Poles {
  int n[kLevels];
  R s[kLevels][NP], w[kLevels][NP];
};

// Jacobi's elliptic functions of parameter 1 - m1 by the arithmetic-geometric
// mean (Abramowitz & Stegun 17.6, 16.4): the quarter period K, and sn / cn at u
// in (0, K) as the tangent of the amplitude, which is halved down the scale.
struct Elliptic {
  double agm = 1.0, ratio[32], K;   // the mean, half differences over means on the way to it
  int steps = 0;
  explicit Elliptic(double m1) {
    double b = std::sqrt(m1);
    while (agm - b > 1e-16 * agm && steps < 32) {
      const double mean = 0.5 * (agm + b);
      ratio[steps++] = 0.5 * (agm - b) / mean;
      b = std::sqrt(agm * b);
      agm = mean;
    }
    K = 1.5707963267948966 / agm;
  }
  double sc(double u) const {
    double phi = std::ldexp(agm * u, steps);
    for (int i = steps; i-- > 0;) phi = 0.5 * (phi + std::asin(ratio[i] * std::sin(phi)));
    return std::tan(phi);
  }
};

// Smallest term counts whose error over [1, 4^(level + 1)] is below `tol`
// (NP at most: the wide levels, whose condition leaves the working precision
// no digits at the small end anyway, keep the error NP terms give).
template <class R, int NP>
Poles<R, NP> make_poles(double tol) {
  Poles<R, NP> P{};
  for (int l = 0; l < kLevels; l++) {
    const double kappa = std::ldexp(1.0, 2 * (l + 1)), m1 = 1.0 / kappa;
    const Elliptic E(m1);
    double s[NP], w[NP];
    for (int n = 3; n <= NP; n++) {
      for (int j = 0; j < n; j++) {
        // t = sn / cn: 1 / cn^2 = 1 + t^2, dn^2 / cn^2 = 1 + m1 t^2
        const double t = E.sc((j + 0.5) * E.K / n), t2 = t * t;
        s[j] = t2;
        w[j] = 2.0 * E.K / (3.14159265358979323846 * n) * std::sqrt((1.0 + t2) * (1.0 + m1 * t2));
      }
      double err = 0.0;
      for (int t = 0; t <= 400; t++) {
        const double x = std::exp(std::log(kappa) * t / 400.0);
        double f = 0.0;
        for (int j = 0; j < n; j++) f += w[j] / (x + s[j]);
        err = std::max(err, std::fabs(f * std::sqrt(x) - 1.0));
      }
      P.n[l] = n;
      if (err <= tol) break;
    }
    for (int j = 0; j < P.n[l]; j++) { P.s[l][j] = (R)s[j]; P.w[l][j] = (R)w[j]; }
  }
  return P;
}

using PolesF = Poles<float, 16>;
using PolesD = Poles<double, 32>;
// a quarter of the working precision's unit roundoff (FP64: what 32 terms and
// the evaluation in double reach)
const PolesF &poles_f() { static const PolesF P = make_poles<float, 16>(1.5e-8); return P; }
const PolesD &poles_d() { static const PolesD P = make_poles<double, 32>(2e-15); return P; }
template <class R> struct PolesOf;
template <> struct PolesOf<float> { using type = PolesF; static const PolesF &get() { return poles_f(); } };
template <> struct PolesOf<double> { using type = PolesD; static const PolesD &get() { return poles_d(); } };

__device__ __forceinline__ float fmar(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmar(double a, double b, double c) { return __fma_rn(a, b, c); }
// the smallest scale treated as zero, per precision
template <class R> struct Lim;
// (`zero`: a squared norm that no rounding of the diagonal, at least 1, can see)
template <> struct Lim<float> {
  static constexpr float tiny = 1e-30f, zero = 1e-34f;
};
template <> struct Lim<double> {
  static constexpr double tiny = 1e-300, zero = 1e-200;
};

// Two values of neighbouring lane columns.  FP32: a register pair for the
// packed multiply-add, which does both in one issue slot.
template <class R> struct Pair;
template <>
struct Pair<float> : F2 {
  __device__ __forceinline__ Pair() {}
  __device__ __forceinline__ Pair(F2 v) : F2(v) {}
  __device__ __forceinline__ Pair(float x, float y) : F2(x, y) {}
};
template <>
struct Pair<double> {
  double a, b;
  __device__ __forceinline__ Pair() {}
  __device__ __forceinline__ Pair(double x, double y) : a(x), b(y) {}
  __device__ __forceinline__ double x() const { return a; }
  __device__ __forceinline__ double y() const { return b; }
};
__device__ __forceinline__ Pair<float> pfma(Pair<float> a, Pair<float> b, Pair<float> c) { return f2_fma(a, b, c); }
__device__ __forceinline__ Pair<double> pfma(Pair<double> a, Pair<double> b, Pair<double> c) {
  return Pair<double>(__fma_rn(a.a, b.a, c.a), __fma_rn(a.b, b.b, c.b));
}
__device__ __forceinline__ Pair<float> padd(Pair<float> a, Pair<float> b) { return f2_add(a, b); }
__device__ __forceinline__ Pair<double> padd(Pair<double> a, Pair<double> b) { return Pair<double>(a.a + b.a, a.b + b.b); }

// the element of lane column i (a constant after unrolling) of a row of pairs
template <class R>
__device__ __forceinline__ R get(const Pair<R> *p, int i) { return i & 1 ? p[i / 2].y() : p[i / 2].x(); }
template <class R>
__device__ __forceinline__ void set(Pair<R> *p, int i, R v) {
  p[i / 2] = i & 1 ? Pair<R>(p[i / 2].x(), v) : Pair<R>(v, p[i / 2].y());
}

// two pairs, 16-byte aligned in FP32
__device__ __forceinline__ void ld2(const float *p, Pair<float> *v) { f2_load2(p, v[0], v[1]); }
__device__ __forceinline__ void ld2(const double *p, Pair<double> *v) {
  const double2 t = *reinterpret_cast<const double2 *>(p), u = *reinterpret_cast<const double2 *>(p + 2);
  v[0] = Pair<double>(t.x, t.y);
  v[1] = Pair<double>(u.x, u.y);
}
__device__ __forceinline__ void st2(float *p, Pair<float> a, Pair<float> b) { f2_store2(p, a, b); }
__device__ __forceinline__ void st2(double *p, Pair<double> a, Pair<double> b) {
  *reinterpret_cast<double2 *>(p) = make_double2(a.a, a.b);
  *reinterpret_cast<double2 *>(p + 2) = make_double2(b.a, b.b);
}

// sqrt and reciprocal of positive normal values (FP32: within an ulp,
// lgpu_f32x2.cuh; the FP64 overloads would hide these without the declarations)
using lgpu::rcp_pos;
using lgpu::sqrt_pos;
__device__ __forceinline__ double sqrt_pos(double x) { return sqrt(x); }
__device__ __forceinline__ double rcp_pos(double x) { return __drcp_rn(x); }
static_assert(std::is_same<decltype(sqrt_pos(1.0f)), float>::value && std::is_same<decltype(rcp_pos(1.0f)), float>::value,
              "FP32 roots stay FP32");

// 16 bytes global -> shared, asynchronously
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The lane grid of one unit: RN rows and CN columns per lane; LA is a
// multiple of LB, and LB <= 8 divides a warp, so the lanes of a row lie in one warp.
template <class R_, int RN_, int CN_, int LA_, int LB_, int MB_>
struct Grid {
  using R = R_;
  static constexpr int RN = RN_, CN = CN_, LA = LA_, LB = LB_;
  static constexpr int MB = MB_;                            // blocks per SM the registers are bounded for
  static constexpr int L = LA * LB;
  static constexpr int CH2 = CN / 2;                        // column pairs per lane
  using Row = Pair<R>[CN / 2];
  static constexpr int KR = LA * RN, KC = LB * CN;          // covered rows, columns
  // values of one lane column: whole 16-byte vectors, one more where the lane
  // columns' vectors would start in the same banks
  static constexpr int CP4 = (CN + 3) / 4 * 4;
  static constexpr int CP = LB > 1 && CP4 % (64 / LB) == 0 ? CP4 + 4 : CP4;
  static constexpr int NV = (CN + 3) / 4;                   // vectors of a lane's column pairs (CP may hold one more)
  static_assert(2 * (NV - 1) < CH2, "every vector holds a column pair of the lane");
  static constexpr int VB = LB * CP;                        // one column-ordered vector
  static constexpr int NP = sizeof(R) == 4 ? 16 : 32;
  static constexpr int KM = KR > KC ? KR : KC;
  static constexpr int KN = (KM + 3) / 4 * 4;               // one naturally ordered vector
  // one shift's arrays: rho (8 zeros of slack), g, LB-products; the lanes'
  // arrays start a 16-byte bank group apart
  static constexpr int PS = (2 * KN + 8 + VB + 27) / 32 * 32 + 4;
  static constexpr int VEC = 4 * KN;                        // d, e, tau, z
  static constexpr int STEP = 6 * VB;                       // reduction: x, v, w (double-buffered); back: w, ring of 4 v
  static constexpr int CH = L >= 32 ? NP : L - 2;           // shifts of one pass: with the solve and the test, a lane each
  static constexpr int POLE = (CH + 2) * PS;
  static constexpr int TRANS = LA * VB;                     // one row group
  static constexpr int PACK = KC * (KC + 3) / 2;            // the packed Gram block
  static constexpr int WORK0 = STEP > POLE ? STEP : POLE, WORK1 = WORK0 > TRANS ? WORK0 : TRANS;
  static constexpr int UNIT0 = VEC + (WORK1 > PACK ? WORK1 : PACK);
  // values of one unit: 8 past a multiple of 32, so that the units of a warp
  // read different banks
  static constexpr int UNIT = (UNIT0 + 23) / 32 * 32 + 8;
  static constexpr int REFL = KC * VB;                      // the reflectors of one unit (global scratch)
  static constexpr int UPW = L < 32 ? 32 / L : 1;           // units per warp
  static constexpr int UPB = L <= 32 ? 4 * UPW : 1;         // units per block
  static constexpr int THREADS = L <= 32 ? 128 : L;
  static_assert(LA % LB == 0 && LB <= 8 && CN % 2 == 0, "lane grid");
  static_assert(KR / LB <= CP && KR >= KC && (L > 32 || KR == KC), "every row has a place in a column-ordered vector");
};

template <class G>
__device__ __forceinline__ void team_sync() {
  if constexpr (G::L <= 32) __syncwarp();
  else __syncthreads();
}

// sum over the lanes of a row (consecutive lanes)
template <class G, class R>
__device__ __forceinline__ R sum_b(R v) {
#pragma unroll
  for (int o = 1; o < G::LB; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// position of row / column c in a column-ordered vector (lane column c % LB first)
template <class G>
__device__ __forceinline__ int vpos(int c) { return (c % G::LB) * G::CP + c / G::LB; }

// the lane's column pairs q >= Q0 of a column-ordered vector
template <class G, int Q0, class R>
__device__ __forceinline__ void load_cols(const R *buf, int b, Pair<R> *v) {
  const R *p = buf + b * G::CP;
#pragma unroll
  for (int q = Q0 / 2; q < G::NV; q++) {
    Pair<R> t[2];
    ld2(p + 4 * q, t);
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (2 * q + j >= Q0 && 2 * q + j < G::CH2) v[2 * q + j] = t[j];
  }
}

// the lane's rows r >= R0 of a column-ordered vector: row a + LA r sits at
// lane column a % LB, place a / LB + (LA / LB) r
template <class G, int R0, class R>
__device__ __forceinline__ void load_rows(const R *buf, int a, R *v) {
  const R *p = buf + (a % G::LB) * G::CP + a / G::LB;
#pragma unroll
  for (int r = R0; r < G::RN; r++) v[r] = p[(G::LA / G::LB) * r];
}

template <class G, int R0, class R>
__device__ __forceinline__ void store_rows(R *buf, int a, const R *v) {
  R *p = buf + (a % G::LB) * G::CP + a / G::LB;
#pragma unroll
  for (int r = R0; r < G::RN; r++) p[(G::LA / G::LB) * r] = v[r];
}

// the lane's column pairs into a column-ordered vector, from the 16-byte group
// of pair Q0 on
template <class G, int Q0, class R>
__device__ __forceinline__ void store_cols(R *buf, int b, const Pair<R> *v) {
  R *p = buf + b * G::CP;
#pragma unroll
  for (int q = Q0 / 2; q < G::NV; q++)
    st2(p + 4 * q, v[2 * q], 2 * q + 1 < G::CH2 ? v[2 * q + 1] : Pair<R>(R(0), R(0)));
}

// the unit's shared-memory vectors
template <class G>
struct UnitMem {
  using R = typename G::R;
  R *d, *e, *tau, *z, *work;
  __device__ explicit UnitMem(R *base) {
    d = base;
    e = d + G::KN; tau = e + G::KN; z = tau + G::KN;
    work = z + G::KN;
  }
  __device__ R *w(int j) const { return work + (j & 1) * G::VB; }
  __device__ R *x(int j) const { return work + (2 + (j & 1)) * G::VB; }     // reduction: raw row
  __device__ R *v(int j) const { return work + (4 + (j & 1)) * G::VB; }     // reduction: reflector
  __device__ R *ring(int j) const { return work + (2 + (j & 3)) * G::VB; }  // back-transformation: reflectors
};

// The right-hand side (then z) of a unit on one warp: one warp's lanes hold
// elements l + S q, in registers; a team keeps them in shared memory.
template <class G>
struct Vec {
  using R = typename G::R;
  static constexpr int S = G::L < 32 ? G::L : 32, Q = (G::KM + S - 1) / S;
  R z[Q];
  __device__ __forceinline__ void load(const UnitMem<G> &U, int l) {
    if constexpr (G::L <= 32) {
#pragma unroll
      for (int q = 0; q < Q; q++) z[q] = l + S * q < G::KN ? U.z[l + S * q] : R(0);
    }
  }
  __device__ __forceinline__ void store(const UnitMem<G> &U, int l) {
    if constexpr (G::L <= 32) {
#pragma unroll
      for (int q = 0; q < Q; q++)
        if (l + S * q < G::KN) U.z[l + S * q] = z[q];
    }
  }
  // z -= t (v.z) v, v column-ordered and zero before C0; a team's warp `warp` does it
  template <int C0>
  __device__ __forceinline__ void reflect(const UnitMem<G> &U, int k, int l, int warp, R t, const R *vbuf) {
    if constexpr (G::L > 32) {
      if ((l >> 5) != warp) return;
      l &= 31;
    }
    R v[Q], s = R(0);
#pragma unroll
    for (int q = C0 / S; q < Q; q++) {
      const int c = l + S * q;
      v[q] = (q > C0 / S || c >= C0) && (q < Q - 1 || c < G::KC) ? vbuf[vpos<G>(c)] : R(0);
      if constexpr (G::L > 32) z[q] = c < k ? U.z[c] : R(0);
      s = fmar(v[q], z[q], s);
    }
#pragma unroll
    for (int o = 1; o < S; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s *= t;
#pragma unroll
    for (int q = C0 / S; q < Q; q++) {
      z[q] = fmar(-s, v[q], z[q]);
      if constexpr (G::L > 32)
        if (l + S * q < k) U.z[l + S * q] = z[q];
    }
  }
};

// The two-sided update M -= v w^T + w v^T with w = p - (t/2)(p.v) v, p = t M v.
// vcol / vrow: the reflector at the lane's column pairs from Q0 and rows from
// R0, zero up to j.  FULL (back-transformation): every row and column; else
// (reduction) the trailing block, where w is zero up to j.
template <class G, int R0, int Q0, bool FULL>
__device__ __forceinline__ void two_sided(typename G::Row (&A)[G::RN], typename G::R *wb, int j, int a, int b,
                                          typename G::R t, const Pair<typename G::R> *vcol, const typename G::R *vrow) {
  using R = typename G::R;
  using P2 = Pair<R>;
  constexpr int W0 = FULL ? 0 : R0, C0 = FULL ? 0 : Q0;
  R w[G::RN];
#pragma unroll
  for (int r = W0; r < G::RN; r++) {
    P2 acc(R(0), R(0));
#pragma unroll
    for (int q = Q0; q < G::CH2; q++) acc = pfma(A[r][q], vcol[q], acc);
    w[r] = acc.x() + acc.y();
  }
#pragma unroll
  for (int r = W0; r < G::RN; r++) w[r] = t * sum_b<G>(w[r]);
  if constexpr (G::L <= 32) {
    // one warp: p.v over the rows, then the finished w is published
    R pv = R(0);
#pragma unroll
    for (int r = R0; r < G::RN; r++) pv = fmar(w[r], vrow[r], pv);
#pragma unroll
    for (int o = G::LB; o < G::L; o <<= 1) pv += __shfl_xor_sync(0xffffffffu, pv, o);
    const R beta = R(0.5) * t * pv;
#pragma unroll
    for (int r = R0; r < G::RN; r++) w[r] = fmar(-beta, vrow[r], w[r]);
    if (!FULL) w[R0] = a + G::LA * R0 > j ? w[R0] : R(0);
    if (b == 0) store_rows<G, W0>(wb, a, w);
    team_sync<G>();
    P2 nw[G::RN], nv[G::RN];
#pragma unroll
    for (int r = W0; r < G::RN; r++) {
      nw[r] = P2(-w[r], -w[r]);
      if (r >= R0) nv[r] = P2(-vrow[r], -vrow[r]);
    }
    const R *wp = wb + b * G::CP;
#pragma unroll
    for (int q = C0 / 2; q < G::NV; q++) {
      P2 wc[2];
      ld2(wp + 4 * q, wc);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = 2 * q + h;
        if (i < C0 || i >= G::CH2) continue;
#pragma unroll
        for (int r = W0; r < G::RN; r++) {
          P2 x = A[r][i];
          if (i >= Q0) x = pfma(nw[r], vcol[i], x);
          if (r >= R0) x = pfma(nv[r], wc[h], x);
          A[r][i] = x;
        }
      }
    }
  } else {
    // a team of warps: p is published, and p.v is summed over the columns,
    // whose lanes share a warp
    if (!FULL) w[R0] = a + G::LA * R0 > j ? w[R0] : R(0);
    if (b == 0) store_rows<G, W0>(wb, a, w);
    team_sync<G>();
    P2 wc[G::CH2], pv(R(0), R(0));
    load_cols<G, C0>(wb, b, wc);
#pragma unroll
    for (int q = Q0; q < G::CH2; q++) pv = pfma(wc[q], vcol[q], pv);
    const R beta = R(0.5) * t * sum_b<G>(pv.x() + pv.y());
    const P2 nb(-beta, -beta);
#pragma unroll
    for (int q = Q0; q < G::CH2; q++) wc[q] = pfma(nb, vcol[q], wc[q]);
#pragma unroll
    for (int r = R0; r < G::RN; r++) w[r] = fmar(-beta, vrow[r], w[r]);
#pragma unroll
    for (int r = W0; r < G::RN; r++) {
      const P2 nw(-w[r], -w[r]), nv(r >= R0 ? -vrow[r] : R(0), r >= R0 ? -vrow[r] : R(0));
#pragma unroll
      for (int q = C0; q < G::CH2; q++) {
        P2 x = A[r][q];
        if (q >= Q0) x = pfma(nw, vcol[q], x);
        if (r >= R0) x = pfma(nv, wc[q], x);
        A[r][q] = x;
      }
    }
  }
}

// alpha = -sign(x0) |x| and t = 2 / v^T v of v = x - alpha e_1 (t = 0, alpha =
// x0: x is e_1's multiple to the last bit)
template <class R>
__device__ __forceinline__ void reflector(bool on, R s1, R x0, R &alpha, R &t) {
  const R sig = fmar(x0, x0, s1);
  const bool live = on && s1 > Lim<R>::tiny * sig && sig > Lim<R>::zero;
  const R root = -copysign(sqrt_pos(sig), x0);
  const R rt = rcp_pos(fmar(-root, x0, sig));
  alpha = live ? root : x0;
  t = live ? rt : R(0);
}

// Reduction steps of rows [LA P, LA P + LA): d, e, tau, the reflectors to the
// scratch gv (one column-ordered vector a step), y = Q^T b.
template <class G, int P>
__device__ __forceinline__ void reduce_phase(typename G::Row (&A)[G::RN], const UnitMem<G> &U, Vec<G> &z,
                                             typename G::R *gv, int k, int l, int a, int b) {
  using R = typename G::R;
  constexpr int R0 = P, I0 = (P * G::LA + 1) / G::LB, Q0 = I0 / 2;
  constexpr int CB = P * G::LA / G::LB;                       // column group of column LA P
  constexpr int NB = G::LA / G::LB;                           // column groups of the phase's columns
  const int jend = k < P * G::LA + G::LA ? k : P * G::LA + G::LA;
  R tp = R(0);
#pragma unroll 1
  for (int j = P * G::LA; j < jend; j++) {
    const bool own = a == j - P * G::LA;
    Pair<R> vcol[G::CH2];
    R vrow[G::RN], t = R(0);
    if constexpr (G::L <= 32) {
      // one warp: the row is published as it stands, and every lane forms the
      // reflector from its own columns; the right-hand side takes the
      // reflector of the step before meanwhile
      R *xb = U.x(j), *vb = U.v(j);
      if (own) store_cols<G, CB / 2>(xb, b, A[R0]);
      team_sync<G>();
      const R x0 = j + 1 < G::KC ? xb[vpos<G>(j + 1)] : R(0);
      if (j >= k - 2) {                        // the last 2 x 2 block
        if (l == 0) { U.d[j] = xb[vpos<G>(j)]; U.e[j] = j < k - 1 ? x0 : R(0); }
        continue;
      }
      load_cols<G, Q0>(xb, b, vcol);
      load_rows<G, R0>(xb, a, vrow);
      if (j > P * G::LA) z.template reflect<P * G::LA>(U, k, l, 0, tp, U.v(j - 1));
#pragma unroll
      for (int i = 2 * Q0; i < G::CN; i++)
        if (i <= CB + NB) set(vcol, i, b + G::LB * i > j + 1 ? get(vcol, i) : R(0));
      Pair<R> s2[2] = {Pair<R>(R(0), R(0)), Pair<R>(R(0), R(0))};
#pragma unroll
      for (int q = Q0; q < G::CH2; q++) s2[q & 1] = pfma(vcol[q], vcol[q], s2[q & 1]);
      R alpha;
      reflector(true, sum_b<G>((s2[0].x() + s2[0].y()) + (s2[1].x() + s2[1].y())), x0, alpha, t);
      const R v0 = x0 - alpha;
#pragma unroll
      for (int i = 2 * Q0; i < G::CN; i++)
        if (i <= CB + NB) set(vcol, i, b + G::LB * i == j + 1 ? v0 : get(vcol, i));
#pragma unroll
      for (int r = R0; r < G::RN; r++)
        if (r <= R0 + 1) {
          const int row = a + G::LA * r;
          vrow[r] = row > j + 1 ? vrow[r] : (row == j + 1 ? v0 : R(0));
        }
      if (own) {
        if (Q0 > CB / 2) vcol[CB / 2] = Pair<R>(R(0), R(0));
        store_cols<G, CB / 2>(vb, b, vcol);
        store_cols<G, CB / 2>(gv + (size_t)j * G::VB, b, vcol);
      }
      if (l == 0) { U.tau[j] = t; U.e[j] = alpha; U.d[j] = xb[vpos<G>(j)]; }
    } else {
      // a team: the warp of the row forms the reflector and publishes it
      R *vb = U.v(j);
      if ((l >> 5) == (j - P * G::LA) * G::LB / 32) {
        R x0 = R(0), dj = R(0);
        Pair<R> x[G::CH2], s2(R(0), R(0));
#pragma unroll
        for (int q = CB / 2; q < G::CH2; q++) x[q] = A[R0][q];
#pragma unroll
        for (int i = CB / 2 * 2; i < G::CN; i++)
          if (i <= CB + NB) {
            const int c = b + G::LB * i;
            const R xi = get(x, i);
            if (c == j + 1) x0 = xi;
            if (c == j) dj = xi;
            set(x, i, c > j + 1 ? xi : R(0));
          }
#pragma unroll
        for (int q = CB / 2; q < G::CH2; q++) s2 = pfma(x[q], x[q], s2);
        R alpha;
        x0 = sum_b<G>(x0);
        reflector(j < k - 2, sum_b<G>(s2.x() + s2.y()), x0, alpha, t);
        const R v0 = x0 - alpha;
        if (own) {
#pragma unroll
          for (int i = CB / 2 * 2; i < G::CN; i++)
            if (i <= CB + NB) set(x, i, b + G::LB * i == j + 1 ? v0 : get(x, i));
          store_cols<G, CB / 2>(vb, b, x);
          store_cols<G, CB / 2>(gv + (size_t)j * G::VB, b, x);
          if (b == 0) { U.tau[j] = t; U.e[j] = alpha; }
          if (b == j % G::LB) U.d[j] = dj;
        }
      }
      if (j >= k - 2) continue;
      team_sync<G>();
      t = U.tau[j];
      load_cols<G, Q0>(vb, b, vcol);
      load_rows<G, R0>(vb, a, vrow);
    }
    two_sided<G, R0, Q0, false>(A, U.w(j), j, a, b, t, vcol, vrow);
    if constexpr (G::L > 32)
      z.template reflect<P * G::LA>(U, k, l, ((j - P * G::LA) * G::LB / 32 + G::L / 64) % (G::L / 32), t, U.v(j));
    tp = t;
  }
  if constexpr (G::L <= 32) {
    // the phase's last reflector
    const int jl = jend - 1 < k - 3 ? jend - 1 : k - 3;
    if (jl >= P * G::LA) z.template reflect<P * G::LA>(U, k, l, 0, tp, U.v(jl));
  }
}

// the reflector of step j into its ring slot
template <class G>
__device__ __forceinline__ void fetch_reflector(const UnitMem<G> &U, const typename G::R *gv, int j, int l) {
  using R = typename G::R;
  constexpr int E = 16 / (int)sizeof(R);
  if (j >= 0)
    for (int c = l; c < G::VB / E; c += G::L) copy16_async(U.ring(j) + c * E, gv + (size_t)j * G::VB + c * E);
  copy_commit();
}

// Back-transformation steps of columns [LA P, LA P + LA), last first:
// M <- H_j M H_j and z <- H_j z.
template <class G, int P>
__device__ __forceinline__ void back_phase(typename G::Row (&A)[G::RN], const UnitMem<G> &U, Vec<G> &z,
                                           const typename G::R *gv, int k, int l, int a, int b) {
  using R = typename G::R;
  constexpr int R0 = P, Q0 = (P * G::LA + 1) / G::LB / 2;
  const int jtop = k - 3 < P * G::LA + G::LA - 1 ? k - 3 : P * G::LA + G::LA - 1;
#pragma unroll 1
  for (int j = jtop; j >= P * G::LA; j--) {
    copy_wait<2>();
    team_sync<G>();
    fetch_reflector<G>(U, gv, j - 3, l);       // into the slot of step j + 1, which every lane has left
    const R *vb = U.ring(j);
    const R t = U.tau[j];
    Pair<R> vcol[G::CH2];
    R vrow[G::RN];
    load_cols<G, Q0>(vb, b, vcol);
    load_rows<G, R0>(vb, a, vrow);
    if constexpr (G::L <= 32) z.template reflect<P * G::LA>(U, k, l, 0, t, vb);
    two_sided<G, R0, Q0, true>(A, U.w(j), j, a, b, t, vcol, vrow);
    if constexpr (G::L > 32) z.template reflect<P * G::LA>(U, k, l, j % (G::L / 32), t, vb);
  }
}

template <class G, int P>
__device__ __forceinline__ void reduce_all(typename G::Row (&A)[G::RN], const UnitMem<G> &U, Vec<G> &z,
                                           typename G::R *gv, int k, int l, int a, int b) {
  if constexpr (P < G::RN) {
    reduce_phase<G, P>(A, U, z, gv, k, l, a, b);
    reduce_all<G, P + 1>(A, U, z, gv, k, l, a, b);
  }
}

template <class G, int P>
__device__ __forceinline__ void back_all(typename G::Row (&A)[G::RN], const UnitMem<G> &U, Vec<G> &z,
                                         const typename G::R *gv, int k, int l, int a, int b) {
  if constexpr (P >= 0) {
    back_phase<G, P>(A, U, z, gv, k, l, a, b);
    back_all<G, P - 1>(A, U, z, gv, k, l, a, b);
  }
}

// M's lower triangle from its upper one, one row group at a time through
// shared memory
template <class G, int P>
__device__ __forceinline__ void mirror_all(typename G::Row (&A)[G::RN], typename G::R *buf, int a, int b) {
  if constexpr (P < G::RN) {
    constexpr int CB = P * G::LA / G::LB, NB = G::LA / G::LB;
    team_sync<G>();
    store_cols<G, CB / 2>(buf + a * G::VB, b, A[P]);
    team_sync<G>();
#pragma unroll
    for (int i = CB; i < CB + NB && i < G::CN; i++) {
      typename G::R s[G::RN];
      load_rows<G, P>(buf + (b + G::LB * (i - CB)) * G::VB, a, s);
#pragma unroll
      for (int r = P; r < G::RN; r++)
        set(A[r], i, r > P || a + G::LA * r > b + G::LB * i ? s[r] : get(A[r], i));
    }
    mirror_all<G, P + 1>(A, buf, a, b);
  }
}

// any lane of the unit
template <class G>
__device__ __forceinline__ bool unit_any(bool x) {
  if constexpr (G::L <= 32) {
    const unsigned m = G::L == 32 ? 0xffffffffu : ((1u << (G::L & 31)) - 1u) << ((threadIdx.x & 31) / G::L * G::L);
    return (__ballot_sync(0xffffffffu, x) & m) != 0;
  } else {
    return __syncthreads_or(x) != 0;
  }
}

// One unit's transform from its packed Gram block (null: a lane slot without a
// unit; it runs along on A = I).  Returns status bits (1: non-finite, 2: not
// positive definite).
template <class G>
__device__ __forceinline__ int unit_transform(typename G::R *mem, const typename PolesOf<typename G::R>::type &tab,
                                              typename G::R *gv, int k, float infl, const float *Gin, float *Tout,
                                              float *wout, float *de, int l) {
  using R = typename G::R;
  const UnitMem<G> U(mem);
  const int a = l / G::LB, b = l % G::LB;
  // ---- A = G + (k-1)/infl I, src/letkf_core.F90:101-104
  const R shift = (R)(k - 1) * R(1) / (R)infl;
  typename G::Row A[G::RN];
  float *gs = reinterpret_cast<float *>(U.work);
  if (Gin) {
    // the packed block through shared memory, in order
    const int nf = packed_size(k);
#pragma unroll 8
    for (int f = l; f < nf; f += G::L) gs[f] = Gin[f];
  }
  team_sync<G>();
#pragma unroll
  for (int r = 0; r < G::RN; r++) {
    const int row = a + G::LA * r, ro = tri_off(row, k) - row;
#pragma unroll
    for (int i = 0; i < G::CN; i++) {
      const int col = b + G::LB * i;
      R v = R(0);
      if (row < k && col < k) {
        if (Gin) v = (R)gs[row < col ? ro + col : tri_off(col, k) - col + row];
        if (row == col) v += shift;
      }
      set(A[r], i, v);
    }
  }
  for (int c = l; c < G::KN; c += G::L) {
    U.z[c] = Gin && c < k ? (R)gs[k * (k + 1) / 2 + c] : R(0);
    U.d[c] = R(1);
    U.e[c] = R(0);
    U.tau[c] = R(0);
  }
  team_sync<G>();
  Vec<G> z;
  z.load(U, l);
  reduce_all<G, 0>(A, U, z, gv, k, l, a, b);
  z.store(U, l);
  team_sync<G>();
  if (de) {
    for (int c = l; c < k; c += G::L) { de[c] = (float)U.d[c]; de[k + c] = (float)U.e[c]; }
  }
  // ---- S^(-1/2) by partial fractions
  constexpr int S = G::L < 32 ? G::L : 32;
  R lmax = R(0);
  for (int c = l % S; c < k; c += S) {
    const R g = U.d[c] + fabs(U.e[c]) + (c > 0 ? fabs(U.e[c - 1]) : R(0));
    lmax = fabs(g) < R(3e38) ? fmax(lmax, g) : R(INFINITY);
  }
#pragma unroll
  for (int o = 1; o < S; o <<= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
  const bool nan = !(lmax < R(3e38));
  // l0 bounds the spectrum from below unless the input is no Gram matrix or
  // its condition is beyond the working precision: then lower bounds are
  // tried, down to the last level
  R l0 = R(0.9) * shift;
  int level = 0, np = 0;
  bool bad = false;
#pragma unroll
  for (int r = 0; r < G::RN; r++)
#pragma unroll
    for (int i = G::LA * r / G::LB; i < G::CN; i++)
      set(A[r], i, b + G::LB * i >= a + G::LA * r ? R(0) : get(A[r], i));
  for (int p0 = 0;;) {
    if (p0 == 0) {
      level = nan ? 0 : ilogb((double)fmax(lmax / l0, R(1))) >> 1;
      level = level < kLevels - 1 ? level : kLevels - 1;
      np = tab.n[level];
    }
    const int nc = np - p0 < G::CH ? np - p0 : G::CH;
    // one lane a shift: the pivots from the last row up (u = 1, or the
    // right-hand side of S z = y), then the diagonal of the inverse (or z)
    // down, and the products of LB consecutive ratios.  Slot CH solves
    // S z = y, slot CH + 1 tests S - 0.999 l0 I (both in the first pass).
    bool fail = false, neg0 = false;
    const int jobs = p0 == 0 ? nc + 2 : nc;
    for (int q = l; q < jobs; q += G::L) {
      const bool solve = q == nc, test = q == nc + 1;
      const R s = solve ? R(0) : (test ? R(-0.999) * l0 : l0 * tab.s[level][p0 + (q < nc ? q : 0)]);
      R *rho = U.work + (q < nc ? q : G::CH + q - nc) * G::PS, *g = rho + G::KN + 8, *lp = g + G::KN;
#pragma unroll
      for (int t = 0; t < 8; t++) rho[G::KM - 1 + t] = R(0);
      R eta = U.d[G::KM - 1] + s, inv = rcp_pos(eta), u = solve ? U.z[G::KM - 1] : R(1);
      bool neg = k == G::KM && !(eta > R(0));
      g[G::KM - 1] = u * inv;
#pragma unroll 4
      for (int j = G::KM - 2; j >= 0; j--) {
        const R ej = U.e[j], rj = -ej * inv;
        rho[j] = rj;
        eta = fmar(ej, rj, U.d[j] + s);
        neg |= j < k && !(eta > R(0));
        inv = rcp_pos(eta);
        u = solve ? fmar(rj, u, U.z[j]) : R(1);
        g[j] = u * inv;
      }
      R gi = g[0];
      R win[G::LB];
#pragma unroll
      for (int t = 0; t < G::LB; t++) win[t] = R(0);
      lp[0] = R(0);
#pragma unroll 4
      for (int j = 0; j < G::KM - 1; j++) {
        const R rj = rho[j];
        gi = fmar(solve ? rj : rj * rj, gi, g[j + 1]);
        g[j + 1] = gi;
#pragma unroll
        for (int t = 0; t + 1 < G::LB; t++) win[t] = win[t + 1];
        win[G::LB - 1] = rj;
        R pr = win[0];
#pragma unroll
        for (int t = 1; t < G::LB; t++) pr *= win[t];
        if (j + 1 < G::KC) lp[vpos<G>(j + 1)] = pr;
      }
      fail |= test && neg;
      neg0 |= solve && neg;
    }
    if (p0 == 0) {
      fail = unit_any<G>(fail) && level < kLevels - 1 && !nan;
      bad = unit_any<G>(neg0);
      // every lane of the warp (team) starts over together
      if (G::L < 32 ? __any_sync(0xffffffffu, fail) : fail) {
        if (fail) l0 *= R(1.0 / 16.0);
        team_sync<G>();
        continue;
      }
    }
    team_sync<G>();
    // the upper triangle of sqrt(k-1) S^(-1/2)
    const R scale = sqrt(l0 * (R)(k - 1));
#pragma unroll 1
    for (int q = 0; q < nc; q++) {
      const R wp = scale * tab.w[level][p0 + q];
      const R *rho = U.work + q * G::PS, *g = rho + G::KN + 8, *lp = g + G::KN;
      Pair<R> prod[G::CH2];
      load_cols<G, 0>(lp, b, prod);
#pragma unroll
      for (int r = 0; r < G::RN; r++) {
        const int row = a + G::LA * r;
        // the lane's first column at or right of the diagonal lies `first` steps off it
        const int first = (b - a + G::LA) & (G::LB - 1);
        R f = wp * g[row];
#pragma unroll
        for (int t = 0; t + 1 < G::LB; t++) f = t < first ? f * rho[row + t] : f;
        R cur = R(0), even = R(0);
        constexpr int X = G::LB;
#pragma unroll
        for (int i = G::LA * r / X; i < G::CN; i++) {
          if (i <= (G::LA * r + G::LA - 1) / X + 1) {
            const int off = b + X * i - row;
            cur = off < 0 ? R(0) : (off < X ? f : cur * get(prod, i));
          } else {
            cur *= get(prod, i);
          }
          if (i & 1) A[r][i / 2] = padd(A[r][i / 2], Pair<R>(i > G::LA * r / X ? even : R(0), cur));
          even = cur;
        }
      }
    }
    if (p0 == 0) {
      for (int c = l; c < k; c += G::L) U.z[c] = U.work[G::CH * G::PS + G::KN + 8 + c];
    }
    p0 += nc;
    const bool more = p0 < np;
    // a unit of the warp that is done repeats nothing (nc = 0)
    if (G::L < 32 ? !__any_sync(0xffffffffu, more) : !more) break;
    team_sync<G>();
  }
  // ---- W = Q S^(-1/2) Q^T, wbar = Q z
  mirror_all<G, 0>(A, U.work, a, b);
  team_sync<G>();   // the steps' buffers overlay the shifts' arrays
  z.load(U, l);
  fetch_reflector<G>(U, gv, k - 3, l);
  fetch_reflector<G>(U, gv, k - 4, l);
  fetch_reflector<G>(U, gv, k - 5, l);
  back_all<G, G::RN - 1>(A, U, z, gv, k, l, a, b);
  copy_wait<0>();
  z.store(U, l);
  team_sync<G>();
  R zr[G::RN];
#pragma unroll
  for (int r = 0; r < G::RN; r++) zr[r] = U.z[a + G::LA * r];
  if (Tout) {
#pragma unroll
    for (int r = 0; r < G::RN; r++) {
      const int row = a + G::LA * r;
#pragma unroll
      for (int i = 0; i < G::CN; i++) {
        const int col = b + G::LB * i;
        if (row < k && col < k) Tout[row * k + col] = (float)(get(A[r], i) + zr[r]);
      }
    }
    if (wout)
      for (int c = l; c < k; c += G::L) wout[c] = (float)U.z[c];
  }
  return nan ? 1 : (bad ? 2 : 0);
}

template <class G>
__global__ void __launch_bounds__(G::THREADS, G::MB) k_transform(EigArgs a, typename PolesOf<typename G::R>::type tab,
                                                          EigSplit sp, typename G::R *vscr, int u0, int nb,
                                                          const int *range, int above, int upto) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using R = typename G::R;
  const int slot = threadIdx.x / G::L, l = threadIdx.x % G::L;
  R *mem = reinterpret_cast<R *>(smem_raw) + (size_t)slot * G::UNIT;
  R *gv = vscr + ((size_t)blockIdx.x * G::UPB + slot) * G::REFL;
  // units u0 .. u0 + nb (through ulist), or the flagged entries not yet
  // re-solved, if there are more than `above` and at most `upto`
  int beg = 0, end = nb;
  const int *list = a.ulist;
  if (range) {
    beg = range[1];
    end = min(range[0], a.flag_cap);
    if (end - beg <= above || end - beg > upto) return;
    list = a.flag_list;
    u0 = 0;
  }
  for (int first = beg + blockIdx.x * G::UPB; first < end; first += gridDim.x * G::UPB) {
    const int un = first + slot;
    int unit = -1;
    if (un < end) unit = list ? list[u0 + un] : u0 + un;
    // no local observations: the update keeps the background
    const bool on = unit >= 0 && a.nkept[unit] > 0;
    if (G::L > 32) {
      if (!on) continue;
    } else if (!__any_sync(0xffffffffu, on)) {
      continue;
    }
    const int k = a.k;
    float *de = on && sp.DE ? sp.DE + (size_t)un * 2 * k : nullptr;
    const int bad = unit_transform<G>(mem, tab, gv, k, a.infl, on ? a.G + (size_t)unit * packed_size(k) : nullptr,
                                      on ? a.T + (size_t)unit * k * k : nullptr,
                                      on && a.wbar ? a.wbar + (size_t)unit * k : nullptr, de, l);
    if (on && l == 0) {
      // with flagging, the FP64 re-solve takes a failed unit
      if (sp.DE) sp.bad[un] = bad;
      else if (bad) atomicOr(a.status, bad);
    }
    team_sync<G>();
  }
}

// FP32_RESOLVE: the units of a batch for the FP64 re-solve, on the tridiagonal
// form k_transform left.  A unit is flagged when its FP32 solve failed, an
// eigenvalue is not positive, or two relevant eigenvalues lie within
// gap_thresh * max l of each other.  The eigenvalues at the (k-1)/infl floor
// (the null space of the Gram, k - n of them when n < k) are exactly degenerate
// and harmless, since T is a function of the matrix and not of the basis chosen
// in an eigenspace; they are left out of the test.
//
// Each thread bisects one eigenvalue of one unit on the count of negative
// pivots of T - x I (Sturm; Wilkinson & Reinsch, Handbook for Automatic
// Computation II, 1971, contribution II/5): kBisect halvings of the Gershgorin
// interval, past which FP32 resolves nothing of max l.  A block's threads run
// over the eigenvalues of as many units as fill it: with a warp per unit,
// k = 37 took two rounds, the second on five lanes (4,248 units: 129 us, now
// 80).
constexpr int kBisect = 26;
constexpr int GAPT = 256;                 // most threads per block; at least two units of kMaxK
constexpr int GAPU = 8;                   // most units per block
inline int gap_units(int k) { return std::min(GAPU, GAPT / k); }
static_assert(GAPT >= kMaxK, "a unit's eigenvalues fit a block");

__global__ void __launch_bounds__(GAPT) k_eig_gap(EigArgs a, EigSplit sp, int u0, int nb, int upb) {
  // rows of k values, one apart from a multiple of the banks
  __shared__ float sd[GAPT + GAPU], se[GAPT + GAPU], sl[GAPT + GAPU];
  __shared__ int sflag[GAPU];
  const int k = a.k, pitch = k + (k % 32 == 0);
  const int u = threadIdx.x / k, i = threadIdx.x - u * k;
  const int ub = blockIdx.x * upb + u;
  int unit = -1;
  if (u < upb && ub < nb) {
    unit = a.ulist ? a.ulist[u0 + ub] : u0 + ub;
    if (a.nkept[unit] <= 0) unit = -1;
  }
  const bool failed = unit >= 0 && sp.bad[ub] != 0, test = unit >= 0 && !failed;
  float *d = sd + u * pitch, *e2 = se + u * pitch, *lam = sl + u * pitch;
  if (unit >= 0 && i == 0) sflag[u] = failed;
  if (test) {
    const float *de = sp.DE + (size_t)ub * 2 * k;
    d[i] = de[i];
    e2[i] = fabsf(i > 0 ? de[k + i - 1] : 0.0f);   // |e| first, for the interval
    lam[i] = i < k - 1 ? fabsf(de[k + i]) : 0.0f;
  }
  __syncthreads();
  float lo = 3.0e38f, hi = -3.0e38f, el = 0.0f;
  if (test) {
    for (int j = 0; j < k; j++) {
      lo = fminf(lo, d[j] - e2[j] - lam[j]);
      hi = fmaxf(hi, d[j] + e2[j] + lam[j]);
    }
    el = e2[i];
  }
  __syncthreads();
  if (test) e2[i] = el * el;
  __syncthreads();
  if (test) {
    const float tiny = fmaxf(1e-30f, 1e-14f * fmaxf(fabsf(lo), fabsf(hi)));
    for (int it = 0; it < kBisect; it++) {
      const float x = 0.5f * (lo + hi);
      int below = 0;
      float q = 1.0f;
#pragma unroll 4
      for (int j = 0; j < k; j++) {
        q = (d[j] - x) - __fdividef(e2[j], q);
        q = fabsf(q) < tiny ? -tiny : q;
        below += q < 0.0f;
      }
      if (below > i) hi = x;
      else lo = x;
    }
    lam[i] = 0.5f * (lo + hi);
  }
  __syncthreads();
  if (test) {
    const float li = lam[i], lmax = lam[k - 1], bound = a.gap_thresh * lmax;
    // rounding level of the FP32 eigenvalues: a few k eps of the largest
    const float floor_v = (float)(k - 1) / a.infl;
    const float tol = 4.0f * (float)k * 1.1920929e-7f * lmax;
    // ascending: the nearest relevant neighbour is the next one
    const bool near = li - floor_v > tol && i + 1 < k && fabsf(lam[i + 1 < k ? i + 1 : i] - li) <= bound;
    if (near || !(li > 0.0f) || 3.0e38f <= bound) sflag[u] = 1;
  }
  __syncthreads();
  if (unit >= 0 && i == 0 && sflag[u]) {
    const int pos = atomicAdd(a.flag_n, 1);
    if (pos < a.flag_cap) a.flag_list[pos] = unit;
    else atomicOr(a.status, 128);   // list full: the unit keeps its FP32 solve
  }
}

// resident blocks of the whole GPU: the register bound, or shared memory
template <class G>
constexpr int resident_blocks() {
  const int bytes = G::UPB * G::UNIT * (int)sizeof(typename G::R) + 1024, fit = 227 * 1024 / bytes;
  return 152 * (fit < G::MB ? fit : G::MB);
}

// The grid is one wave, each block striding over the units: the reflectors'
// scratch is one slot per resident unit and stays in L2.
template <class G>
cudaError_t launch_g(cudaStream_t st, const EigArgs &a, const EigSplit &sp, int u0, int nb, const int *range,
                     int above, int upto, int *launches) {
  const size_t smem = (size_t)G::UPB * G::UNIT * sizeof(typename G::R);
  cudaError_t e = cudaFuncSetAttribute(k_transform<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int grid = std::min(resident_blocks<G>(), (std::min(nb, a.slots) + G::UPB - 1) / G::UPB);
  k_transform<G><<<grid, G::THREADS, smem, st>>>(a, PolesOf<typename G::R>::get(), sp,
                                                 reinterpret_cast<typename G::R *>(a.scratch), u0, nb, range,
                                                 above, upto);
  (*launches)++;
  return cudaGetLastError();
}

// calls f with the lane grid of an ensemble size
// FP32: one warp holds four units up to k = 24, two up to 40, one up to 72; a
// team of two warps a unit up to 112, of four above.
template <class F>
auto with_grid_f32(int k, F f) {
#define LGPU_GRID(...) return f(Grid<float, __VA_ARGS__>())
  switch ((k + 7) / 8) {
  case 1: LGPU_GRID(1, 8, 8, 1, 6);
  case 2: LGPU_GRID(2, 16, 8, 1, 5);
  case 3: LGPU_GRID(3, 24, 8, 1, 3);
  case 4: LGPU_GRID(4, 16, 8, 2, 3);
  case 5: LGPU_GRID(5, 20, 8, 2, 2);
  case 6: LGPU_GRID(6, 12, 8, 4, 3);
  case 7: LGPU_GRID(7, 14, 8, 4, 2);
  case 8: LGPU_GRID(8, 16, 8, 4, 2);
  case 9: LGPU_GRID(9, 18, 8, 4, 2);
  case 10: LGPU_GRID(5, 20, 16, 4, 6);
  case 11: LGPU_GRID(6, 22, 16, 4, 4);
  case 12: LGPU_GRID(6, 24, 16, 4, 4);
  case 13: LGPU_GRID(7, 26, 16, 4, 4);
  case 14: LGPU_GRID(7, 28, 16, 4, 4);
  default: LGPU_GRID(8, 16, 16, 8, 2);
  }
#undef LGPU_GRID
}

// FP64: GB300 runs FP64 at 1/64 of the FP32 rate, two multiply-adds a clock on
// an SM, so the grids follow the size closely: one warp a unit up to k = 48
// (the most a lane's registers hold), two up to 64, four up to 112, eight above
template <class F>
auto with_grid_f64(int k, F f) {
#define LGPU_GRID(...) return f(Grid<double, __VA_ARGS__>())
  if (k <= 16) LGPU_GRID(2, 4, 8, 4, 4);
  if (k <= 24) LGPU_GRID(3, 6, 8, 4, 4);
  if (k <= 32) LGPU_GRID(4, 8, 8, 4, 2);
  if (k <= 40) LGPU_GRID(5, 10, 8, 4, 2);
  if (k <= 48) LGPU_GRID(6, 12, 8, 4, 1);
  if (k <= 64) LGPU_GRID(8, 8, 8, 8, 4);
  if (k <= 80) LGPU_GRID(5, 10, 16, 8, 2);
  if (k <= 96) LGPU_GRID(6, 12, 16, 8, 2);
  if (k <= 112) LGPU_GRID(7, 14, 16, 8, 2);
  LGPU_GRID(4, 16, 32, 8, 1);
#undef LGPU_GRID
}

// FP64 grids for a list of few flagged units: four warps or more a unit.  A
// warp issues FP64 to its own quarter of the SM, one multiply-add in two
// clocks, so one warp a unit runs a lone unit at a quarter of the SM's rate
// (k = 37, up to 112 units: 433 us, now 321).  The list's length stays on the
// device: both kernels are launched, and the one whose range it is not in
// returns at once.
template <class F>
auto with_grid_f64_few(int k, F f) {
#define LGPU_GRID(...) return f(Grid<double, __VA_ARGS__>())
  if (k <= 16) LGPU_GRID(1, 2, 16, 8, 2);
  if (k <= 32) LGPU_GRID(2, 4, 16, 8, 2);
  if (k <= 48) LGPU_GRID(3, 6, 16, 8, 2);
  if (k <= 64) LGPU_GRID(4, 8, 16, 8, 2);
#undef LGPU_GRID
  return with_grid_f64(k, f);
}

cudaError_t launch_f32(cudaStream_t st, const EigArgs &a, const EigSplit &sp, int u0, int nb, int *launches) {
  return with_grid_f32(a.k, [&](auto g) { return launch_g<decltype(g)>(st, a, sp, u0, nb, nullptr, 0, 0, launches); });
}

cudaError_t launch_f64(cudaStream_t st, const EigArgs &a, int u0, int nb, int *launches) {
  return with_grid_f64(
      a.k, [&](auto g) { return launch_g<decltype(g)>(st, a, EigSplit{}, u0, nb, nullptr, 0, 0, launches); });
}

// The longest list that takes these grids.  The block scheduler starts to put
// two blocks on an SM between 112 and 120 of them.  Beyond, where this grid
// covers more rows than the other one (k = 17 to 24: 32 to 24; 33 to 40: 48 to
// 40) or both cover 16, the other is the faster one at once (us, this grid and
// the other, 120 to 304 units: k = 16 104 and 94, k = 24 226 and 175, k = 37
// 473 and 434).  Where both cover the same this one holds to its full wave of
// two blocks an SM (304 units: k = 32 270 and 289, k = 48 543 and 653, k = 64
// 950 and 1,219; 456 units: 524 and 287, 1,072 and 653, 1,877 and 1,228).
constexpr int kOneAnSM = 112;
template <class G>
int few_units(int k) {
  return k <= 24 || (k > 32 && k <= 40) ? kOneAnSM : resident_blocks<G>();
}

constexpr int kAll = 0x7fffffff;

// the entries [range[1], range[0]) of the flagged list (as many blocks as
// nunits units have scratch for; the list itself may be longer)
cudaError_t launch_f64_list(cudaStream_t st, const EigArgs &a, const int *range, int *launches) {
  int few = kAll;   // lists up to here on the first grid
  cudaError_t e = with_grid_f64_few(a.k, [&](auto g) {
    using G = decltype(g);
    with_grid_f64(a.k, [&](auto h) {
      if (!std::is_same<G, decltype(h)>::value) few = few_units<G>(a.k);
    });
    return launch_g<G>(st, a, EigSplit{}, 0, a.nunits, range, 0, few, launches);
  });
  if (e != cudaSuccess || few == kAll || a.flag_cap <= few) return e;
  return with_grid_f64(
      a.k, [&](auto g) { return launch_g<decltype(g)>(st, a, EigSplit{}, 0, a.nunits, range, few, kAll, launches); });
}

struct ScratchOf {
  int units;
  template <class G>
  size_t operator()(G) const {
    const size_t blocks = std::min<size_t>(resident_blocks<G>(), ((size_t)units + G::UPB - 1) / G::UPB);
    return blocks * G::UPB * G::REFL * sizeof(typename G::R);
  }
};

}  // namespace

size_t eig_scratch_bytes(int k, int units, bool fp32, bool fp64) {
  const ScratchOf f{std::max(1, units)};
  return std::max(fp32 ? with_grid_f32(k, f) : 0,
                  fp64 ? std::max(with_grid_f64(k, f), with_grid_f64_few(k, f)) : 0);
}

cudaError_t launch_eig64(cudaStream_t st, const EigArgs &a, int ubase, int *launches) {
  if (a.nunits <= 0) return cudaSuccess;
  return launch_f64(st, a, ubase, a.nunits, launches);
}

cudaError_t launch_eig64_flagged(cudaStream_t st, const EigArgs &a, int *launches) {
  if (!a.flag_list || a.flag_cap <= 0) return cudaSuccess;
  // the count stays on the device: the wave of blocks strides over the list
  cudaError_t e = launch_f64_list(st, a, a.flag_n, launches);
  if (e != cudaSuccess) return e;
  return cudaMemcpyAsync(a.flag_n + 1, a.flag_n, sizeof(int), cudaMemcpyDeviceToDevice, st);
}

size_t eig_split_bytes_per_unit(int k) { return (size_t)2 * k * 4 + 4; }

cudaError_t launch_eig_split(cudaStream_t st, const EigArgs &a, const EigSplit &sp, int batch, int ustart, int ucount,
                             int *launches) {
  if (ucount <= 0) return cudaSuccess;
  if (!a.flag_list) return launch_f32(st, a, EigSplit{}, ustart, ucount, launches);
  cudaError_t e = cudaSuccess;
  const int uend = ustart + ucount;
  for (int u0 = ustart; u0 < uend; u0 += batch) {
    const int nb = uend - u0 < batch ? uend - u0 : batch;
    if ((e = launch_f32(st, a, sp, u0, nb, launches)) != cudaSuccess) return e;
    const int upb = gap_units(a.k);
    k_eig_gap<<<(nb + upb - 1) / upb, (upb * a.k + 31) / 32 * 32, 0, st>>>(a, sp, u0, nb, upb);
    (*launches)++;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_eig_debug(cudaStream_t st, int nunits, int k, const float *G, const int *nkept, float *T,
                             int *status, int prec, float gap_thresh, int *nfp64) {
  EigArgs a;
  a.wbar = nullptr;
  a.ulist = nullptr;
  a.flag_list = nullptr;
  a.flag_n = nullptr;
  a.flag_cap = 0;
  a.gap_thresh = gap_thresh;
  a.nunits = nunits;
  a.k = k;
  a.infl = 1.0f;
  a.G = G;
  a.nkept = nkept;
  a.T = T;
  a.status = status;
  *nfp64 = 0;
  int l = 0;
  // as lgpu_solver_run uses it
  const size_t n = nunits > 0 ? nunits : 1;
  const bool resolve = prec == LGPU_PREC_FP32_RESOLVE;
  unsigned char *buf = nullptr;
  const size_t vb = eig_scratch_bytes(k, (int)n, prec != LGPU_PREC_FP64, prec != LGPU_PREC_FP32);
  // four arrays, each start rounded up to 256 bytes
  cudaError_t e = cudaMalloc(&buf, vb + (resolve ? eig_split_bytes_per_unit(k) * n + 16 + 4 * n : 0) + 4 * 256);
  if (e != cudaSuccess) return e;
  size_t off = 0;
  auto take = [&](size_t bytes) { unsigned char *p = buf + off; off += (bytes + 255) & ~(size_t)255; return p; };
  a.scratch = take(vb);
  a.slots = (int)n;
  if (prec == LGPU_PREC_FP64) {
    e = launch_eig64(st, a, 0, &l);
    cudaError_t e2 = cudaStreamSynchronize(st);
    cudaFree(buf);
    *nfp64 = nunits;
    return e != cudaSuccess ? e : e2;
  }
  EigSplit sp{};
  if (resolve) {
    sp.DE = reinterpret_cast<float *>(take(n * 2 * k * 4));
    sp.bad = reinterpret_cast<int *>(take(n * 4));
    a.flag_n = reinterpret_cast<int *>(take(16 + 4 * n));
    a.flag_list = a.flag_n + 4;
    a.flag_cap = (int)n;
    e = cudaMemsetAsync(a.flag_n, 0, 16, st);
  }
  if (e == cudaSuccess) e = launch_eig_split(st, a, sp, (int)n, 0, nunits, &l);
  if (e == cudaSuccess && a.flag_list) e = launch_eig64_flagged(st, a, &l);
  if (e == cudaSuccess && a.flag_n) e = cudaMemcpyAsync(nfp64, a.flag_n, 4, cudaMemcpyDeviceToHost, st);
  cudaError_t e2 = cudaStreamSynchronize(st);
  cudaFree(buf);
  if (*nfp64 > (int)n) *nfp64 = (int)n;
  return e != cudaSuccess ? e : e2;
}

}  // namespace lgpu
