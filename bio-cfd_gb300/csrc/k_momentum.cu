// Momentum predictor (nsMomentum2order, src/NavierStokes.f90:252-912) and the
// boundary conditions of src/BoundaryConditions.f90.
//
// One thread per interior cell; non-fluid cells are skipped.  The reference
// loops over the fluid list in (k,j,i) order, and that order matters only next
// to thin-surface (TS) cells: there the loop substitutes ghost values into
// u,v,w,p before a cell's stencil and restores them after it
// (src/NavierStokes.f90:310-490, 860-907), so a cell may read values written
// by earlier cells.  Cells within reach of a TS cell go through a second
// kernel whose reads reproduce that serial order exactly (TsReader below);
// every other cell reads the fields directly.  FP64, compiled without FMA
// contraction, expressions in the reference's evaluation order (T = double);
// the same stencil in FP32 arithmetic serves the mixed-precision path.
#include <type_traits>
#include <utility>

#include "bcfd_host.h"

namespace bcfd {

namespace {

// deltat, re, and what div_any needs to divide by re (re_k: DivKind bits)
struct MomArgs {
  double dt, re, re_y;
  unsigned re_k;
};

// Divisors of the stencil along one axis at grid index q (dl, d, dr the
// spacings of q - 1, q, q + 1; CA / CK the sixth column of the axis's own (self)
// and transverse (cross) coefficient tables), then its grid-only quotients and
// the tables' first five columns.  Groups of 32 indices hold 32 consecutive
// entries per slot: a warp's x entries are contiguous and every slot sits at a
// constant offset from a thread's first one (immediate addresses).
enum MomDiv {
  MD_HALF_R = 0,  // 0.5 (d + dr)
  MD_HALF_L,      // 0.5 (d + dl)
  MD_SA,          // CAself dr
  MD_SK,          // (2 CKself) d
  MD_XA,          // CAcross (0.5 (d + dr))
  MD_XK,          // (2 CKcross) (0.5 (d + dl))
  MD_D,           // d
  MD_R,           // dr
  N_MD
};
enum MomQuot { MQ_R = 0, MQ_2, MQ_C, N_MQ };  // dr / (d + dr), 2 / (d + dr), 2 / (0.5 ((d + dr) + (d + dl)))
// FP64 slots: divisor and reciprocal of each MomDiv, the quotients, CA and CK
// 1..5 self, CA and CK 1..5 cross; FP32 slots: reciprocals, quotients by
// __fdividef, divisors, IEEE quotients, the same coefficients
constexpr int kMtQ = 2 * N_MD, kMtC = kMtQ + N_MQ, kMtSlots = kMtC + 20;
constexpr int kMfQ = N_MD, kMfD = kMfQ + N_MQ, kMfI = kMfD + N_MD, kMfC = kMfI + N_MQ, kMfSlots = kMfC + 20;

// first entry of grid index q (0-based) of an axis whose groups start at g0
__host__ __device__ inline int64_t mom_slot0(int g0, int q, int slots) {
  return ((int64_t)(g0 + (q >> 5)) * slots) * 32 + (q & 31);
}
__host__ __device__ inline int mom_groups(int n) { return (n + 31) >> 5; }

// how a divisor's reciprocal may be used: bit s of the axis word, the quotient
// needs a second correction; bit 8 + s, the division itself is needed
__host__ __device__ inline unsigned div_kind(double d, double y) {
  const double m = d < 0 ? -d : d;
  if (!(m > 0x1p-300 && m < 0x1p300)) return 0x100u;
  double e = fma(-d, y, 1.0);
  if (e < 0) e = -e;
  return e > 0x1p-54 ? 1u : 0u;
}

__device__ __noinline__ double ieee_quot(double v, double d) { return v / d; }
// v / d, correctly rounded, from y = RN(1/d): Markstein's remainder step (IBM
// J. Res. Dev. 34, 1990), a second one where q = RN(v y) may be more than an
// ulp off (|1 - d y| > 2^-54).  A zero remainder leaves q as it is (its sign
// too).  Numerators out of the range in which every intermediate is normal
// take the division.
__device__ __forceinline__ double div_any(double v, double d, double y, unsigned kind, int s) {
  auto fix = [&](double q) {
    const double r = fma(-q, d, v);
    const double c = fma(r, y, q);
    return (((unsigned)__double2hiint(r) << 1) | (unsigned)__double2loint(r)) ? c : q;
  };
  double q = fix(v * y);
  if ((kind >> s) & 1u) q = fix(q);
  const unsigned vh = (unsigned)__double2hiint(v) & 0x7fffffffu;
  const bool usual = vh - 0x2d300000u < 0x25800000u || (vh | (unsigned)__double2loint(v)) == 0u;
  if (!usual || ((kind >> (8 + s)) & 1u)) q = ieee_quot(v, d);
  return q;
}

__device__ __forceinline__ bool adj_ok(const int8_t* c, const Dims& d, bool big, int i, int j, int k,
                                       int s) {
  // check_adjacent_cell (src/NavierStokes.f90:1002-1022): false if any of the
  // 6 cells at distance s has tag 2
  auto at = [&](int a, int b, int e) { return big ? c[d.idx3(a, b, e)] : c[d.idx(a, b, e)]; };
  if (at(i - s, j, k) == 2) return false;
  if (at(i + s, j, k) == 2) return false;
  if (at(i, j - s, k) == 2) return false;
  if (at(i, j + s, k) == 2) return false;
  if (at(i, j, k - s) == 2) return false;
  if (at(i, j, k + s) == 2) return false;
  return true;
}

// FP32 number of the mixed path's momentum stencil.  Every divisor of the
// stencil is a grid quantity (spacings, their sums, coefficient-table
// entries, re), so the quotient is taken as a reciprocal times the dividend
// (__fdividef, within 2 ulp of the IEEE quotient) instead of the IEEE
// division's instruction sequence; the stencil's FP32 rounding dominates that
// difference.  The FP64 drop-in stencil keeps IEEE division.
struct FastF {
  float v;
  FastF() = default;
  __device__ __forceinline__ constexpr FastF(float x) : v(x) {}
  __device__ __forceinline__ explicit FastF(double x) : v((float)x) {}
  __device__ __forceinline__ explicit operator double() const { return (double)v; }
};
__device__ __forceinline__ FastF operator+(FastF a, FastF b) { return FastF(a.v + b.v); }
__device__ __forceinline__ FastF operator-(FastF a, FastF b) { return FastF(a.v - b.v); }
__device__ __forceinline__ FastF operator-(FastF a) { return FastF(-a.v); }
__device__ __forceinline__ FastF operator*(FastF a, FastF b) { return FastF(a.v * b.v); }
__device__ __forceinline__ FastF operator/(FastF a, FastF b) { return FastF(__fdividef(a.v, b.v)); }
__device__ __forceinline__ FastF fabs(FastF a) { return FastF(fabsf(a.v)); }

// Forward-mode dual number (value, tangent): the stencil evaluated in it gives
// the reference's FP64 value (the value part performs exactly the double
// operations) and the exact derivative of the discrete stencil along the
// input tangent (the tangent-linear model).
struct Dual {
  double v, d;
  __device__ Dual() : v(0.0), d(0.0) {}
  __device__ Dual(double x) : v(x), d(0.0) {}
  __device__ Dual(double x, double dx) : v(x), d(dx) {}
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual(a.v - b.v, a.d - b.d); }
__device__ __forceinline__ Dual operator-(Dual a) { return Dual(-a.v, -a.d); }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return Dual(a.v * b.v, a.d * b.v + a.v * b.d); }
// |x| with the derivative of the branch the value takes (sign(0) = +); the
// global float/double overloads stay visible next to it
using ::fabs;
__device__ __forceinline__ Dual fabs(Dual a) { return a.v < 0.0 ? -a : a; }

// The same with four tangents: one evaluation carries the derivatives along
// four seeds at once.  Each tangent lane performs exactly the operations of
// Dual's tangent on the same operands, so lane l equals the Dual tangent of
// seed l bit for bit.
struct Dual4 {
  double v, d[4];
  __device__ Dual4() : v(0.0), d{0.0, 0.0, 0.0, 0.0} {}
  __device__ Dual4(double x) : v(x), d{0.0, 0.0, 0.0, 0.0} {}
};
__device__ __forceinline__ Dual4 operator+(const Dual4& a, const Dual4& b) {
  Dual4 r(a.v + b.v);
#pragma unroll
  for (int l = 0; l < 4; ++l) r.d[l] = a.d[l] + b.d[l];
  return r;
}
__device__ __forceinline__ Dual4 operator-(const Dual4& a, const Dual4& b) {
  Dual4 r(a.v - b.v);
#pragma unroll
  for (int l = 0; l < 4; ++l) r.d[l] = a.d[l] - b.d[l];
  return r;
}
__device__ __forceinline__ Dual4 operator-(const Dual4& a) {
  Dual4 r(-a.v);
#pragma unroll
  for (int l = 0; l < 4; ++l) r.d[l] = -a.d[l];
  return r;
}
__device__ __forceinline__ Dual4 operator*(const Dual4& a, const Dual4& b) {
  Dual4 r(a.v * b.v);
#pragma unroll
  for (int l = 0; l < 4; ++l) r.d[l] = a.d[l] * b.v + a.v * b.d[l];
  return r;
}
__device__ __forceinline__ Dual4 fabs(const Dual4& a) { return a.v < 0.0 ? -a : a; }

// Grid quantities have no tangent: plain numbers beside the dual types, the
// tangent's products with their zeros left out.  Those products are zeros only
// while the values are finite; an infinite or NaN value makes the tangent of
// everything that it enters NaN, and a derivative taken at such a state must
// not look like a number.  EXACT keeps them: the grid quantities are dual
// numbers with tangent 0, with the operations of a dual quotient.  Every value
// that enters an output makes that output non-finite when it is not finite
// itself, so finite outputs tell that the short form gives EXACT's bits.
template <typename T, bool EXACT>
struct GridNum {
  using type = T;
};
template <>
struct GridNum<Dual, false> {
  using type = double;
};
template <>
struct GridNum<Dual4, false> {
  using type = double;
};
__device__ __forceinline__ Dual operator*(double c, Dual a) { return Dual(c * a.v, c * a.d); }
__device__ __forceinline__ Dual operator*(Dual a, double c) { return Dual(a.v * c, a.d * c); }
__device__ __forceinline__ Dual operator+(Dual a, double c) { return Dual(a.v + c, a.d); }
__device__ __forceinline__ Dual operator+(double c, Dual a) { return Dual(c + a.v, a.d); }
__device__ __forceinline__ Dual operator-(Dual a, double c) { return Dual(a.v - c, a.d); }
__device__ __forceinline__ Dual operator-(double c, Dual a) { return Dual(c - a.v, -a.d); }
__device__ __forceinline__ Dual4 operator*(double c, const Dual4& a) {
  Dual4 r(c * a.v);
#pragma unroll
  for (int l = 0; l < 4; ++l) r.d[l] = c * a.d[l];
  return r;
}

// One axis's tables at one grid index.
template <typename T, bool EXACT>
struct MomAxis {
  static constexpr int n = 32;  // entries between slots
  const double* t;
  const float* f;
  unsigned k;
  __device__ __forceinline__ MomAxis(const DevBlock& B, int g0, int q)
      : t(B.mt + mom_slot0(g0, q - 1, kMtSlots)), f(B.mtf + mom_slot0(g0, q - 1, kMfSlots)),
        k(B.mtk[32 * g0 + q - 1]) {}
  using G = typename GridNum<T, EXACT>::type;
  // numerator / divisor s: FP64 by div_any (the division's bits); FP32 of the
  // mixed path by the reciprocal (the bits of __fdividef)
  // (V: T, or double where a static seed leaves the operand no tangent)
  template <typename V>
  __device__ __forceinline__ V div(const V& a, int s) const {
    if constexpr (std::is_same<T, FastF>::value) {
      return FastF(a.v * f[s * n]);
    } else if constexpr (std::is_same<T, float>::value) {
      return a / f[(kMfD + s) * n];
    } else {
      const double d = t[2 * s * n], y = t[(2 * s + 1) * n];
      if constexpr (std::is_same<V, double>::value) {
        return div_any(a, d, y, k, s);
      } else if constexpr (std::is_same<V, Dual>::value) {
        const double q = div_any(a.v, d, y, k, s);
        return Dual(q, div_any(EXACT ? a.d - q * 0.0 : a.d, d, y, k, s));
      } else {
        Dual4 r(div_any(a.v, d, y, k, s));
#pragma unroll
        for (int l = 0; l < 4; ++l) r.d[l] = div_any(EXACT ? a.d[l] - r.v * 0.0 : a.d[l], d, y, k, s);
        return r;
      }
    }
  }
  __device__ __forceinline__ G quot(int s) const {
    if constexpr (std::is_same<T, FastF>::value) return G(f[(kMfQ + s) * n]);
    else if constexpr (std::is_same<T, float>::value) return f[(kMfI + s) * n];
    else return G(t[(kMtQ + s) * n]);
  }
  // column c (1..5) of CA (kind 0) / CK (1) self, CA (2) / CK (3) cross
  __device__ __forceinline__ G coef(int kind, int c) const {
    if constexpr (std::is_same<T, FastF>::value || std::is_same<T, float>::value)
      return G(f[(kMfC + 5 * kind + c - 1) * n]);
    else return G(t[(kMtC + 5 * kind + c - 1) * n]);
  }
};

// division by re
template <bool EXACT, typename T>
__device__ __forceinline__ T div_re(const T& a, const MomArgs& m) {
  if constexpr (std::is_same<T, double>::value) {
    return div_any(a, m.re, m.re_y, m.re_k, 0);
  } else if constexpr (std::is_same<T, Dual>::value) {
    const double q = div_any(a.v, m.re, m.re_y, m.re_k, 0);
    return Dual(q, div_any(EXACT ? a.d - q * 0.0 : a.d, m.re, m.re_y, m.re_k, 0));
  } else if constexpr (std::is_same<T, Dual4>::value) {
    Dual4 r(div_any(a.v, m.re, m.re_y, m.re_k, 0));
#pragma unroll
    for (int l = 0; l < 4; ++l) r.d[l] = div_any(EXACT ? a.d[l] - r.v * 0.0 : a.d[l], m.re, m.re_y, m.re_k, 0);
    return r;
  } else {
    return a / T(m.re);
  }
}

__device__ __forceinline__ bool not_finite(double v) {
  return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u;
}

// where a stencil's three results go
struct StoreOut {
  double *ut, *vt, *wt;
  template <typename T>
  __device__ __forceinline__ void put(int q, int64_t c, T val) const {
    (q == 0 ? ut : q == 1 ? vt : wt)[c] = (double)val;
  }
};
struct DualOut {
  double *ut, *vt, *wt, *dut, *dvt, *dwt;
  __device__ __forceinline__ void put(int q, int64_t c, Dual val) const {
    (q == 0 ? ut : q == 1 ? vt : wt)[c] = val.v;
    (q == 0 ? dut : q == 1 ? dvt : dwt)[c] = val.d;
  }
};

// Field reads of the stencil: field f (0 u, 1 v, 2 w, 3 p) at cell (a,b,e),
// linear index x.  The plain reader loads the array.
struct PlainReader {
  const double* f[4];
  __device__ __forceinline__ double get(int q, int, int, int, int64_t x) const { return __ldg(f[q] + x); }
};

// the FP32 copies of the fields (mixed path)
struct PlainReaderF {
  const float* f[4];
  __device__ __forceinline__ float get(int q, int, int, int, int64_t x) const { return __ldg(f[q] + x); }
};

// A seed known at compile time: 1 at field F, offset (A,B,E) from the cell.
// Reads elsewhere are plain numbers, so that the tangent's products with
// structural zeros are never formed; ok is the cell's third-order test.
template <int F, int A, int B, int E>
struct StaticSeed {
  const double* f[4];
  bool ok;
};
template <typename Rd>
struct SeedOf {
  static constexpr bool is = false;
};
template <int F, int A, int B, int E>
struct SeedOf<StaticSeed<F, A, B, E>> {
  static constexpr bool is = true;
  __host__ __device__ static constexpr bool at(int q, int a, int b, int e) { return q == F && a == A && b == B && e == E; }
};
template <typename T, int Q, int A, int B, int E, class Rd>
__device__ __forceinline__ auto mom_read(const Rd& rd, int i, int j, int k, int64_t x) {
  if constexpr (SeedOf<Rd>::is) {
    const double v = __ldg(rd.f[Q] + x);
    if constexpr (SeedOf<Rd>::at(Q, A, B, E)) return Dual(v, 1.0);
    else return v;
  } else {
    return (T)rd.get(Q, i, j, k, x);
  }
}
// the tangent of output Q alone
template <int Q>
struct TangentOut {
  double* t;
  __device__ __forceinline__ void put(int, int64_t, Dual val) const { *t = val.d; }
};
template <class Out>
struct OutputOf {  // the one output wanted, -1: all three
  static constexpr int q = -1;
};
template <int Q>
struct OutputOf<TangentOut<Q>> {
  static constexpr int q = Q;
};

// third-order differences where no cell around carries tag 2; inside the
// index range (a superset of the three components') the distance-2
// neighbours exist
__device__ __forceinline__ bool mom_smooth(const DevBlock& B, int i, int j, int k) {
  const Dims& d = B.d;
  const bool inner = i > 2 && j > 2 && k > 2 && i < d.nx + 1 && j < d.ny + 1 && k < d.nz + 1;
  return inner && adj_ok(B.cell, d, false, i, j, k, 1) && adj_ok(B.cell2, d, true, i, j, k, 2);
}

// One fluid cell (i,j,k) of nsMomentum2order.  T = double: the reference
// arithmetic (bit-exact drop-in).  T = FastF or float: the FP32 momentum stencil
// of the mixed-precision path (it reads the fields' FP32 copies, beside
// thin-surface cells the FP64 fields rounded on load; ut/vt/wt are stored as
// FP64).  EXACT: see GridNum.
template <typename T, bool EXACT = false, class Rd, class Out>
__device__ __forceinline__ void momentum_cell(const DevBlock& B, const MomArgs& a, int i, int j, int k,
                                              int64_t c, const Rd& rd, const Out& out) {
  using G = typename GridNum<T, EXACT>::type;
  const G Q25 = G(0.25), HALF = G(0.5), alpha = G(1.0);
  const Dims& d = B.d;
  const G deltat = G(a.dt);
  const int gy = mom_groups(d.NX), gz = gy + mom_groups(d.NY);
  const MomAxis<T, EXACT> AX(B, 0, i), AY(B, gy, j), AZ(B, gz, k);
  const int nx_var = d.nx, ny_var = d.ny, nz_var = d.nz;
  const int64_t SX = 1, SY = d.NX, SZ = (int64_t)d.NX * d.NY;
  {
#define u(a, b, e) \
  mom_read<T, 0, a, b, e>(rd, i + (a), j + (b), k + (e), c + (a) * SX + (b) * SY + (e) * SZ)
#define v(a, b, e) \
  mom_read<T, 1, a, b, e>(rd, i + (a), j + (b), k + (e), c + (a) * SX + (b) * SY + (e) * SZ)
#define w(a, b, e) \
  mom_read<T, 2, a, b, e>(rd, i + (a), j + (b), k + (e), c + (a) * SX + (b) * SY + (e) * SZ)
#define p(a, b, e) \
  mom_read<T, 3, a, b, e>(rd, i + (a), j + (b), k + (e), c + (a) * SX + (b) * SY + (e) * SZ)
    // offsets are relative to (i,j,k): u(-1,0,0) is u(i-1,j,k)

    const auto u1a = u(-1, 0, 0) + u(0, 0, 0);
    const auto u22 = u(-1, 0, 0) - u(0, 0, 0);
    const auto u3 = u(0, 0, 0) + u(1, 0, 0);
    const auto u4 = u(0, 0, 0) - u(1, 0, 0);
    const auto u5 = u(0, -1, 0) + u(0, 0, 0);
    const auto u6 = u(0, -1, 0) - u(0, 0, 0);
    const auto u7 = u(0, 0, 0) + u(0, 1, 0);
    const auto u8 = u(0, 0, 0) - u(0, 1, 0);
    const auto u9 = u(0, 0, -1) + u(0, 0, 0);
    const auto u10 = u(0, 0, -1) - u(0, 0, 0);
    const auto u11 = u(0, 0, 0) + u(0, 0, 1);
    const auto u12 = u(0, 0, 0) - u(0, 0, 1);
    const auto u13 = u(-1, 0, 0) + u(-1, 1, 0);
    const auto u14 = u7;
    const auto u15 = u(-1, 0, 0) + u(-1, 0, 1);
    const auto u16 = u11;

    const auto v1a = v(0, -1, 0) + v(1, -1, 0);
    const auto v22 = v(0, 0, 0) + v(1, 0, 0);
    const auto v3 = v(-1, 0, 0) + v(0, 0, 0);
    const auto v4 = v(-1, 0, 0) - v(0, 0, 0);
    const auto v5 = v(0, 0, 0) + v(1, 0, 0);
    const auto v6 = v(0, 0, 0) - v(1, 0, 0);
    const auto v7 = v(0, -1, 0) + v(0, 0, 0);
    const auto v8 = v(0, -1, 0) - v(0, 0, 0);
    const auto v9 = v(0, 0, 0) + v(0, 1, 0);
    const auto v10 = v(0, 0, 0) - v(0, 1, 0);
    const auto v11 = v(0, 0, -1) + v(0, 0, 0);
    const auto v12 = v(0, 0, -1) - v(0, 0, 0);
    const auto v13 = v(0, 0, 0) + v(0, 0, 1);
    const auto v14 = v(0, 0, 0) - v(0, 0, 1);
    const auto v15 = v(0, -1, 0) + v(0, -1, 1);
    const auto v16 = v13;

    const auto w1a = w(0, 0, -1) + w(1, 0, -1);
    const auto w22 = w(0, 0, 0) + w(1, 0, 0);
    const auto w3 = w(0, 0, -1) + w(0, 1, -1);
    const auto w4 = w(0, 0, 0) + w(0, 1, 0);
    const auto w5 = w(-1, 0, 0) + w(0, 0, 0);
    const auto w6 = w(-1, 0, 0) - w(0, 0, 0);
    const auto w7 = w(0, 0, 0) + w(1, 0, 0);
    const auto w8 = w(0, 0, 0) - w(1, 0, 0);
    const auto w9 = w(0, -1, 0) + w(0, 0, 0);
    const auto w10 = w(0, -1, 0) - w(0, 0, 0);
    const auto w11 = w(0, 0, 0) + w(0, 1, 0);
    const auto w12 = w(0, 0, 0) - w(0, 1, 0);
    const auto w13 = w(0, 0, -1) + w(0, 0, 0);
    const auto w14 = w(0, 0, -1) - w(0, 0, 0);
    const auto w15 = w(0, 0, 0) + w(0, 0, 1);
    const auto w16 = w(0, 0, 0) - w(0, 0, 1);

    const auto dpdx = AX.div(p(0, 0, 0) - p(1, 0, 0), MD_HALF_R);
    const auto dpdy = AY.div(p(0, 0, 0) - p(0, 1, 0), MD_HALF_R);
    const auto dpdz = AZ.div(p(0, 0, 0) - p(0, 0, 1), MD_HALF_R);

    bool smooth;
    if constexpr (SeedOf<Rd>::is) smooth = rd.ok;
    else smooth = mom_smooth(B, i, j, k);
    const bool near_ib = !smooth, near_ts2 = false;
    (void)near_ib;

    // ---------------- U momentum ----------------
    if constexpr (OutputOf<Out>::q < 0 || OutputOf<Out>::q == 0) {
      const auto vu_e = v(1, 0, 0) + AX.quot(MQ_R) * (v(0, 0, 0) - v(1, 0, 0));
      const auto vu_w = v(1, -1, 0) + AX.quot(MQ_R) * (v(0, -1, 0) - v(1, -1, 0));
      const auto v_in_um = HALF * (vu_e + vu_w);
      const auto wu_n = w(1, 0, 0) + AX.quot(MQ_R) * (w(0, 0, 0) - w(1, 0, 0));
      const auto wu_s = w(1, 0, -1) + AX.quot(MQ_R) * (w(0, 0, -1) - w(1, 0, -1));
      const auto w_in_um = HALF * (wu_n + wu_s);
      T duudx, dvudy, dwudz;
      const bool third = (i > 2 && i < nx_var && j > 2 && j < ny_var + 1 && k > 2 && k < nz_var + 1) &&
                         !near_ib && !near_ts2;
      if (third) {
        duudx =
            AX.div(u(0, 0, 0) * (AX.coef(0, 1) * u(2, 0, 0) + AX.coef(0, 2) * u(1, 0, 0) + AX.coef(0, 3) * u(0, 0, 0) + AX.coef(0, 4) * u(-1, 0, 0) + AX.coef(0, 5) * u(-2, 0, 0)), MD_SA) +
            AX.div(fabs(u(0, 0, 0)) * (AX.coef(1, 1) * u(2, 0, 0) + AX.coef(1, 2) * u(1, 0, 0) + AX.coef(1, 3) * u(0, 0, 0) + AX.coef(1, 4) * u(-1, 0, 0) + AX.coef(1, 5) * u(-2, 0, 0)), MD_SK);
        dvudy =
            AY.div(v_in_um * (AY.coef(2, 1) * u(0, 2, 0) + AY.coef(2, 2) * u(0, 1, 0) + AY.coef(2, 3) * u(0, 0, 0) + AY.coef(2, 4) * u(0, -1, 0) + AY.coef(2, 5) * u(0, -2, 0)), MD_XA) +
            AY.div(fabs(v_in_um) * (AY.coef(3, 1) * u(0, 2, 0) + AY.coef(3, 2) * u(0, 1, 0) + AY.coef(3, 3) * u(0, 0, 0) + AY.coef(3, 4) * u(0, -1, 0) + AY.coef(3, 5) * u(0, -2, 0)), MD_XK);
        dwudz =
            AZ.div(w_in_um * (AZ.coef(2, 1) * u(0, 0, 2) + AZ.coef(2, 2) * u(0, 0, 1) + AZ.coef(2, 3) * u(0, 0, 0) + AZ.coef(2, 4) * u(0, 0, -1) + AZ.coef(2, 5) * u(0, 0, -2)), MD_XA) +
            AZ.div(fabs(w_in_um) * (AZ.coef(3, 1) * u(0, 0, 2) + AZ.coef(3, 2) * u(0, 0, 1) + AZ.coef(3, 3) * u(0, 0, 0) + AZ.coef(3, 4) * u(0, 0, -1) + AZ.coef(3, 5) * u(0, 0, -2)), MD_XK);
      } else {
        duudx = AX.div(-Q25 * (u1a * u1a + alpha * fabs(u1a) * u22 - u3 * u3 - alpha * fabs(u3) * u4), MD_D);
        dvudy = AY.div(-Q25 * (v1a * u5 + alpha * fabs(v1a) * u6 - v22 * u7 - alpha * fabs(v22) * u8), MD_D);
        dwudz = AZ.div(-Q25 * (w1a * u9 + alpha * fabs(w1a) * u10 - w22 * u11 - alpha * fabs(w22) * u12), MD_D);
      }
      const auto d2udx2 = AX.quot(MQ_2) * (AX.div(-u4, MD_R) + AX.div(u22, MD_D));
      const auto d2udy2 =
          AY.quot(MQ_C) * (AY.div(-u8, MD_HALF_R) + AY.div(u6, MD_HALF_L));
      const auto d2udz2 =
          AZ.quot(MQ_C) * (AZ.div(-u12, MD_HALF_R) + AZ.div(u10, MD_HALF_L));
      const auto xtt2 = div_re<EXACT>(d2udx2 + d2udy2 + d2udz2, a);
      const auto residu = (-duudx - dvudy - dwudz + xtt2);
      out.put(0, c, u(0, 0, 0) + deltat * (residu + dpdx));
    }
    // ---------------- V momentum ----------------
    if constexpr (OutputOf<Out>::q < 0 || OutputOf<Out>::q == 1) {
      const auto uv_e = u(0, 1, 0) + AY.quot(MQ_R) * (u(0, 0, 0) - u(0, 1, 0));
      const auto uv_w = u(-1, 1, 0) + AY.quot(MQ_R) * (u(-1, 0, 0) - u(-1, 1, 0));
      const auto u_in_vm = HALF * (uv_e + uv_w);
      const auto wv_n = w(0, 1, 0) + AY.quot(MQ_R) * (w(0, 0, 0) - w(0, 1, 0));
      const auto wv_s = w(0, 1, -1) + AY.quot(MQ_R) * (w(0, 0, -1) - w(0, 1, -1));
      const auto w_in_vm = HALF * (wv_n + wv_s);
      T duvdx, dvvdy, dwvdz;
      const bool third = (i > 2 && i < nx_var + 1 && j > 2 && j < ny_var && k > 2 && k < nz_var + 1) &&
                         !near_ib && !near_ts2;
      if (third) {
        duvdx =
            AX.div(u_in_vm * (AX.coef(2, 1) * v(2, 0, 0) + AX.coef(2, 2) * v(1, 0, 0) + AX.coef(2, 3) * v(0, 0, 0) + AX.coef(2, 4) * v(-1, 0, 0) + AX.coef(2, 5) * v(-2, 0, 0)), MD_XA) +
            AX.div(fabs(u_in_vm) * (AX.coef(3, 1) * v(2, 0, 0) + AX.coef(3, 2) * v(1, 0, 0) + AX.coef(3, 3) * v(0, 0, 0) + AX.coef(3, 4) * v(-1, 0, 0) + AX.coef(3, 5) * v(-2, 0, 0)), MD_XK);
        dvvdy =
            AY.div(v(0, 0, 0) * (AY.coef(0, 1) * v(0, 2, 0) + AY.coef(0, 2) * v(0, 1, 0) + AY.coef(0, 3) * v(0, 0, 0) + AY.coef(0, 4) * v(0, -1, 0) + AY.coef(0, 5) * v(0, -2, 0)), MD_SA) +
            AY.div(fabs(v(0, 0, 0)) * (AY.coef(1, 1) * v(0, 2, 0) + AY.coef(1, 2) * v(0, 1, 0) + AY.coef(1, 3) * v(0, 0, 0) + AY.coef(1, 4) * v(0, -1, 0) + AY.coef(1, 5) * v(0, -2, 0)), MD_SK);
        dwvdz =
            AZ.div(w_in_vm * (AZ.coef(2, 1) * v(0, 0, 2) + AZ.coef(2, 2) * v(0, 0, 1) + AZ.coef(2, 3) * v(0, 0, 0) + AZ.coef(2, 4) * v(0, 0, -1) + AZ.coef(2, 5) * v(0, 0, -2)), MD_XA) +
            AZ.div(fabs(w_in_vm) * (AZ.coef(3, 1) * v(0, 0, 2) + AZ.coef(3, 2) * v(0, 0, 1) + AZ.coef(3, 3) * v(0, 0, 0) + AZ.coef(3, 4) * v(0, 0, -1) + AZ.coef(3, 5) * v(0, 0, -2)), MD_XK);
      } else {
        duvdx = AX.div(-Q25 * (u13 * v3 + alpha * fabs(u13) * v4 - u14 * v5 - alpha * fabs(u14) * v6), MD_D);
        dvvdy = AY.div(-Q25 * (v7 * v7 + alpha * fabs(v7) * v8 - v9 * v9 - alpha * fabs(v9) * v10), MD_D);
        dwvdz = AZ.div(-Q25 * (w3 * v11 + alpha * fabs(w3) * v12 - w4 * v13 - alpha * fabs(w4) * v14), MD_D);
      }
      const auto d2vdx2 =
          AX.quot(MQ_C) * (AX.div(-v6, MD_HALF_R) + AX.div(v4, MD_HALF_L));
      const auto d2vdy2 = AY.quot(MQ_2) * (AY.div(-v10, MD_R) + AY.div(v8, MD_D));
      const auto d2vdz2 =
          AZ.quot(MQ_C) * (AZ.div(-v14, MD_HALF_R) + AZ.div(v12, MD_HALF_L));
      const auto ytt2 = div_re<EXACT>(d2vdx2 + d2vdy2 + d2vdz2, a);
      const auto residv = (-duvdx - dvvdy - dwvdz + ytt2);
      out.put(1, c, v(0, 0, 0) + deltat * (residv + dpdy));
    }
    // ---------------- W momentum ----------------
    if constexpr (OutputOf<Out>::q < 0 || OutputOf<Out>::q == 2) {
      const auto uw_e = u(0, 0, 1) + AZ.quot(MQ_R) * (u(0, 0, 0) - u(0, 0, 1));
      const auto uw_w = u(-1, 0, 1) + AZ.quot(MQ_R) * (u(-1, 0, 0) - u(-1, 0, 1));
      const auto u_in_wm = HALF * (uw_e + uw_w);
      const auto vw_n = v(0, 0, 1) + AZ.quot(MQ_R) * (v(0, 0, 0) - v(0, 0, 1));
      const auto vw_s = v(0, -1, 1) + AZ.quot(MQ_R) * (v(0, -1, 0) - v(0, -1, 1));
      const auto v_in_wm = HALF * (vw_n + vw_s);
      T duwdx, dvwdy, dwwdz;
      const bool third = (i > 2 && i < nx_var + 1 && j > 2 && j < ny_var + 1 && k > 2 && k < nz_var) &&
                         !near_ib && !near_ts2;
      if (third) {
        duwdx =
            AX.div(u_in_wm * (AX.coef(2, 1) * w(2, 0, 0) + AX.coef(2, 2) * w(1, 0, 0) + AX.coef(2, 3) * w(0, 0, 0) + AX.coef(2, 4) * w(-1, 0, 0) + AX.coef(2, 5) * w(-2, 0, 0)), MD_XA) +
            AX.div(fabs(u_in_wm) * (AX.coef(3, 1) * w(2, 0, 0) + AX.coef(3, 2) * w(1, 0, 0) + AX.coef(3, 3) * w(0, 0, 0) + AX.coef(3, 4) * w(-1, 0, 0) + AX.coef(3, 5) * w(-2, 0, 0)), MD_XK);
        dvwdy =
            AY.div(v_in_wm * (AY.coef(2, 1) * w(0, 2, 0) + AY.coef(2, 2) * w(0, 1, 0) + AY.coef(2, 3) * w(0, 0, 0) + AY.coef(2, 4) * w(0, -1, 0) + AY.coef(2, 5) * w(0, -2, 0)), MD_XA) +
            AY.div(fabs(v_in_wm) * (AY.coef(3, 1) * w(0, 2, 0) + AY.coef(3, 2) * w(0, 1, 0) + AY.coef(3, 3) * w(0, 0, 0) + AY.coef(3, 4) * w(0, -1, 0) + AY.coef(3, 5) * w(0, -2, 0)), MD_XK);
        dwwdz =
            AZ.div(w(0, 0, 0) * (AZ.coef(0, 1) * w(0, 0, 2) + AZ.coef(0, 2) * w(0, 0, 1) + AZ.coef(0, 3) * w(0, 0, 0) + AZ.coef(0, 4) * w(0, 0, -1) + AZ.coef(0, 5) * w(0, 0, -2)), MD_SA) +
            AZ.div(fabs(w(0, 0, 0)) * (AZ.coef(1, 1) * w(0, 0, 2) + AZ.coef(1, 2) * w(0, 0, 1) + AZ.coef(1, 3) * w(0, 0, 0) + AZ.coef(1, 4) * w(0, 0, -1) + AZ.coef(1, 5) * w(0, 0, -2)), MD_SK);
      } else {
        duwdx = AX.div(-HALF * (u15 * w5 + alpha * fabs(u15) * w6 - u16 * w7 - alpha * fabs(u16) * w8), MD_D);
        dvwdy = AY.div(-HALF * (v15 * w9 + alpha * fabs(v15) * w10 - v16 * w11 - alpha * fabs(v16) * w12), MD_D);
        dwwdz = AZ.div(-HALF * (w13 * w13 + alpha * fabs(w13) * w14 - w15 * w15 - alpha * fabs(w15) * w16), MD_D);
      }
      const auto d2wdx2 =
          AX.quot(MQ_C) * (AX.div(-w8, MD_HALF_R) + AX.div(w6, MD_HALF_L));
      const auto d2wdy2 =
          AY.quot(MQ_C) * (AY.div(-w12, MD_HALF_R) + AY.div(w10, MD_HALF_L));
      const auto d2wdz2 = AZ.quot(MQ_2) * (AZ.div(-w16, MD_R) + AZ.div(w14, MD_D));
      const auto ztt2 = div_re<EXACT>(d2wdx2 + d2wdy2 + d2wdz2, a);
      const auto residw = (-duwdx - dvwdy - dwwdz + ztt2);
      out.put(2, c, w(0, 0, 0) + deltat * (residw + dpdz));
    }
#undef u
#undef v
#undef w
#undef p
  }
}

template <typename T>
struct MomentumOp {
  MomArgs a;
  __device__ __forceinline__ static auto reader(const DevBlock& B) {
    if constexpr (std::is_same<T, FastF>::value) return PlainReaderF{{B.mf[0], B.mf[1], B.mf[2], B.mf[3]}};
    else return PlainReader{{B.u, B.v, B.w, B.p}};
  }
  __device__ void run(const DevBlock& B, int cta, int ncta) const {
    const auto rd = reader(B);
    FOR_INTERIOR(B, cta, ncta) {
      INTERIOR_CELL(B);
      if (B.cell[c] != 0) continue;
      if (B.tsnear[c]) continue;  // done by MomentumTsOp
      momentum_cell<T>(B, a, i, j, k, c, rd, StoreOut{B.ut, B.vt, B.wt});
    }
  }
};

// u,v,w,p rounded to FP32 once per point: the FP32 stencil reads each value
// about 77 times, and GB300 converts FP64 to FP32 in the FP64 pipe (two lanes
// per cycle and SM), where those conversions alone took half of its time
struct CvtOp {
  __device__ void run(const DevBlock& B, int cta, int ncta) const {
    const int64_t n = B.d.npts(), step = (int64_t)ncta * blockDim.x;
    for (int64_t t = (int64_t)cta * blockDim.x + threadIdx.x; t < n; t += step) {
      B.mf[0][t] = (float)B.u[t];
      B.mf[1][t] = (float)B.v[t];
      B.mf[2][t] = (float)B.w[t];
      B.mf[3][t] = (float)B.p[t];
    }
  }
};

// ---------------------------------------------------------------------------
// Thin-surface overlay.  Every position the reference substitutes or
// restores is one of a TS cell T's seven own positions; the kind K of the
// position fixes the ghost slot, the element list and the face coordinate of
// its sign test:
//   U2 u(T), U1 u(T-ex), V2 v(T), V1 v(T-ey), W2 w(T), W1 w(T-ez), P p(T).
// A fluid cell F whose +d neighbour is T handles six of them (direction d
// excludes one kind: +x U1, -x U2, +y V1, -y V2, +z W1, -z W2):
//  * before its stencil it writes kind K with ghost_K(nn) for the last TS
//    list entry nn whose sign test at F's own face is negative (the test does
//    not depend on which TS cell is F's neighbour);
//  * after its stencil it restores kind K with tghost_K(n_ts), the saved value
//    of the last TS entry (the index the reference's loop leaves behind).
// So a cell G reads position X as: its own write if it made one, else the
// restore of the latest fluid cell before G (list order = linear index order)
// that restores X, else the original value; and after the loop X holds the
// restore of the latest restorer overall (k_ts_restore).
// ---------------------------------------------------------------------------
enum TsKind { K_U2 = 0, K_U1, K_V2, K_V1, K_W2, K_W1, K_P, N_KIND };

__device__ __forceinline__ int ghost_slot(int K) {
  // ghost[] order: p, pt, u2, u2t, v2, v2t, w2, w2t, u1, u1t, v1, v1t, w1, w1t
  return K == K_P ? G_P : (K & 1) ? (G_U1 + 2 * (K >> 1)) : (G_U2 + 2 * (K >> 1));
}
__device__ __forceinline__ int nel_slot(int K) {
  // nel[] order: p, u1, u2, v1, v2, w1, w2
  return K == K_P ? N_P : (N_U1 + 2 * (K >> 1) + ((K & 1) ? 0 : 1));
}
// the kind direction d (0..5 = +x,-x,+y,-y,+z,-z) does not handle
__device__ __forceinline__ int excluded_kind(int dir) {
  return 2 * (dir >> 1) + ((dir & 1) ? 0 : 1);
}
__device__ __forceinline__ void dir_vec(int dir, int& a, int& b, int& e) {
  const int s = (dir & 1) ? -1 : 1;
  a = (dir >> 1) == 0 ? s : 0;
  b = (dir >> 1) == 1 ? s : 0;
  e = (dir >> 1) == 2 ? s : 0;
}

// latest restorer F (linear index < before) of position kind K of TS cell T;
// updates best / val / kind
__device__ __forceinline__ void latest_restore(const DevBlock& B, int ti, int tj, int tk, int K,
                                               int64_t before, const double* rconst, int64_t& best,
                                               double& val, int& kind) {
  const Dims& d = B.d;
#pragma unroll
  for (int dir = 0; dir < 6; ++dir) {
    if (K == excluded_kind(dir)) continue;
    int a, b, e;
    dir_vec(dir, a, b, e);
    // F's +dir neighbour is T
    const int fi = ti - a, fj = tj - b, fk = tk - e;
    if (fi < 2 || fj < 2 || fk < 2 || fi > d.nx + 1 || fj > d.ny + 1 || fk > d.nz + 1) continue;
    const int64_t lf = d.idx(fi, fj, fk);
    if (lf >= before || lf <= best) continue;
    if (B.cell[lf] != 0) continue;
    best = lf;
    val = rconst[K];
    kind = K;
  }
}

// the (up to two) TS cells and kinds a position of field q belongs to
__device__ __forceinline__ int owners(const DevBlock& B, int q, int xi, int xj, int xk, int ot[2][4]) {
  const Dims& d = B.d;
  int n = 0;
  auto ts = [&](int a, int b, int e) {
    return a >= 1 && b >= 1 && e >= 1 && a <= d.nx + 3 && b <= d.ny + 3 && e <= d.nz + 3 &&
           B.cell2[d.idx3(a, b, e)] == 2;
  };
  if (q == 3) {
    if (ts(xi, xj, xk)) { ot[n][0] = xi; ot[n][1] = xj; ot[n][2] = xk; ot[n][3] = K_P; ++n; }
    return n;
  }
  if (ts(xi, xj, xk)) { ot[n][0] = xi; ot[n][1] = xj; ot[n][2] = xk; ot[n][3] = 2 * q; ++n; }
  const int ai = xi + (q == 0), aj = xj + (q == 1), ak = xk + (q == 2);
  if (ts(ai, aj, ak)) { ot[n][0] = ai; ot[n][1] = aj; ot[n][2] = ak; ot[n][3] = 2 * q + 1; ++n; }
  return n;
}

// One read of position x (field q) by cell G near TS cells, in the
// reference's serial order: the value and where it came from (how 0: the
// array, 1: G's own substitution of kind K, the ghost value of TS entry
// last[K]; 2: the restore of kind K, the t-ghost value of the last entry).
struct TsHit {
  double v;
  int how, K;
};
// not inlined: one copy of the overlay logic serves all ~150 stencil reads
__device__ __noinline__ TsHit ts_read(const DevBlock& B, int gi, int gj, int gk, int64_t glin, const int* last,
                                      const double* rconst, int q, int xi, int xj, int xk, int64_t x) {
  const double* f = q == 0 ? B.u : q == 1 ? B.v : q == 2 ? B.w : B.p;
  const double orig = __ldg(f + x);
  int ot[2][4];
  const int n = owners(B, q, xi, xj, xk, ot);
  if (n == 0) return TsHit{orig, 0, 0};
  // own substitution: T is an axis neighbour of G and the direction handles K
  for (int m = 0; m < n; ++m) {
    const int di = ot[m][0] - gi, dj = ot[m][1] - gj, dk = ot[m][2] - gk;
    const int ad = abs(di) + abs(dj) + abs(dk);
    if (ad != 1) continue;
    const int dir = di ? (di > 0 ? 0 : 1) : dj ? (dj > 0 ? 2 : 3) : (dk > 0 ? 4 : 5);
    const int K = ot[m][3];
    if (K == excluded_kind(dir)) continue;
    if (last[K] >= 0) return TsHit{B.ghost[ghost_slot(K)][last[K]], 1, K};
  }
  int64_t best = -1;
  double val = orig;
  int kind = 0;
  for (int m = 0; m < n; ++m)
    latest_restore(B, ot[m][0], ot[m][1], ot[m][2], ot[m][3], glin, rconst, best, val, kind);
  return best >= 0 ? TsHit{val, 2, kind} : TsHit{orig, 0, 0};
}

// Reads of a cell G near TS cells, in the reference's serial order.
struct TsReader {
  const DevBlock* B;
  int gi, gj, gk;
  int64_t glin;
  int last[N_KIND];      // own substitution: last TS entry with a negative test, -1: none
  double rconst[N_KIND]; // restore value of each kind
  __device__ __forceinline__ double get(int q, int xi, int xj, int xk, int64_t x) const {
    return ts_read(*B, gi, gj, gk, glin, last, rconst, q, xi, xj, xk, x).v;
  }
};

__device__ __forceinline__ void restore_consts(const DevBlock& B, int nts, double* rc) {
#pragma unroll
  for (int K = 0; K < N_KIND; ++K) rc[K] = nts > 0 ? B.ghost[ghost_slot(K) + 1][nts - 1] : 0.0;
}

// sign tests of src/NavierStokes.f90:321-354 for every TS entry: the last
// entry with a negative test, per kind.  The reference's loop keeps the last
// hit, so the entries are visited from the end and each kind stops at its
// first hit: the same entry, the same sign test arithmetic, and usually a few
// entries instead of all of them.
__device__ void own_substitution(const DevBlock& B, int i, int j, int k, int nts, int* last) {
  const double X[N_KIND] = {B.x1[i], B.x1[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1]};
  const double Y[N_KIND] = {B.yp[j - 1], B.yp[j - 1], B.y1[j], B.y1[j - 1], B.yp[j - 1], B.yp[j - 1], B.yp[j - 1]};
  const double Z[N_KIND] = {B.zp[k - 1], B.zp[k - 1], B.zp[k - 1], B.zp[k - 1], B.z1[k], B.z1[k - 1], B.zp[k - 1]};
#pragma unroll
  for (int K = 0; K < N_KIND; ++K) last[K] = -1;
  unsigned open = (1u << N_KIND) - 1u;  // kinds still without a hit
  for (int nn = nts - 1; nn >= 0 && open; --nn) {
    const int bt = B.ts_idx[nn] - 1;
#pragma unroll
    for (int K = 0; K < N_KIND; ++K) {
      if (!(open & (1u << K))) continue;
      const int e = B.nel[nel_slot(K)][bt] - 1;
      const double t = (X[K] - B.xcent[e]) * B.cosA[e] + (Y[K] - B.ycent[e]) * B.cosB[e] +
                       (Z[K] - B.zcent[e]) * B.cosG[e];
      if (t < 0) {
        last[K] = nn;
        open &= ~(1u << K);
      }
    }
  }
}

// own_substitution of one cell by a whole warp, 32 entries at a time; lane 0
// writes the entries to last[]
__device__ __forceinline__ void own_substitution_warp(const DevBlock& B, int i, int j, int k, int nts, int* last) {
  const int lane = threadIdx.x & 31;
  const double X[N_KIND] = {B.x1[i], B.x1[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1], B.xp[i - 1]};
  const double Y[N_KIND] = {B.yp[j - 1], B.yp[j - 1], B.y1[j], B.y1[j - 1], B.yp[j - 1], B.yp[j - 1], B.yp[j - 1]};
  const double Z[N_KIND] = {B.zp[k - 1], B.zp[k - 1], B.zp[k - 1], B.zp[k - 1], B.z1[k], B.z1[k - 1], B.zp[k - 1]};
  unsigned open = (1u << N_KIND) - 1u;
  for (int base = nts - 1; base >= 0 && open; base -= 32) {
    const int nn = base - lane;
    const int bt = nn >= 0 ? B.ts_idx[nn] - 1 : 0;
#pragma unroll
    for (int K = 0; K < N_KIND; ++K) {
      if (!(open & (1u << K))) continue;
      bool hit = false;
      if (nn >= 0) {
        const int e = B.nel[nel_slot(K)][bt] - 1;
        const double t = (X[K] - B.xcent[e]) * B.cosA[e] + (Y[K] - B.ycent[e]) * B.cosB[e] +
                         (Z[K] - B.zcent[e]) * B.cosG[e];
        hit = t < 0;
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit);
      if (hits) {
        if (lane == 0) last[K] = base - (__ffs(hits) - 1);
        open &= ~(1u << K);
      }
    }
  }
  if (lane == 0)
#pragma unroll
    for (int K = 0; K < N_KIND; ++K)
      if (open & (1u << K)) last[K] = -1;
}

// The cells near TS cells.  A CTA's cells next to one search their
// substituting entries warp by warp before the stencils run: the search goes
// back through the list until each kind has hit, mostly one entry but up to
// thousands, and one thread per cell left the kernel waiting for its longest
// search (256x192x192 plate block, 6709 entries: 3.35 -> 1.16 ms).
template <typename T>
struct MomentumTsOp {
  MomArgs a;
  __device__ void run(const DevBlock& B, int cta, int ncta) const {
    constexpr int NT = 128;
    __shared__ int s_last[NT][N_KIND], s_list[NT], s_n;
    const Dims& d = B.d;
    const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
    if (nts == 0) return;  // no cell is near one
    const int64_t n = (int64_t)d.nx * d.ny * d.nz;
    // 32-bit divisions when the interior count fits them
    auto cell_at = [&](int64_t t, int& i, int& j, int& k) {
      if (n <= 0x7fffffffLL) {
        const unsigned r = (unsigned)t / (unsigned)d.nx;
        i = 2 + (int)((unsigned)t - r * (unsigned)d.nx);
        k = 2 + (int)(r / (unsigned)d.ny);
        j = 2 + (int)(r - (unsigned)(k - 2) * (unsigned)d.ny);
      } else {
        i = 2 + (int)(t % d.nx);
        const int64_t r = t / d.nx;
        j = 2 + (int)(r % d.ny);
        k = 2 + (int)(r / d.ny);
      }
    };
    for (int64_t t0 = (int64_t)cta * NT; t0 < n; t0 += (int64_t)ncta * NT) {
      const int64_t t = t0 + threadIdx.x;
      int i = 2, j = 2, k = 2;
      if (t < n) cell_at(t, i, j, k);
      const int64_t c = d.idx(i, j, k);
      const bool near = t < n && B.tsnear[c] && B.cell[c] == 0;
      if (threadIdx.x == 0) s_n = 0;
      if (!__syncthreads_or(near)) continue;
      const bool adj = near && !adj_ok(B.cell2, d, true, i, j, k, 1);
      if (adj) s_list[atomicAdd(&s_n, 1)] = threadIdx.x;
      __syncthreads();
      for (int q = threadIdx.x >> 5; q < s_n; q += NT / 32) {
        int ci, cj, ck;
        cell_at(t0 + s_list[q], ci, cj, ck);
        own_substitution_warp(B, ci, cj, ck, nts, s_last[s_list[q]]);
      }
      __syncthreads();
      if (!near) continue;
      TsReader rd;
      rd.B = &B;
      rd.gi = i;
      rd.gj = j;
      rd.gk = k;
      rd.glin = c;
      restore_consts(B, nts, rd.rconst);
#pragma unroll
      for (int K = 0; K < N_KIND; ++K) rd.last[K] = adj ? s_last[threadIdx.x][K] : -1;
      momentum_cell<T>(B, a, i, j, k, c, rd, StoreOut{B.ut, B.vt, B.wt});
    }
  }
};

// tangent-linear stencil: reads (u,v,w,p) and their tangents
struct DualReader {
  const double* f[4];
  const double* df[4];
  __device__ __forceinline__ Dual get(int q, int, int, int, int64_t x) const {
    return Dual(__ldg(f[q] + x), __ldg(df[q] + x));
  }
};

// DualOut that notes whether a value is not finite
struct DualOutChecked {
  DualOut o;
  bool* bad;
  __device__ __forceinline__ void put(int q, int64_t c, Dual val) const {
    o.put(q, c, val);
    *bad |= not_finite(val.v);
  }
};

struct MomentumTlmOp {
  MomArgs a;
  const double* du[4];
  double *ut, *vt, *wt, *dut, *dvt, *dwt;
  __device__ void run(const DevBlock& B, int cta, int ncta) const {
    const DualReader rd{{B.u, B.v, B.w, B.p}, {du[0], du[1], du[2], du[3]}};
    const DualOut out{ut, vt, wt, dut, dvt, dwt};
    FOR_INTERIOR(B, cta, ncta) {
      INTERIOR_CELL(B);
      if (B.cell[c] != 0) continue;
      if (B.tsnear[c]) {
        set_err(B.err, BCFD_E_STATE);  // the thin-surface overlay has no tangent model
        continue;
      }
      bool bad = false;
      momentum_cell<Dual>(B, a, i, j, k, c, rd, DualOutChecked{out, &bad});
      if (bad) momentum_cell<Dual, true>(B, a, i, j, k, c, rd, out);
    }
  }
};

// ---------------------------------------------------------------------------
// Adjoint (reverse mode) of the predictor, as a gather: the adjoint of input
// position X of field f is  sum over fluid cells C that read X, over the
// three outputs q, of  seed_q(C) * dF_q(C)/dX_f.  Each partial is the tangent
// of the dual-number stencil at C seeded with 1 at (f, X), so it is the exact
// transpose of the tangent-linear model, summed in a fixed order (footprint
// offsets ascending, outputs U,V,W): deterministic, no atomics.
// The footprint (the (field, offset) pairs the stencil reads, offsets in
// [-2,2]^3) is collected once per call from the block's own branches.
// ---------------------------------------------------------------------------
constexpr int kFootWords = 16;  // 4 fields x 125 offsets, 4 words per field

struct FootReader {
  const double* f[4];
  uint32_t* m;  // per-thread mask
  int ci, cj, ck;
  int* err;
  __device__ __forceinline__ double get(int q, int ii, int jj, int kk, int64_t x) const {
    const int a = ii - ci, b = jj - cj, e = kk - ck;
    if (a < -2 || a > 2 || b < -2 || b > 2 || e < -2 || e > 2) {
      set_err(err, BCFD_E_STATE);  // a read outside [-2,2]^3 (none in the stencil)
    } else {
      const int o = (a + 2) + 5 * (b + 2) + 25 * (e + 2);
      m[4 * q + (o >> 5)] |= 1u << (o & 31);
    }
    return __ldg(f[q] + x);
  }
};
struct FiniteOut {  // whether an output is not finite
  bool* bad;
  __device__ __forceinline__ void put(int, int64_t, double v) const { *bad |= not_finite(v); }
};
// bit of foot[3] past the 125 offsets: a seed or an output is not finite
constexpr uint32_t kFootNonFinite = 0x80000000u;

// the footprint of a cell near TS cells: its reads go through the overlay,
// so its branches are those of the forward loop
struct FootTsReader {
  const DevBlock* B;
  int gi, gj, gk;
  int64_t glin;
  const int* last;
  const double* rconst;
  uint32_t* m;
  __device__ __forceinline__ double get(int q, int ii, int jj, int kk, int64_t x) const {
    const int a = ii - gi, b = jj - gj, e = kk - gk;
    if (a < -2 || a > 2 || b < -2 || b > 2 || e < -2 || e > 2) {
      set_err(B->err, BCFD_E_STATE);
    } else {
      const int o = (a + 2) + 5 * (b + 2) + 25 * (e + 2);
      m[4 * q + (o >> 5)] |= 1u << (o & 31);
    }
    return ts_read(*B, gi, gj, gk, glin, last, rconst, q, ii, jj, kk, x).v;
  }
};

// ts_last: per point, the own-substitution entries of the cells near TS
// cells (k_ts_last); nullptr: such cells are skipped
__global__ void k_mom_footprint(DevBlock B, MomArgs a, uint32_t* foot, const double* ubar_t, const double* vbar_t,
                                const double* wbar_t, const int* ts_last) {
  bool bad = false;
  uint32_t m[kFootWords];
#pragma unroll
  for (int w = 0; w < kFootWords; ++w) m[w] = 0u;
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  double rc[N_KIND];
  restore_consts(B, nts, rc);
  const int64_t n = (int64_t)d.nx * d.ny * d.nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = 2 + (int)(t % d.nx);
    const int64_t r = t / d.nx;
    const int j = 2 + (int)(r % d.ny), k = 2 + (int)(r / d.ny);
    const int64_t c = d.idx(i, j, k);
    if (B.cell[c] != 0) continue;
    bad |= not_finite(__ldg(ubar_t + c)) || not_finite(__ldg(vbar_t + c)) || not_finite(__ldg(wbar_t + c));
    if (B.tsnear[c]) {
      if (!ts_last) continue;
      const FootTsReader rd{&B, i, j, k, c, ts_last + N_KIND * c, rc, m};
      momentum_cell<double>(B, a, i, j, k, c, rd, FiniteOut{&bad});
      continue;
    }
    const FootReader rd{{B.u, B.v, B.w, B.p}, m, i, j, k, B.err};
    momentum_cell<double>(B, a, i, j, k, c, rd, FiniteOut{&bad});
  }
  if (bad) m[3] |= kFootNonFinite;
#pragma unroll
  for (int w = 0; w < kFootWords; ++w) {
    uint32_t v = m[w];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, s);
    if ((threadIdx.x & 31) == 0 && v) atomicOr(foot + w, v);
  }
}

// four-lane dual reader: lane f carries the seed 1 at (field f, linear index sx)
struct SeedReader4 {
  const double* f[4];
  int64_t sx;
  __device__ __forceinline__ Dual4 get(int q, int, int, int, int64_t x) const {
    Dual4 r(__ldg(f[q] + x));
    if (x == sx) r.d[q] = 1.0;
    return r;
  }
};
// the same for a cell near TS cells: a read the overlay redirects to a ghost
// or t-ghost value does not depend on the array value at x
struct TsSeedReader4 {
  const DevBlock* B;
  int gi, gj, gk;
  int64_t glin;
  const int* last;
  const double* rconst;
  int64_t sx;
  __device__ __forceinline__ Dual4 get(int q, int xi, int xj, int xk, int64_t x) const {
    const TsHit h = ts_read(*B, gi, gj, gk, glin, last, rconst, q, xi, xj, xk, x);
    Dual4 r(h.v);
    if (h.how == 0 && x == sx) r.d[q] = 1.0;
    return r;
  }
};
// lanes on the ghost scalars a cell near TS cells reads: scalar s (0..6 the
// own substitution of kind s, 7..13 the restore of kind s - 7) is lane
// s - 4 pass of the pass
struct TsGhostReader4 {
  const DevBlock* B;
  int gi, gj, gk;
  int64_t glin;
  const int* last;
  const double* rconst;
  int pass;
  __device__ __forceinline__ Dual4 get(int q, int xi, int xj, int xk, int64_t x) const {
    const TsHit h = ts_read(*B, gi, gj, gk, glin, last, rconst, q, xi, xj, xk, x);
    Dual4 r(h.v);
    if (h.how) {
      const int l = (h.how == 1 ? h.K : N_KIND + h.K) - 4 * pass;
      if (l >= 0 && l < 4) r.d[l] = 1.0;
    }
    return r;
  }
};

// adds seed_q(C) * dF_q(C)/dX_f to field f's sum, for the fields whose
// footprint holds this offset (the others' partials are zero)
struct AdjOut4 {
  const double* sb[3];
  double* acc;
  unsigned fmask;
  __device__ __forceinline__ void put(int q, int64_t c, const Dual4& val) const {
    const double s = __ldg(sb[q] + c);
#pragma unroll
    for (int f = 0; f < 4; ++f)
      if ((fmask >> f) & 1u) acc[f] += s * val.d[f];
  }
};

// Which reads an output depends on: itself along the axes up to distance 2;
// another velocity component f at 0 or -1 along f's axis and 0 or 1 along its
// own; the pressure at 0 or 1 along its own axis.
__host__ __device__ constexpr bool mom_reads(int q, int f, int a, int b, int e) {
  const int o[3] = {a, b, e};
  if (f == q) return (a != 0) + (b != 0) + (e != 0) <= 1;
  for (int x = 0; x < 3; ++x) {
    const int lo = x == f ? -1 : 0, hi = x == q ? 1 : 0;
    if (o[x] < lo || o[x] > hi) return false;
  }
  return true;
}
__host__ __device__ constexpr bool mom_reads_any(int q, int a, int b, int e) {
  return mom_reads(q, 0, a, b, e) || mom_reads(q, 1, a, b, e) || mom_reads(q, 2, a, b, e) || mom_reads(q, 3, a, b, e);
}
__host__ __device__ constexpr int off_x(int o) { return o % 5 - 2; }
__host__ __device__ constexpr int off_y(int o) { return o / 5 % 5 - 2; }
__host__ __device__ constexpr int off_z(int o) { return o / 25 - 2; }

// the fluid cell that reads point (xi,xj,xk) at offset o, -1: none
__device__ __forceinline__ int64_t reading_cell(const DevBlock& B, int o, int xi, int xj, int xk) {
  const Dims& d = B.d;
  const int ci = xi - off_x(o), cj = xj - off_y(o), ck = xk - off_z(o);
  if (ci < 2 || ci > d.nx + 1 || cj < 2 || cj > d.ny + 1 || ck < 2 || ck > d.nz + 1) return -1;
  const int64_t c = d.idx(ci, cj, ck);
  return B.cell[c] != 0 ? -1 : c;
}
template <int... O>
__device__ __forceinline__ bool any_near_ts(const DevBlock& B, int xi, int xj, int xk,
                                            std::integer_sequence<int, O...>) {
  bool near = false;
  auto at = [&](auto oc) {
    constexpr int o = decltype(oc)::value, a = off_x(o), b = off_y(o), e = off_z(o);
    if constexpr (mom_reads_any(0, a, b, e) || mom_reads_any(1, a, b, e) || mom_reads_any(2, a, b, e)) {
      const int64_t c = reading_cell(B, o, xi, xj, xk);
      near = near || (c >= 0 && B.tsnear[c]);
    }
  };
  (at(std::integral_constant<int, O>{}), ...);
  return near;
}
using FootOffsets = std::make_integer_sequence<int, 125>;

// seed_Q(C) * dF_Q(C)/dX_F of the cell C that reads X at offset O
template <int Q, int F, int O>
__device__ __forceinline__ void adj_term(const DevBlock& B, const MomArgs& a, int ci, int cj, int ck, int64_t c,
                                         bool ok, double s, double* acc) {
  if constexpr (mom_reads(Q, F, off_x(O), off_y(O), off_z(O))) {
    double t = 0.0;
    const StaticSeed<F, off_x(O), off_y(O), off_z(O)> rd{{B.u, B.v, B.w, B.p}, ok};
    momentum_cell<Dual>(B, a, ci, cj, ck, c, rd, TangentOut<Q>{&t});
    acc[F] += s * t;
  }
}
template <int Q, int O>
__device__ __forceinline__ void adj_output(const DevBlock& B, const MomArgs& a, int ci, int cj, int ck, int64_t c,
                                           bool ok, const double* sb, double* acc) {
  if constexpr (mom_reads_any(Q, off_x(O), off_y(O), off_z(O))) {
    const double s = __ldg(sb + c);
    adj_term<Q, 0, O>(B, a, ci, cj, ck, c, ok, s, acc);
    adj_term<Q, 1, O>(B, a, ci, cj, ck, c, ok, s, acc);
    adj_term<Q, 2, O>(B, a, ci, cj, ck, c, ok, s, acc);
    adj_term<Q, 3, O>(B, a, ci, cj, ck, c, ok, s, acc);
  }
}
template <int O>
__device__ __forceinline__ void adj_offset(const DevBlock& B, const MomArgs& a, int xi, int xj, int xk,
                                           const double* s0, const double* s1, const double* s2, double* acc) {
  constexpr int x = off_x(O), y = off_y(O), z = off_z(O);
  if constexpr (mom_reads_any(0, x, y, z) || mom_reads_any(1, x, y, z) || mom_reads_any(2, x, y, z)) {
    const int64_t c = reading_cell(B, O, xi, xj, xk);
    if (c < 0) return;
    const int ci = xi - x, cj = xj - y, ck = xk - z;
    const bool ok = mom_smooth(B, ci, cj, ck);
    adj_output<0, O>(B, a, ci, cj, ck, c, ok, s0, acc);
    adj_output<1, O>(B, a, ci, cj, ck, c, ok, s1, acc);
    adj_output<2, O>(B, a, ci, cj, ck, c, ok, s2, acc);
  }
}
template <int... O>
__device__ __forceinline__ void adj_offsets(const DevBlock& B, const MomArgs& a, int xi, int xj, int xk,
                                            const double* s0, const double* s1, const double* s2, double* acc,
                                            std::integer_sequence<int, O...>) {
  (adj_offset<O>(B, a, xi, xj, xk, s0, s1, s2, acc), ...);
}

// The gather with every seed known at compile time, for the points that no
// cell near a TS cell reads, when all seeds and outputs are finite.  An
// evaluation carrying four seeds through all three outputs at each of the 19
// offsets spends its FP64 instructions on tangents that are structurally
// zero: 69 (output, field, offset) triples of the 228 can be nonzero, and of
// each only the few terms that hold the seed.  Here the 69 are written out by
// the compiler, a value without a tangent is a plain number, and what the
// tangent does not need is not computed.  The terms left out are zeros times
// finite numbers and the sums keep their order, so the results are the same
// bits; where a value is not finite they are not zeros, and k_mom_adjoint
// takes all points instead.
// (80 registers against 255 with spills; bound by the FP64 pipe; gradient of
// drag and lift through two steps of a 48^3 sphere: 64.6 -> 45.1 ms, the two
// calls' 22 ms of it nearly gone)
__global__ void __launch_bounds__(128) k_mom_adjoint_static(DevBlock B, MomArgs a, const uint32_t* __restrict__ foot,
                                                            const double* ubar_t, const double* vbar_t,
                                                            const double* wbar_t, double* ub, double* vb,
                                                            double* wb, double* pb) {
  if (__ldg(foot + 3) & kFootNonFinite) return;
  const Dims& d = B.d;
  const int64_t n = d.npts();
  const bool ts = B.cnt[C_TS] != 0;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    const int xi = 1 + (int)(x % d.NX);
    const int64_t r = x / d.NX;
    const int xj = 1 + (int)(r % d.NY), xk = 1 + (int)(r / d.NY);
    if (ts && any_near_ts(B, xi, xj, xk, FootOffsets{})) continue;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    adj_offsets(B, a, xi, xj, xk, ubar_t, vbar_t, wbar_t, acc, FootOffsets{});
    ub[x] += acc[0];
    vb[x] += acc[1];
    wb[x] += acc[2];
    pb[x] += acc[3];
  }
}

// The points that k_mom_adjoint_static leaves out: those that cells near TS
// cells read, or (EXACT) all of them when a seed or an output is not finite.
// One dual evaluation per (point, footprint offset) gives the partials of all
// four fields at that point; each field's sum takes the offsets in ascending
// order and, within one, the outputs U, V, W: the order of one evaluation per
// field and offset, so the sums are those of four single-seed gathers.
template <bool EXACT>
__global__ void __launch_bounds__(128) k_mom_adjoint(DevBlock B, MomArgs a, const uint32_t* __restrict__ foot,
                                                     const double* ubar_t, const double* vbar_t,
                                                     const double* wbar_t, double* ub, double* vb, double* wb,
                                                     double* pb, const int* ts_last) {
  const Dims& d = B.d;
  const int64_t n = d.npts();
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  if (((__ldg(foot + 3) & kFootNonFinite) != 0) != EXACT) return;
  if (!EXACT && B.cnt[C_TS] == 0) return;
  double rc[N_KIND];
  restore_consts(B, nts, rc);
  uint32_t m[kFootWords];
#pragma unroll
  for (int w = 0; w < kFootWords; ++w) m[w] = __ldg(foot + w);
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    const int xi = 1 + (int)(x % d.NX);
    const int64_t r = x / d.NX;
    const int xj = 1 + (int)(r % d.NY), xk = 1 + (int)(r / d.NY);
    if (!EXACT && !any_near_ts(B, xi, xj, xk, FootOffsets{})) continue;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int o = 0; o < 125; ++o) {
      unsigned fmask = 0u;
#pragma unroll
      for (int f = 0; f < 4; ++f) fmask |= ((m[4 * f + (o >> 5)] >> (o & 31)) & 1u) << f;
      if (!fmask) continue;
      const int ci = xi - (o % 5 - 2), cj = xj - ((o / 5) % 5 - 2), ck = xk - (o / 25 - 2);
      if (ci < 2 || ci > d.nx + 1 || cj < 2 || cj > d.ny + 1 || ck < 2 || ck > d.nz + 1) continue;
      const int64_t c = d.idx(ci, cj, ck);
      if (B.cell[c] != 0) continue;
      if (B.tsnear[c]) {
        if (!ts_last) {
          set_err(B.err, BCFD_E_STATE);  // the overlay's entries are needed
          continue;
        }
        const TsSeedReader4 rd{&B, ci, cj, ck, c, ts_last + N_KIND * c, rc, x};
        momentum_cell<Dual4, EXACT>(B, a, ci, cj, ck, c, rd, AdjOut4{{ubar_t, vbar_t, wbar_t}, acc, fmask});
        continue;
      }
      const SeedReader4 rd{{B.u, B.v, B.w, B.p}, x};
      momentum_cell<Dual4, EXACT>(B, a, ci, cj, ck, c, rd, AdjOut4{{ubar_t, vbar_t, wbar_t}, acc, fmask});
    }
    ub[x] += acc[0];
    vb[x] += acc[1];
    wb[x] += acc[2];
    pb[x] += acc[3];
  }
}

// u,v,w,p at TS positions after the loop: the restore of the latest restorer
struct TsRestoreOp {
  __device__ void run(const DevBlock& B, int cta, int ncta) const {
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  double rc[N_KIND];
  restore_consts(B, nts, rc);
  for (int t = cta * blockDim.x + threadIdx.x; t < nts * N_KIND; t += ncta * blockDim.x) {
    const int nn = t / N_KIND, K = t % N_KIND;
    const int bt = B.ts_idx[nn] - 1;
    const int ti = B.ib_i[bt], tj = B.ib_j[bt], tk = B.ib_k[bt];
    const int q = K == K_P ? 3 : K >> 1;
    const int xi = ti - (K == K_U1), xj = tj - (K == K_V1), xk = tk - (K == K_W1);
    int ot[2][4];
    const int n = owners(B, q, xi, xj, xk, ot);
    int64_t best = -1;
    double val = 0.0;
    int kind = 0;
    for (int m = 0; m < n; ++m)
      latest_restore(B, ot[m][0], ot[m][1], ot[m][2], ot[m][3], INT64_MAX, rc, best, val, kind);
    if (best < 0) continue;
    double* f = q == 0 ? B.u : q == 1 ? B.v : q == 2 ? B.w : B.p;
    f[d.idx(xi, xj, xk)] = val;
  }
  }
};

// ---------------------------------------------------------------------------
// Adjoint of the thin-surface overlay.  A cell near TS cells reads, besides
// array values, 14 scalars: the ghost value of kind K of TS entry last[K]
// (its own substitution) and the t-ghost value of kind K of the last TS entry
// (the restore).  Their adjoints go to the ghost arrays' adjoint gb (14
// arrays of cap entries, the ghost[] order); the loop's final restore is
// transposed first.  Sums in a fixed order: one thread per accumulation.
// ---------------------------------------------------------------------------

// the own-substitution entries of every fluid cell near TS cells
__global__ void k_ts_last(DevBlock B, int* last) {
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  const int64_t n = (int64_t)d.nx * d.ny * d.nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = 2 + (int)(t % d.nx);
    const int64_t r = t / d.nx;
    const int j = 2 + (int)(r % d.ny), k = 2 + (int)(r / d.ny);
    const int64_t c = d.idx(i, j, k);
    if (B.cell[c] != 0 || !B.tsnear[c]) continue;
    int l[N_KIND];
    if (!adj_ok(B.cell2, d, true, i, j, k, 1)) {
      own_substitution(B, i, j, k, nts, l);
    } else {
#pragma unroll
      for (int K = 0; K < N_KIND; ++K) l[K] = -1;
    }
#pragma unroll
    for (int K = 0; K < N_KIND; ++K) last[N_KIND * c + K] = l[K];
  }
}

// per fluid cell near TS cells: seed . dF/d(scalar s) for its 14 scalars
// (EXACT: when a seed or an output is not finite)
template <bool EXACT>
__global__ void __launch_bounds__(128) k_mom_ghost_contrib(DevBlock B, MomArgs a, const uint32_t* __restrict__ foot,
                                                           const int* last,
                                                           const double* ubar_t, const double* vbar_t,
                                                           const double* wbar_t, double* contrib) {
  if (((__ldg(foot + 3) & kFootNonFinite) != 0) != EXACT) return;
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  double rc[N_KIND];
  restore_consts(B, nts, rc);
  const int64_t n = (int64_t)d.nx * d.ny * d.nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = 2 + (int)(t % d.nx);
    const int64_t r = t / d.nx;
    const int j = 2 + (int)(r % d.ny), k = 2 + (int)(r / d.ny);
    const int64_t c = d.idx(i, j, k);
    if (B.cell[c] != 0 || !B.tsnear[c]) continue;
    for (int pass = 0; pass < 4; ++pass) {
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      const TsGhostReader4 rd{&B, i, j, k, c, last + N_KIND * c, rc, pass};
      momentum_cell<Dual4, EXACT>(B, a, i, j, k, c, rd, AdjOut4{{ubar_t, vbar_t, wbar_t}, acc, 0xFu});
#pragma unroll
      for (int l = 0; l < 4; ++l)
        if (4 * pass + l < 2 * N_KIND) contrib[2 * N_KIND * c + 4 * pass + l] = acc[l];
    }
  }
}

// the cells near TS cells in list (linear index) order, inside the box of the
// TS cells grown by the stencil's reach: contributions into gb
__global__ void k_mom_ghost_acc(DevBlock B, const int* last, const double* contrib, double* gb, int64_t cap) {
  if (blockIdx.x || threadIdx.x) return;
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  if (nts <= 0) return;
  int lo[3] = {d.nx + 1, d.ny + 1, d.nz + 1}, hi[3] = {2, 2, 2};
  for (int nn = 0; nn < nts; ++nn) {
    const int bt = B.ts_idx[nn] - 1;
    const int p[3] = {B.ib_i[bt], B.ib_j[bt], B.ib_k[bt]};
    for (int q = 0; q < 3; ++q) {
      lo[q] = min(lo[q], p[q] - 3);
      hi[q] = max(hi[q], p[q] + 3);
    }
  }
  lo[0] = max(lo[0], 2); lo[1] = max(lo[1], 2); lo[2] = max(lo[2], 2);
  hi[0] = min(hi[0], d.nx + 1); hi[1] = min(hi[1], d.ny + 1); hi[2] = min(hi[2], d.nz + 1);
  for (int k = lo[2]; k <= hi[2]; ++k)
    for (int j = lo[1]; j <= hi[1]; ++j)
      for (int i = lo[0]; i <= hi[0]; ++i) {
        const int64_t c = d.idx(i, j, k);
        if (B.cell[c] != 0 || !B.tsnear[c]) continue;
        for (int K = 0; K < N_KIND; ++K) {
          const int l = last[N_KIND * c + K];
          if (l >= 0) gb[ghost_slot(K) * cap + l] += contrib[2 * N_KIND * c + K];
          gb[(ghost_slot(K) + 1) * cap + nts - 1] += contrib[2 * N_KIND * c + N_KIND + K];
        }
      }
}

// the final restore transposed: a restored position's adjoint goes to the
// t-ghost value it received; positions shared by two TS cells are visited
// twice, the second visit adds the zero the first left
__global__ void k_ts_restore_adj(DevBlock B, double* ub, double* vb, double* wb, double* pb, double* gb,
                                 int64_t cap) {
  if (blockIdx.x || threadIdx.x) return;
  const Dims& d = B.d;
  const int nts = (int)min(B.cnt[C_TS], (int64_t)B.cap_ib);
  double rc[N_KIND];
  restore_consts(B, nts, rc);
  for (int t = 0; t < nts * N_KIND; ++t) {
    const int nn = t / N_KIND, K = t % N_KIND;
    const int bt = B.ts_idx[nn] - 1;
    const int ti = B.ib_i[bt], tj = B.ib_j[bt], tk = B.ib_k[bt];
    const int q = K == K_P ? 3 : K >> 1;
    const int xi = ti - (K == K_U1), xj = tj - (K == K_V1), xk = tk - (K == K_W1);
    int ot[2][4];
    const int n = owners(B, q, xi, xj, xk, ot);
    int64_t best = -1;
    double val = 0.0;
    int kind = 0;
    for (int m = 0; m < n; ++m)
      latest_restore(B, ot[m][0], ot[m][1], ot[m][2], ot[m][3], INT64_MAX, rc, best, val, kind);
    if (best < 0) continue;
    double* f = q == 0 ? ub : q == 1 ? vb : q == 2 ? wb : pb;
    const int64_t x = d.idx(xi, xj, xk);
    gb[(ghost_slot(kind) + 1) * cap + nts - 1] += f[x];
    f[x] = 0.0;
  }
}

// velocityBC loop 1 (x faces), src/BoundaryConditions.f90:16-40
__global__ void k_vbc_x(DevBlock B, double deltat, double uc) {
  const Dims& d = B.d;
  const int n = d.ny * d.nz;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int j = 2 + t % d.ny, k = 2 + t / d.ny;
    const int nx = d.nx;
    const int64_t c1 = d.idx(1, j, k), cn = d.idx(nx, j, k), cn1 = d.idx(nx + 1, j, k),
                  cn2 = d.idx(nx + 2, j, k);
    B.ut[c1] = uc;
    B.vt[c1] = -B.vt[cn1];
    B.wt[c1] = -B.wt[cn1];
    B.ut[cn1] = B.u[cn1] - (deltat / B.dxa[nx]) * uc * (B.u[cn1] - B.u[cn]);
    B.vt[cn2] = -B.vt[cn1] + B.v[cn2] + B.v[cn1] -
                (2.0 * deltat / B.dxa[nx + 1]) * uc * (B.v[cn2] - B.v[cn1]);
    B.wt[cn2] = -B.wt[cn1] + B.w[cn2] + B.w[cn1] -
                (2.0 * deltat / B.dxa[nx + 1]) * uc * (B.w[cn2] - B.w[cn1]);
  }
}

// velocityBC loop 2 (y faces), src/BoundaryConditions.f90:42-58
__global__ void k_vbc_y(DevBlock B) {
  const Dims& d = B.d;
  const int n = d.nx * d.nz;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int i = 2 + t % d.nx, k = 2 + t / d.nx;
    const int ny = d.ny;
    B.ut[d.idx(i, 1, k)] = B.ut[d.idx(i, 2, k)];
    B.wt[d.idx(i, 1, k)] = B.wt[d.idx(i, 2, k)];
    B.vt[d.idx(i, 2, k)] = 0.0;
    B.ut[d.idx(i, ny + 2, k)] = B.ut[d.idx(i, ny + 1, k)];
    B.wt[d.idx(i, ny + 2, k)] = B.wt[d.idx(i, ny + 1, k)];
    B.vt[d.idx(i, ny + 1, k)] = 0.0;
  }
}

// velocityBC loop 3 (z faces), src/BoundaryConditions.f90:60-73
__global__ void k_vbc_z(DevBlock B) {
  const Dims& d = B.d;
  const int n = d.nx * d.ny;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int i = 2 + t % d.nx, j = 2 + t / d.nx;
    const int nz = d.nz;
    B.ut[d.idx(i, j, 1)] = B.ut[d.idx(i, j, 2)];
    B.vt[d.idx(i, j, 1)] = B.vt[d.idx(i, j, 2)];
    B.wt[d.idx(i, j, 1)] = 0.0;
    B.ut[d.idx(i, j, nz + 2)] = B.ut[d.idx(i, j, nz + 1)];
    B.vt[d.idx(i, j, nz + 2)] = B.vt[d.idx(i, j, nz + 1)];
    B.wt[d.idx(i, j, nz + 1)] = 0.0;
  }
}

// solidCellBC / solidCellBC_move (src/BoundaryConditions.f90:76-115)
__global__ void k_solid_bc(DevBlock B, int move) {
  const Dims& d = B.d;
  const int64_t n = (int64_t)d.nx * d.ny * d.nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = 2 + (int)(t % d.nx);
    const int64_t r = t / d.nx;
    const int j = 2 + (int)(r % d.ny), k = 2 + (int)(r / d.ny);
    const int64_t c = d.idx(i, j, k);
    if (B.cell[c] != 1) continue;
    B.ut[c] = 0.0;
    B.vt[c] = 0.0;
    B.wt[c] = 0.0;
    B.p[c] = 0.0;
    if (move) {
      B.u[c] = 0.0;
      B.v[c] = 0.0;
      B.w[c] = 0.0;
    }
  }
}


// the stencil's tables from the spacings and the coefficient tables, with the
// operations and the order the stencil's expressions have in each precision
__global__ void k_mom_tables(DevBlock B, double* mt, float* mtf, unsigned* mtk) {
  const Dims& D = B.d;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 >= D.NX + D.NY + D.NZ) return;
  const int ax = t0 < D.NX ? 0 : t0 < D.NX + D.NY ? 1 : 2;
  const int first = ax == 0 ? 0 : ax == 1 ? D.NX : D.NX + D.NY, len = ax == 0 ? D.NX : ax == 1 ? D.NY : D.NZ;
  const int gy = mom_groups(D.NX), g0 = ax == 0 ? 0 : ax == 1 ? gy : gy + mom_groups(D.NY);
  const int q = t0 - first + 1;  // 1-based grid index
  constexpr int N = 32;          // entries between slots
  double* T = mt + mom_slot0(g0, q - 1, kMtSlots);
  float* F = mtf + mom_slot0(g0, q - 1, kMfSlots);
  mtk[32 * g0 + q - 1] = 0xffffu;
  if (q < 2 || q > len - 1) return;  // no cell there
  const double* dd = ax == 0 ? B.dxa : ax == 1 ? B.dya : B.dza;
  const float* df = ax == 0 ? B.dxf : ax == 1 ? B.dyf : B.dzf;
  const int self = ax == 0 ? T_UU : ax == 1 ? T_VV : T_WW, cross = ax == 0 ? T_UW : ax == 1 ? T_VU : T_WU;
  const int64_t col = 6 * (int64_t)(q - 1);
  auto fill = [&](auto half, const auto* dl_, const auto* ca, const auto* ck, const auto* xa, const auto* xk,
                  auto* div) {
    using R = decltype(half);
    const R dl = dl_[q - 2], d = dl_[q - 1], dr = dl_[q], two = R(2.0);
    div[MD_HALF_R] = half * (d + dr);
    div[MD_HALF_L] = half * (d + dl);
    div[MD_SA] = ca[col + 5] * dr;
    div[MD_SK] = two * ck[col + 5] * d;
    div[MD_XA] = xa[col + 5] * (half * (d + dr));
    div[MD_XK] = two * xk[col + 5] * (half * (d + dl));
    div[MD_D] = d;
    div[MD_R] = dr;
  };
  double e[N_MD];
  float f[N_MD];
  fill(0.5, dd, B.ca[self], B.ck[self], B.ca[cross], B.ck[cross], e);
  fill(0.5f, df, B.caf[self], B.ckf[self], B.caf[cross], B.ckf[cross], f);
  unsigned kind = 0;
  for (int s = 0; s < N_MD; ++s) {
    const double y = 1.0 / e[s];
    T[2 * s * N] = e[s];
    T[(2 * s + 1) * N] = y;
    kind |= div_kind(e[s], y) << s;
    F[s * N] = __fdividef(1.0f, f[s]);
    F[(kMfD + s) * N] = f[s];
  }
  mtk[32 * g0 + q - 1] = kind;
  const double r2 = dd[q - 1] + dd[q], l2 = dd[q - 1] + dd[q - 2];
  T[(kMtQ + MQ_R) * N] = dd[q] / r2;
  T[(kMtQ + MQ_2) * N] = 2.0 / r2;
  T[(kMtQ + MQ_C) * N] = 2.0 / (0.5 * (r2 + l2));
  const float g2 = df[q - 1] + df[q], h2 = df[q - 1] + df[q - 2];
  F[(kMfQ + MQ_R) * N] = __fdividef(df[q], g2);
  F[(kMfQ + MQ_2) * N] = __fdividef(2.0f, g2);
  F[(kMfQ + MQ_C) * N] = __fdividef(2.0f, 0.5f * (g2 + h2));
  F[(kMfI + MQ_R) * N] = df[q] / g2;
  F[(kMfI + MQ_2) * N] = 2.0f / g2;
  F[(kMfI + MQ_C) * N] = 2.0f / (0.5f * (g2 + h2));
  for (int c = 0; c < 5; ++c) {
    T[(kMtC + c) * N] = B.ca[self][col + c];
    T[(kMtC + 5 + c) * N] = B.ck[self][col + c];
    T[(kMtC + 10 + c) * N] = B.ca[cross][col + c];
    T[(kMtC + 15 + c) * N] = B.ck[cross][col + c];
    F[(kMfC + c) * N] = B.caf[self][col + c];
    F[(kMfC + 5 + c) * N] = B.ckf[self][col + c];
    F[(kMfC + 10 + c) * N] = B.caf[cross][col + c];
    F[(kMfC + 15 + c) * N] = B.ckf[cross][col + c];
  }
}

MomArgs mom_args(double dt, double re) {
  const double y = 1.0 / re;
  return MomArgs{dt, re, y, div_kind(re, y)};
}

}  // namespace

// (re)builds the momentum stencil's per-line tables; the block's grids and
// coefficient tables are on the device
int launch_momentum_tables(HostBlock* hb) {
  const Dims& d = hb->d.d;
  const size_t n = 32 * (size_t)(mom_groups(d.NX) + mom_groups(d.NY) + mom_groups(d.NZ));
  if (!hb->d.mt) {
    void* p = nullptr;
    if (cudaMalloc(&p, n * (kMtSlots * sizeof(double) + kMfSlots * sizeof(float) + sizeof(unsigned))) != cudaSuccess)
      return BCFD_E_NOMEM;
    hb->allocs.push_back(p);
    double* t = static_cast<double*>(p);
    float* f = reinterpret_cast<float*>(t + n * kMtSlots);
    hb->d.mt = t;
    hb->d.mtf = f;
    hb->d.mtk = reinterpret_cast<unsigned*>(f + n * kMfSlots);
  }
  k_mom_tables<<<grid_for(d.NX + d.NY + d.NZ, 128), 128, 0, stream()>>>(hb->d, const_cast<double*>(hb->d.mt),
                                                               const_cast<float*>(hb->d.mtf),
                                                               const_cast<unsigned*>(hb->d.mtk));
  BCFD_LAUNCHED();
  return 0;
}

// the FP32 copies of u, v, w, p (a block's first mixed step)
static int ensure_f32_fields(HostBlock* hb) {
  if (hb->d.mf[0]) return 0;
  // rows of an odd pitch start anywhere: one array after the other, each on a
  // 256-byte boundary
  const size_t n = ((size_t)hb->d.d.npts() + 63) & ~(size_t)63;
  void* p = nullptr;
  if (cudaMalloc(&p, 4 * n * sizeof(float)) != cudaSuccess) return BCFD_E_NOMEM;
  hb->allocs.push_back(p);
  for (int q = 0; q < 4; ++q) hb->d.mf[q] = static_cast<float*>(p) + q * n;
  return 0;
}

int launch_momentum(const std::vector<HostBlock*>& hbs, double dt, double re, bool fp32) {
  const MomArgs a = mom_args(dt, re);
  const unsigned cap = 1u << 20;
  if (fp32) {
    for (HostBlock* hb : hbs) TRY_R(ensure_f32_fields(hb));
    TRY_R((launch_op<CvtOp, 256>(hbs, CvtOp{}, Extent::Points, 152u * 32u)));
    TRY_R((launch_op<MomentumOp<FastF>, 128>(hbs, MomentumOp<FastF>{a}, Extent::Interior, cap)));
  }
  else TRY_R((launch_op<MomentumOp<double>, 128>(hbs, MomentumOp<double>{a}, Extent::Interior, cap)));
  // cells within reach of TS cells (none without surfaces 51/52), then the
  // values the reference's loop leaves at the TS positions
  std::vector<HostBlock*> body;
  for (HostBlock* hb : hbs)
    if (hb->has_body) body.push_back(hb);
  if (body.empty()) return 0;
  if (fp32) TRY_R((launch_op<MomentumTsOp<float>, 128>(body, MomentumTsOp<float>{a}, Extent::Interior, 2048)));
  else TRY_R((launch_op<MomentumTsOp<double>, 128>(body, MomentumTsOp<double>{a}, Extent::Interior, 2048)));
  // up to 7 positions per TS cell: cap_ib * 7 items bound the grid
  std::vector<HostBlock*> one(1);
  for (HostBlock* hb : body) {
    k_one<TsRestoreOp, 128><<<grid_for((int64_t)hb->d.cap_ib * 7, 128, 256), 128, 0, stream()>>>(hb->d, TsRestoreOp{});
    BCFD_LAUNCHED();
  }
  return 0;
}

int launch_momentum(HostBlock* hb, double dt, double re, bool fp32) {
  return launch_momentum(std::vector<HostBlock*>{hb}, dt, re, fp32);
}

int launch_velocity_bc(HostBlock* hb, double dt, double uc) {
  const Dims& d = hb->d.d;
  k_vbc_x<<<grid_for((int64_t)d.ny * d.nz, 128), 128, 0, stream()>>>(hb->d, dt, uc);
  BCFD_LAUNCHED();
  k_vbc_y<<<grid_for((int64_t)d.nx * d.nz, 128), 128, 0, stream()>>>(hb->d);
  BCFD_LAUNCHED();
  k_vbc_z<<<grid_for((int64_t)d.nx * d.ny, 128), 128, 0, stream()>>>(hb->d);
  BCFD_LAUNCHED();
  return 0;
}

int launch_solid_bc(HostBlock* hb, bool move) {
  const int64_t n = (int64_t)hb->d.d.nx * hb->d.d.ny * hb->d.d.nz;
  k_solid_bc<<<grid_for(n, 256), 256, 0, stream()>>>(hb->d, move ? 1 : 0);
  BCFD_LAUNCHED();
  return 0;
}

// tangent-linear model of nsMomentum2order at the block's current (u,v,w,p):
// val = the predictor's ut,vt,wt (bitwise the FP64 stencil), tan = its
// derivative along (du,dv,dw,dp); device arrays of the block's point count
int launch_momentum_tangent(HostBlock* hb, double dt, double re, const double* const du[4], double* const val[3],
                            double* const tan[3]) {
  MomentumTlmOp op{mom_args(dt, re), {du[0], du[1], du[2], du[3]}, val[0], val[1], val[2], tan[0], tan[1], tan[2]};
  k_one<MomentumTlmOp, 128><<<grid_for((int64_t)hb->d.d.nx * hb->d.d.ny * hb->d.d.nz, 128, 1u << 20), 128, 0,
                              stream()>>>(hb->d, op);
  BCFD_LAUNCHED();
  return 0;
}


// adjoint of nsMomentum2order at the block's current (u,v,w,p): (ub,vb,wb,pb)
// += J^T (ubar_t, vbar_t, wbar_t), J the predictor's Jacobian on fluid cells;
// foot is 16 words of device scratch.  With ts (a block whose body has
// thin-surface cells) the overlay is transposed too: ab at the positions the
// loop's final restore writes goes to ts->gb first, then the cells near TS
// cells read through the overlay and the ghost scalars' adjoints are added
// to ts->gb (the block's ghost arrays must hold the values the forward step
// read); without it such cells set BCFD_E_STATE.
int launch_momentum_adjoint(HostBlock* hb, double dt, double re, const double* const sb[3], double* const ab[4],
                            uint32_t* foot, const MomTsAdj* ts) {
  const MomArgs a = mom_args(dt, re);
  const int64_t ni = (int64_t)hb->d.d.nx * hb->d.d.ny * hb->d.d.nz;
  const int* last = nullptr;
  if (ts) {
    k_ts_restore_adj<<<1, 32, 0, stream()>>>(hb->d, ab[0], ab[1], ab[2], ab[3], ts->gb, ts->cap);
    BCFD_LAUNCHED();
    k_ts_last<<<grid_for(ni, 128, 1u << 16), 128, 0, stream()>>>(hb->d, ts->last);
    BCFD_LAUNCHED();
    last = ts->last;
  }
  BCFD_CUDA(cudaMemsetAsync(foot, 0, kFootWords * sizeof(uint32_t), stream()));
  k_mom_footprint<<<grid_for(ni, 128, 1u << 16), 128, 0, stream()>>>(hb->d, a, foot, sb[0], sb[1], sb[2], last);
  BCFD_LAUNCHED();
  k_mom_adjoint_static<<<grid_for(hb->d.d.npts(), 128, 1u << 20), 128, 0, stream()>>>(
      hb->d, a, foot, sb[0], sb[1], sb[2], ab[0], ab[1], ab[2], ab[3]);
  BCFD_LAUNCHED();
  // of each pair below one returns at once: what is not finite is known on the
  // device only
  for (const auto fn : {k_mom_adjoint<false>, k_mom_adjoint<true>}) {
    fn<<<grid_for(hb->d.d.npts(), 128, 1u << 20), 128, 0, stream()>>>(hb->d, a, foot, sb[0], sb[1], sb[2], ab[0],
                                                                      ab[1], ab[2], ab[3], last);
    BCFD_LAUNCHED();
  }
  if (ts) {
    for (const auto fn : {k_mom_ghost_contrib<false>, k_mom_ghost_contrib<true>}) {
      fn<<<grid_for(ni, 128, 1u << 16), 128, 0, stream()>>>(hb->d, a, foot, ts->last, sb[0], sb[1], sb[2], ts->contrib);
      BCFD_LAUNCHED();
    }
    k_mom_ghost_acc<<<1, 32, 0, stream()>>>(hb->d, ts->last, ts->contrib, ts->gb, ts->cap);
    BCFD_LAUNCHED();
  }
  return 0;
}

}  // namespace bcfd

