// demap_core.cuh -- the per-cell max-log arithmetic shared by the demapper
// kernels (demap.cu, timeint.cu): the point metric in the operation order of
// lab/m44_ldm.py:2447-2450 and the per-bit minima of :2483-2486.  Float32
// for the decode path; float64 for the drop-in of the reference's default
// float64 demap_llr_fast (lab/m16_demap_fast.py:80-119).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace atsc3 {

// The arithmetic of one value type.  metric4 forms the metric of four labels
// k .. k+3 (k a multiple of 4, tables 16-byte aligned),
//   q = (zr*pr + zi*pi) * -2 + |p|^2,  every operation rounded,
// with the multiplication by -2, which is exact, folded into the last addition
// as fma(s, -2, |p|^2): the same bits, one operation fewer.  Float32 takes two
// labels per instruction (mul/fma.rn.f32x2: each half rounded like the scalar
// operation).  The sum of the two products is written as fma(x, 1, y) with the
// 1 read from constant memory: ptxas contracts mul.rn.f32x2 + add.rn.f32x2 into
// one fma.rn.f32x2 (seen in the results, -fmad=false or not), which would skip
// a rounding.  min / min3 ignore a NaN operand q as long as the running
// minimum m is not one; every running minimum starts at +inf.
template <typename T> struct DemapArith;

static __constant__ unsigned long long demap_one2 = 0x3F8000003F800000ull;    // (1, 1)
static __constant__ unsigned long long demap_mone2 = 0xBF800000BF800000ull;   // (-1, -1)

template <> struct DemapArith<float> {
  struct Z { unsigned long long r, i; };            // (zr, zr), (zi, zi)
  struct P4 { ulonglong2 r, i, p; };
  static __device__ __forceinline__ unsigned long long dup(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
  }
  static __device__ __forceinline__ Z pack(float zr, float zi) { return Z{dup(zr), dup(zi)}; }
  static __device__ __forceinline__ P4 load4(const float *r, const float *i, const float *p) {
    return P4{*reinterpret_cast<const ulonglong2 *>(r), *reinterpret_cast<const ulonglong2 *>(i),
              *reinterpret_cast<const ulonglong2 *>(p)};
  }
  using U = unsigned long long;                     // two float32 values
  static __device__ __forceinline__ U mul2(U a, U b) {
    U d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  static __device__ __forceinline__ U fma2(U a, U b, U c) {
    U d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
  }
  static __device__ __forceinline__ U sum2(U x, U y) { return fma2(x, demap_one2, y); }
  static __device__ __forceinline__ U diff2(U x, U y) { return fma2(y, demap_mone2, x); }
  static __device__ __forceinline__ void unpack(U v, float &q0, float &q1) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(q0), "=f"(q1) : "l"(v));
  }
  static __device__ __forceinline__ U join(float a, float b) {
    U d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
  }
  static __device__ __forceinline__ void metric4(const Z &z, const P4 &t, float (&q)[4]) {
    const U m2 = 0xC0000000C0000000ull;             // (-2, -2)
    unpack(fma2(sum2(mul2(z.r, t.r.x), mul2(z.i, t.i.x)), m2, t.p.x), q[0], q[1]);
    unpack(fma2(sum2(mul2(z.r, t.r.y), mul2(z.i, t.i.y)), m2, t.p.y), q[2], q[3]);
  }
  // the four quadrant images of four points (re, im): q[0] (re, im), q[1]
  // (-re, im), q[2] (re, -im), q[3] (-re, -im); m = their minimum, which the
  // largest |s| gives, since rounding keeps order
  static __device__ __forceinline__ void quad4(const Z &z, const P4 &t, float (&q)[4][4],
                                               float (&m)[4]) {
    const U m2 = 0xC0000000C0000000ull, p2 = 0x4000000040000000ull;
    const U tr[2] = {t.r.x, t.r.y}, ti[2] = {t.i.x, t.i.y}, tp[2] = {t.p.x, t.p.y};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const U x = mul2(z.r, tr[h]), y = mul2(z.i, ti[h]);
      const U s = sum2(x, y), d = diff2(x, y);
      unpack(fma2(s, m2, tp[h]), q[0][2 * h], q[0][2 * h + 1]);
      unpack(fma2(d, p2, tp[h]), q[1][2 * h], q[1][2 * h + 1]);
      unpack(fma2(d, m2, tp[h]), q[2][2 * h], q[2][2 * h + 1]);
      unpack(fma2(s, p2, tp[h]), q[3][2 * h], q[3][2 * h + 1]);
      float s0, s1, d0, d1;
      unpack(s, s0, s1);
      unpack(d, d0, d1);
      unpack(fma2(join(fmaxf(fabsf(s0), fabsf(d0)), fmaxf(fabsf(s1), fabsf(d1))), m2, tp[h]),
             m[2 * h], m[2 * h + 1]);
    }
  }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
  static __device__ __forceinline__ float min(float m, float q) { return fminf(m, q); }
  static __device__ __forceinline__ float min3(float m, float q0, float q1) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(m), "f"(q0), "f"(q1));
    return d;
  }
  static __device__ __forceinline__ float inf() { return __int_as_float(0x7f800000); }
  static __device__ __forceinline__ float one(float zr, float zi, float r, float i, float p) {
    return __fmaf_rn(__fadd_rn(__fmul_rn(zr, r), __fmul_rn(zi, i)), -2.0f, p);
  }
  static constexpr float u = 5.9604645e-8f;         // 2^-24, half a unit in the last place of 1
};

template <> struct DemapArith<double> {
  struct Z { double r, i; };
  struct P4 { double2 r[2], i[2], p[2]; };
  static __device__ __forceinline__ Z pack(double zr, double zi) { return Z{zr, zi}; }
  static __device__ __forceinline__ P4 load4(const double *r, const double *i, const double *p) {
    P4 t;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      t.r[h] = reinterpret_cast<const double2 *>(r)[h];
      t.i[h] = reinterpret_cast<const double2 *>(i)[h];
      t.p[h] = reinterpret_cast<const double2 *>(p)[h];
    }
    return t;
  }
  static __device__ __forceinline__ double one(double zr, double zi, double r, double i, double p) {
    return __fma_rn(__dadd_rn(__dmul_rn(zr, r), __dmul_rn(zi, i)), -2.0, p);
  }
  static constexpr double u = 1.1102230246251565e-16;
  static __device__ __forceinline__ void metric4(const Z &z, const P4 &t, double (&q)[4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      q[2 * h] = one(z.r, z.i, t.r[h].x, t.i[h].x, t.p[h].x);
      q[2 * h + 1] = one(z.r, z.i, t.r[h].y, t.i[h].y, t.p[h].y);
    }
  }
  static __device__ __forceinline__ void quad4(const Z &z, const P4 &t, double (&q)[4][4],
                                               double (&m)[4]) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double re = v & 1 ? t.r[v / 2].y : t.r[v / 2].x;
      const double im = v & 1 ? t.i[v / 2].y : t.i[v / 2].x;
      const double p = v & 1 ? t.p[v / 2].y : t.p[v / 2].x;
      const double x = __dmul_rn(z.r, re), y = __dmul_rn(z.i, im);
      const double s = __dadd_rn(x, y), d = __dsub_rn(x, y);
      q[0][v] = __fma_rn(s, -2.0, p);
      q[1][v] = __fma_rn(d, 2.0, p);
      q[2][v] = __fma_rn(d, -2.0, p);
      q[3][v] = __fma_rn(s, 2.0, p);
      // NaN (s or d) loses every comparison below only as the second operand
      m[v] = min(min(min(min(inf(), q[0][v]), q[1][v]), q[2][v]), q[3][v]);
    }
  }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
  // one comparison and two selects; fmin's own NaN handling is several more
  static __device__ __forceinline__ double min(double m, double q) { return q < m ? q : m; }
  static __device__ __forceinline__ double min3(double m, double q0, double q1) {
    return min(min(m, q0), q1);
  }
  static __device__ __forceinline__ double inf() { return __longlong_as_double(0x7ff0000000000000ll); }
};

// Minima over the labels of a cell, split by each label bit: mn[i][b] =
// minimum of q over the labels whose bit i (0 = MSB) equals b; the minimum over
// all labels is min(mn[0][0], mn[0][1]).
//
// The labels are a matrix of rows of 16 (the four low label bits choose the
// column).  Every q enters one row minimum and one column minimum; the high
// bits' minima come from the row minima, the low bits' from the column minima
// at the end: two comparisons a label where updating each low bit's minimum
// directly took five.
//
// Three forms, by what the staged alphabet allows (stage_points looks):
//   general  four operations of the float32 pipe a label.
//   quad     2D-NUCs (16 to 256 points): the two top label bits choose a
//            quadrant of mirrored points, (re, im), (-re, im), (re, -im),
//            (-re, -im).  Their products differ in sign only, and rounding is
//            symmetric, so the four share two products and two sums: about two
//            operations a label, and the minimum over the four is one more.
//   lattice  square grids (1024 and 4096 points), see minima_lattice.
// The bits are the general form's in each.  All are bound by operand reads:
// the register file feeds a scheduler about two 32-bit operands a cycle
// (measured: fma.rn.f32x2 with three register operands 3.0 cycles, with one
// from constant memory 2.0; a three-operand minimum 2.0).  75 Blocks of 64800
// bits with per-cell sigma2, before (one metric and five minima a label) and
// now, launches back to back: 16 points 15.9 -> 14.0 us, 64 points 28.2 -> 19.8,
// 256 points 67.4 -> 29.6, 1024 points 184 -> 33.6, 4096 points 621 -> 37.7.
enum DemapForm { FORM_GENERAL = 0, FORM_STRUCT = 1 };

// the minima of the four low label bits, from those of 16 columns
template <int NB, typename T>
__device__ __forceinline__ void fold_columns(const T (&cm)[16], T (&mn)[NB][2]) {
  using A = DemapArith<T>;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int h = 0; h < 8; h += 2) {
        const int l0 = ((h >> p) << (p + 1)) | (b << p) | (h & ((1 << p) - 1));
        const int l1 = (((h + 1) >> p) << (p + 1)) | (b << p) | ((h + 1) & ((1 << p) - 1));
        mn[NB - 1 - p][b] = A::min3(mn[NB - 1 - p][b], cm[l0], cm[l1]);
      }
}

// row minima of 4 rows (label bits P and P + 1) and, by k0's bits, of the
// label bits from P + 2 to E - 1
template <int NB, int P, int E, typename T>
__device__ __forceinline__ void fold_rows(const T (&rm)[4], int k0, T (&mn)[NB][2]) {
  using A = DemapArith<T>;
  mn[NB - 1 - P][0] = A::min3(mn[NB - 1 - P][0], rm[0], rm[2]);
  mn[NB - 1 - P][1] = A::min3(mn[NB - 1 - P][1], rm[1], rm[3]);
  mn[NB - 2 - P][0] = A::min3(mn[NB - 2 - P][0], rm[0], rm[1]);
  mn[NB - 2 - P][1] = A::min3(mn[NB - 2 - P][1], rm[2], rm[3]);
  if constexpr (E > P + 2) {
    const T all = A::min(A::min3(rm[0], rm[1], rm[2]), rm[3]);
#pragma unroll
    for (int p = P + 2; p < E; ++p) {
      T(&m)[2] = mn[NB - 1 - p];
      if ((k0 >> p) & 1) m[1] = A::min(m[1], all);
      else m[0] = A::min(m[0], all);
    }
  }
}

template <int NB, typename T>
__device__ __forceinline__ void minima_quad(const typename DemapArith<T>::Z &z, const T *spr,
                                            const T *spi, const T *sp2, T (&mn)[NB][2]) {
  using A = DemapArith<T>;
  constexpr int J = 1 << (NB - 2);                // labels of a quadrant
  constexpr int L = J < 16 ? J : 16;
  const T inf = A::inf();
  T cm[16], rq[4], rm[4];
#pragma unroll
  for (int l = 0; l < 16; ++l) cm[l] = inf;
#pragma unroll
  for (int u = 0; u < 4; ++u) rq[u] = rm[u] = inf;
#pragma unroll
  for (int j = 0; j < J; j += 4) {
    const typename A::P4 t = A::load4(spr + j, spi + j, sp2 + j);
    const int l = j % L, r = j / L;
    T q[4][4], m[4];
    A::quad4(z, t, q, m);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      rq[u] = A::min3(rq[u], q[u][0], q[u][1]);
      rq[u] = A::min3(rq[u], q[u][2], q[u][3]);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) cm[l + v] = A::min(cm[l + v], m[v]);
    if constexpr (NB == 8) {
      rm[r] = A::min3(rm[r], m[0], m[1]);
      rm[r] = A::min3(rm[r], m[2], m[3]);
    }
  }
  mn[0][0] = A::min3(inf, rq[0], rq[1]);
  mn[0][1] = A::min3(inf, rq[2], rq[3]);
  mn[1][0] = A::min3(inf, rq[0], rq[2]);
  mn[1][1] = A::min3(inf, rq[1], rq[3]);
  if constexpr (NB == 4) {
    mn[2][0] = A::min3(inf, cm[0], cm[1]);
    mn[2][1] = A::min3(inf, cm[2], cm[3]);
    mn[3][0] = A::min3(inf, cm[0], cm[2]);
    mn[3][1] = A::min3(inf, cm[1], cm[3]);
  } else {
    fold_columns<NB, T>(cm, mn);
  }
  if constexpr (NB == 8) fold_rows<NB, 4, 6, T>(rm, 0, mn);
}

// What stage_points leaves behind the 3*M table values in shared memory.
template <int NB, typename T>
struct LatticeInfo {
  static constexpr int L = 1 << (NB / 2);
  T re[L], im[L];              // the levels, ascending
  T inv_r, inv_i;              // levels per unit, for a first guess
  T gap;                       // below the least squared level spacing
  T e0, kr, ki;                // rounding of two metrics: e0 + kr |zr| + ki |zi|
  T red[3][32];
};

template <int L, typename T>
__device__ __forceinline__ int lattice_below(const T *lev, T z, T inv) {
  // the last level <= z, or -1
  T g = (z - lev[0]) * inv;
  g = g < T(0) ? T(-1) : g;
  int l = min((int)(g > T(L) ? T(L) : g), L - 1);
  while (l + 1 < L && lev[l + 1] <= z) ++l;
  while (l >= 0 && lev[l] > z) --l;
  return l;
}

// A square grid: label = row * L + column, re ascending by row, im by column.
// In real numbers the metric is A(row) + B(column) + e with |e| <= eps, A and B
// parabolas, so the minimum over the labels with one row bit fixed lies at the
// nearest such row below zr or the nearest above, in the column nearest zi.  A
// label further out on the same side is at least gap (the squared level
// spacing) above, so wherever gap exceeds what rounding can move two metrics
// by, no other label's rounded metric can be the smallest: at most 4 labels a
// bit value are formed, with the general form's operations, instead of M / 2.
// Where two columns are nearly as near (within the rounding), both are taken.
// Returns false where the bound does not hold (a cell far outside the grid, an
// infinity or a NaN): the caller takes the general form.
// Rounding of one metric, u = 2^-24 (2^-53): the two products, their sum
// (doubled) and the last addition, u (6 |zr re| + 6 |zi im| + p2) and terms in
// u^2; twice that for two metrics, with room: 13 u, 13 u and 4 u, + 2 eps.
template <int NB, typename T>
__device__ __forceinline__ bool minima_lattice(T zr, T zi, const T *sp2,
                                               const LatticeInfo<NB, T> &w, T (&mn)[NB][2]) {
  using A = DemapArith<T>;
  constexpr int S = NB / 2, L = 1 << S;
  const T az = zr < T(0) ? -zr : zr, bz = zi < T(0) ? -zi : zi;
  const T slack = w.e0 + w.kr * az + w.ki * bz;
  if (!(w.gap > slack)) return false;
  const T inf = A::inf();
  const int lr = lattice_below<L, T>(w.re, zr, w.inv_r);
  const int li = lattice_below<L, T>(w.im, zi, w.inv_i);
  // the nearer of the two levels around a coordinate, and the other one where
  // the difference of the parabolas is within the rounding (its own included)
  auto nearest = [&](const T *lev, int l, T z, T a, int &k0, int &k1) {
    const int lo = max(l, 0), hi = min(l + 1, L - 1);
    const T d = lev[hi] - lev[lo], m = lev[hi] + lev[lo];
    const T diff = d * (m - (z + z));                   // parabola(hi) - parabola(lo)
    k0 = diff >= T(0) ? lo : hi;
    k1 = lo + hi - k0;
    const T ad = diff < T(0) ? -diff : diff;
    const T am = m < T(0) ? -m : m;
    if (ad * (T(1) - 8 * A::u) > slack + 8 * A::u * d * (am + a + a)) k1 = k0;
  };
  int r0, r1, c0, c1;
  nearest(w.re, lr, zr, az, r0, r1);
  nearest(w.im, li, zi, bz, c0, c1);
  // over the rows: the metric of row i, in the column(s) nearest
  auto row = [&](int i) {
    const int k = min(max(i, 0), L - 1);
    const T re = w.re[k];
    T q = A::one(zr, zi, re, w.im[c0], sp2[k * L + c0]);
    if (c1 != c0) q = A::min(q, A::one(zr, zi, re, w.im[c1], sp2[k * L + c1]));
    return i == k ? q : inf;
  };
  auto col = [&](int j) {
    const int k = min(max(j, 0), L - 1);
    const T im = w.im[k];
    T q = A::one(zr, zi, w.re[r0], im, sp2[r0 * L + k]);
    if (r1 != r0) q = A::min(q, A::one(zr, zi, w.re[r1], im, sp2[r1 * L + k]));
    return j == k ? q : inf;
  };
  auto bits = [&](int l, auto &&metric, int top) {
    const int h = l + 1;
    const T ql = metric(l), qh = metric(h);
#pragma unroll
    for (int p = 0; p < S; ++p) {
      // l's and h's neighbours outwards whose bit p is the other one
      const T xl = metric(((l >> p) << p) - 1), xh = metric(((h >> p) + 1) << p);
      const bool bl = (l >> p) & 1, bh = (h >> p) & 1;
      mn[top - p][0] = A::min(bl ? xl : ql, bh ? xh : qh);
      mn[top - p][1] = A::min(bl ? ql : xl, bh ? qh : xh);
    }
  };
  bits(lr, row, S - 1);
  bits(li, col, NB - 1);
  return true;
}

template <int NB, typename T>
__device__ __forceinline__ void minima_general(const typename DemapArith<T>::Z &z,
                                               const T *spr, const T *spi, const T *sp2,
                                               T (&mn)[NB][2]) {
  using A = DemapArith<T>;
  constexpr int M = 1 << NB;
  const T inf = A::inf();
  if constexpr (NB == 2) {
    const typename A::P4 t = A::load4(spr, spi, sp2);
    T q[4];
    A::metric4(z, t, q);
    mn[0][0] = A::min3(inf, q[0], q[1]);
    mn[0][1] = A::min3(inf, q[2], q[3]);
    mn[1][0] = A::min3(inf, q[0], q[2]);
    mn[1][1] = A::min3(inf, q[1], q[3]);
  } else {
    constexpr int L = 16;                         // labels a row
    constexpr int R = NB >= 6 ? 4 : 1;            // rows a pass
    T cm[L];
#pragma unroll
      for (int l = 0; l < L; ++l) cm[l] = inf;
#pragma unroll 1
    for (int k0 = 0; k0 < M; k0 += L * R) {
      T rm[4];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rm[r] = inf;
#pragma unroll
        for (int l = 0; l < L; l += 4) {
          const int k = k0 + r * L + l;
          const typename A::P4 t = A::load4(spr + k, spi + k, sp2 + k);
          T q[4];
          A::metric4(z, t, q);
          rm[r] = A::min3(rm[r], q[0], q[1]);
          rm[r] = A::min3(rm[r], q[2], q[3]);
#pragma unroll
          for (int v = 0; v < 4; ++v) cm[l + v] = A::min(cm[l + v], q[v]);
        }
      }
      if constexpr (NB >= 6) {
        fold_rows<NB, 4, NB, T>(rm, k0, mn);
      }
    }
    fold_columns<NB, T>(cm, mn);
  }
}

template <int NB, typename T>
__device__ __forceinline__ void cell_minima(T zr, T zi, const T *sp,
                                            int form, T (&mn)[NB][2]) {
  using A = DemapArith<T>;
  constexpr int M = 1 << NB;
  const T *spr = sp, *spi = sp + M, *sp2 = sp + 2 * M;
  typename A::Z z = A::pack(zr, zi);
#pragma unroll
  for (int i = 0; i < NB; ++i) mn[i][0] = mn[i][1] = A::inf();
  if constexpr (NB >= 4 && NB <= 8) {
    if (form == FORM_STRUCT) {
      minima_quad<NB, T>(z, spr, spi, sp2, mn);
      return;
    }
  }
  if constexpr (NB >= 10) {
    if (form == FORM_STRUCT &&
        minima_lattice<NB, T>(zr, zi, sp2,
                              *reinterpret_cast<const LatticeInfo<NB, T> *>(sp + 3 * M), mn))
      return;
  }
  minima_general<NB, T>(z, spr, spi, sp2, mn);
}

// Dynamic shared memory of a kernel that stages an alphabet of 2^nb points.
inline int demap_smem_bytes(int nb, int vb) {
  const int l = 1 << (nb / 2);
  return (3 << nb) * vb + (nb >= 10 ? (2 * l + 6 + 3 * 32) * vb : 0);
}

// Stages an alphabet (Re, Im, |p|^2: 3*2^NB values) in shared memory, 16-byte
// copies where the source allows them, and says which form it has: whether the
// quadrants mirror the first one (16 to 256 points) or the points are a grid of
// ascending levels (1024 and 4096).  Every thread of the CTA calls it.
template <int NB, typename T>
__device__ __forceinline__ int stage_points(T *sp, const T *__restrict__ pts) {
  constexpr int M = 1 << NB;
  if ((reinterpret_cast<uintptr_t>(pts) & 15) == 0) {
    const uint4 *src = reinterpret_cast<const uint4 *>(pts);
    uint4 *dst = reinterpret_cast<uint4 *>(sp);
    for (int k = threadIdx.x; k < 3 * M * (int)sizeof(T) / 16; k += blockDim.x)
      dst[k] = __ldg(src + k);
  } else {
    for (int k = threadIdx.x; k < 3 * M; k += blockDim.x) sp[k] = pts[k];
  }
  __syncthreads();
  const T *r = sp, *i = sp + M, *p = sp + 2 * M;
  if constexpr (NB == 2) {
    return FORM_GENERAL;
  } else if constexpr (NB <= 8) {
    constexpr int J = M / 4;
    bool ok = true;
    for (int k = J + threadIdx.x; k < M; k += blockDim.x) {
      const int j = k % J, u = k / J;
      ok = ok && r[k] == (u & 1 ? -r[j] : r[j]) && i[k] == (u & 2 ? -i[j] : i[j]) && p[k] == p[j];
    }
    return __syncthreads_and(ok) ? FORM_STRUCT : FORM_GENERAL;
  } else {
    using A = DemapArith<T>;
    constexpr int L = 1 << (NB / 2);
    LatticeInfo<NB, T> &w = *reinterpret_cast<LatticeInfo<NB, T> *>(sp + 3 * M);
    bool ok = true;
    // least spacing, largest |p2 - re^2 - im^2| (a float's own rounding of it
    // is within 4 u p2), largest p2
    T v[3] = {A::inf(), T(0), T(0)};
    for (int k = threadIdx.x; k < M; k += blockDim.x) {
      const int a = k & ~(L - 1), b = k & (L - 1);
      ok = ok && r[k] == r[a] && i[k] == i[b] && p[k] >= T(0);
      const T e = p[k] - r[k] * r[k] - i[k] * i[k];
      v[1] = e > v[1] ? e : -e > v[1] ? -e : v[1];
      v[2] = p[k] > v[2] ? p[k] : v[2];
      if (b == 0) w.re[a / L] = r[k];
      if (a == 0) w.im[b] = i[k];
      if (b == 0 && a) {
        const T d = r[k] - r[k - L];
        ok = ok && d > T(0);
        v[0] = A::min(v[0], d);
      }
      if (a == 0 && b) {
        const T d = i[k] - i[k - 1];
        ok = ok && d > T(0);
        v[0] = A::min(v[0], d);
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      for (int o = 16; o > 0; o >>= 1) {
        const T x = __shfl_xor_sync(0xffffffffu, v[q], o);
        v[q] = (q == 0) == (x < v[q]) ? x : v[q];
      }
      if ((threadIdx.x & 31) == 0) w.red[q][threadIdx.x >> 5] = v[q];
    }
    const bool all = __syncthreads_and(ok);
    if (threadIdx.x == 0) {
      for (int q = 0; q < 3; ++q)
        for (int o = 1; o < (int)(blockDim.x >> 5); ++o) {
          const T x = w.red[q][o];
          w.red[q][0] = (q == 0) == (x < w.red[q][0]) ? x : w.red[q][0];
        }
      const T d = w.red[0][0], eps = w.red[1][0], p2 = w.red[2][0];
      const T rl = w.re[0], rh = w.re[L - 1], il = w.im[0], ih = w.im[L - 1];
      const T ar = -rl > rh ? -rl : rh, ai = -il > ih ? -il : ih;
      w.inv_r = T(L - 1) / (rh - rl);
      w.inv_i = T(L - 1) / (ih - il);
      w.gap = d * d * (T(1) - 8 * A::u);
      w.e0 = 2 * eps + 12 * A::u * p2 + T(1e-36);
      w.kr = 13 * A::u * ar;
      w.ki = 13 * A::u * ai;
    }
    __syncthreads();
    return all ? FORM_STRUCT : FORM_GENERAL;
  }
}

}  // namespace atsc3
