// Fixed-point element arithmetic of the FP64 stencil.
//
// GB300 issues 2 FP64 thread-operations per SM and clock (measured, DFMA), but
// 32 wide integer multiply-adds (32 x 32 + 64 bits) and 64 64-bit additions, so
// the FP64 element product is formed in 64-bit integers with the precision of
// FP64 or better:
//
//   - a tile's nodal values become X = rint(x * 2^kx), |X| <= 2^57, with kx from the
//     largest value that the tile reads (fx_tile_exponent, which sends tiles whose
//     values are uneven to the FP64 form);
//   - the Walsh-Hadamard transform and every sum of forces are integer
//     additions, exact (and modular: only final sums have to fit 64 bits);
//   - the stiffness entries are integers c = ch * 2^32 + cl of up to 63 bits with
//     one exponent kc for the whole problem, the transformed values are
//     x = xh * 2^32 + xl, and a row is
//         sum xh*ch + (sum xh*cl >> 32) + (sum xl*ch >> 32):
//     three multiply-adds an entry, the dropped xl*cl is below a quarter unit.
//
// Limits, for |X| <= 2^57 (transformed values up to 2^60, shear sums 2^61):
//   sum |xh||cl| <= 9 * 2^59 < 2^63;  sum |xl||ch| < 2^63 by row sums of c below
//   2^63.9, entries below 2^63;  a node's force, bounded by eight times the
//   largest absolute row sum D of the element matrix, stays below 2^63.
//
// Error of K.x against 80-bit arithmetic in the 2-norm, over that of the FP64 form
// on the same inputs (32^3 Voronoi polycrystals, 2 % pores, Zener 0.5 and 3): 0.56
// to 0.60 on random vectors, 0.53 to 0.77 on displacements, 0.53 to 0.69 on the
// gradients before, during and late in a solve (peak to rms up to 23).
#pragma once
#include <cstdint>

#include "e3d_device.cuh"

namespace e3d {

// Table of a phase: 72 entries (ch, cl), two to an int4: the upper triangles of
// M2 (45, second-order modes), C/16 (21, constant mode) and M3 (6, third order).
constexpr int kFxEntries = 72;
constexpr int kFxStride = kFxEntries / 2;  // int4 per phase
constexpr int kFxM2 = 0, kFxC = 45, kFxM3 = 66;

// The problem's table exponent, from the phase tables: kc is the largest that
// keeps the limits above.  ok = 0 sends every tile to the FP64 form: phases whose
// stiffness differs by more than kFxContrast (the softest would keep fewer bits
// than FP64), or entries outside the range that exponent arithmetic covers.
struct FxInfo {
  int kc;
  int ok;
};
constexpr double kFxContrast = 8.0;
constexpr int kFxNodeBits = 57;

// kc from the norms over all phases: the largest absolute row sum d of an
// element matrix (dmin: the smallest positive one), the largest row sum and entry
// of a modal table.
__host__ __device__ inline FxInfo fx_info(double d, double dmin, double rows, double entry) {
  FxInfo f{0, 0};
  if (!(d > 0.0) || !(d < 1e90) || !(d > 1e-90) || !(rows < 1e90) || !(entry < 1e90)) return f;
  if (!(dmin * kFxContrast >= d)) return f;
  // 8 * D * 2^57 * 2^kc / 2^64 <= 2^62.5; row sums < 2^63.9; entries < 2^62.9
  const double a = 66.5 - log2(d), b = 63.9 - log2(rows), c = 62.9 - log2(entry);
  const double m = a < b ? (a < c ? a : c) : (b < c ? b : c);
  f.kc = (int)floor(m);
  f.ok = 1;
  return f;
}

__host__ __device__ inline void fx_split(double v, int kc, int& h, int& l) {
  const long long q = llrint(ldexp(v, kc));
  h = (int)((q + (1ll << 31)) >> 32);
  l = (int)(q - (long long)h * (1ll << 32));
}

// Entry e of a phase's integer table from its FP64 table.
__host__ __device__ inline double fx_source(const double* cs, int e) {
  int base = kM2, n = 9, q = e - kFxM2;
  if (e >= kFxM3) {
    base = kM3, n = 3, q = e - kFxM3;
  } else if (e >= kFxC) {
    base = 0, n = 6, q = e - kFxC;
  }
  int r = 0;
  while (q >= n - r) {
    q -= n - r;
    ++r;
  }
  return cs[base + n * r + r + q];
}

// acc += a * b, 32 x 32 + 64 bits: one instruction.
__device__ __forceinline__ void fx_mad(long long& acc, int a, int b) {
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}
// acc = a * b + c, and acc = a * b.
__device__ __forceinline__ long long fx_mad_from(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ long long fx_mul(int a, int b) {
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
// x = hi * 2^32 + lo with both halves signed: lo is the low word as it is.
__device__ __forceinline__ int fx_hi(long long x) { return (int)(x >> 32) - ((int)x >> 31); }
__device__ __forceinline__ int fx_lo(long long x) { return (int)x; }

// out = M in for a symmetric N x N matrix whose upper triangle starts at entry
// BASE of the table: every entry is loaded once and used for both of its rows.
template <int N, int BASE>
__device__ __forceinline__ void fx_symv(const int4* __restrict__ tab, const long long (&in)[N], long long (&out)[N]) {
  int xh[N], xl[N];
  long long m1[N], m2[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    xh[i] = fx_hi(in[i]);
    xl[i] = fx_lo(in[i]);
  }
  const long long half = 1ll << 31;  // rounds the shifts below
  int4 q = make_int4(0, 0, 0, 0);
#pragma unroll
  for (int r = 0, e = BASE; r < N; ++r) {
#pragma unroll
    for (int c = r; c < N; ++c, ++e) {
      if ((e & 1) == 0 || e == BASE) q = __ldg(tab + (e >> 1));
      const int ch = (e & 1) ? q.z : q.x, cl = (e & 1) ? q.w : q.y;
      // row 0 starts with its first entry; row c starts with row 0's entry c
      if (r == 0 && c == 0) {
        out[0] = fx_mul(xh[0], ch);
        m1[0] = fx_mad_from(xh[0], cl, half);
        m2[0] = fx_mad_from(xl[0], ch, half);
      } else {
        fx_mad(out[r], xh[c], ch);
        fx_mad(m1[r], xh[c], cl);
        fx_mad(m2[r], xl[c], ch);
      }
      if (c != r && r == 0) {
        out[c] = fx_mul(xh[0], ch);
        m1[c] = fx_mad_from(xh[0], cl, half);
        m2[c] = fx_mad_from(xl[0], ch, half);
      } else if (c != r) {
        fx_mad(out[c], xh[r], ch);
        fx_mad(m1[c], xh[r], cl);
        fx_mad(m2[c], xl[r], ch);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] += (m1[i] >> 32) + (m2[i] >> 32);
}

// Element forces in the Hadamard domain (element_modal in fixed point): h[c][b]
// -> f[c][b], b = 1..7.
__device__ __forceinline__ void element_modal_fx(const int4* __restrict__ tab, const long long (&h)[3][8],
                                                 long long (&f)[3][8]) {
  {
    const long long in[9] = {h[0][HXY], h[1][HXY], h[2][HXY], h[0][HXZ], h[1][HXZ],
                             h[2][HXZ], h[0][HYZ], h[1][HYZ], h[2][HYZ]};
    long long out[9];
    fx_symv<9, kFxM2>(tab, in, out);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      f[c][HXY] = out[c];
      f[c][HXZ] = out[3 + c];
      f[c][HYZ] = out[6 + c];
    }
  }
  {
    const long long e[6] = {h[0][HX_],
                            h[1][HY_],
                            h[2][HZ_],
                            h[0][HZ_] + h[2][HX_],
                            h[1][HZ_] + h[2][HY_],
                            h[0][HY_] + h[1][HX_]};
    long long s[6];
    fx_symv<6, kFxC>(tab, e, s);
    f[0][HX_] = s[0];
    f[1][HY_] = s[1];
    f[2][HZ_] = s[2];
    f[0][HZ_] = s[3];
    f[2][HX_] = s[3];
    f[1][HZ_] = s[4];
    f[2][HY_] = s[4];
    f[0][HY_] = s[5];
    f[1][HX_] = s[5];
  }
  {
    const long long in[3] = {h[0][HXYZ], h[1][HXYZ], h[2][HXYZ]};
    long long out[3];
    fx_symv<3, kFxM3>(tab, in, out);
    f[0][HXYZ] = out[0];
    f[1][HXYZ] = out[1];
    f[2][HXYZ] = out[2];
  }
}

// v * 2^kx to the nearest integer (halves up in magnitude), |result| < 2^kFxNodeBits, in integer
// instructions: the conversion instruction issues on the FP64 pipe, where it
// would cost as much as 32 of these.
__device__ __forceinline__ long long fx_from_double(double v, int kx) {
  const int hi = __double2hiint(v);
  const int e = (hi >> 20) & 0x7ff;
  // |v| = m * 2^(e - 1075); t = m << 10; result = t >> (1085 - kx - e), rounded
  const unsigned long long t = (((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(v)) << 10;
  const int n = 1084 - kx - e;  // one bit short of it; at least 5
  const unsigned long long q = ((t >> min(n, 63)) + 1) >> 1;
  const long long r = n > 63 ? 0 : (long long)q;
  return hi < 0 ? -r : r;
}
// d * 2^ko for d = (double) of an integer.
__device__ __forceinline__ double fx_scale(double d, int ko20) {
  const int hi = __double2hiint(d);
  return __hiloint2double(hi != 0 ? hi + ko20 : 0, __double2loint(d));
}

}  // namespace e3d
