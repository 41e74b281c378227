// FP32 stencil with two elements a thread, in packed FP32 arithmetic.
//
// The FP32 sweep is bound by issue slots, not by HBM or the FP32 pipe: with one
// element a thread it issued some 700 instructions a node, half of them
// addresses, shared-memory traffic and predicates.  Here a thread owns two
// columns that are neighbours in y.  One packed instruction (add / mul / fma
// .f32x2) works on both elements, loads and indices are shared, and the force
// exchange between the two needs no memory.
#pragma once
#include <cstdint>

#include "e3d_device.cuh"

namespace e3d {

using f2 = unsigned long long;  // two floats: low word first

__device__ __forceinline__ f2 f2_pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2_lo(f2 v) {
  float a;
  asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(v));
  return a;
}
__device__ __forceinline__ float f2_hi(f2 v) {
  float b;
  asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(v));
  return b;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// s = sum over the listed columns of C[row][col] e[col]; t: packed upper
// triangle of C/16 of the two elements.
template <int N>
__device__ __forceinline__ f2 f2_row(const f2 (&t)[21], int row, const int (&idx)[N], const f2 (&e)[N]) {
  f2 s = f2_mul(t[sym6(row, idx[0])], e[0]);
#pragma unroll
  for (int c = 1; c < N; ++c) s = f2_fma(t[sym6(row, idx[c])], e[c], s);
  return s;
}
template <int N>
__device__ __forceinline__ f2 f2_row_add(const f2 (&t)[21], int row, const int (&idx)[N], const f2 (&e)[N], f2 s) {
#pragma unroll
  for (int c = 0; c < N; ++c) s = f2_fma(t[sym6(row, idx[c])], e[c], s);
  return s;
}

// element_modal_f32 for two elements: h[c][1..7] -> f[c][1..7] (h is used up);
// w1, w2, w3 gain the shares of h . f of the three Hadamard orders (the element
// energies: w1 + 3 w2 + 9 w3 summed over a mesh is h . K h).
__device__ __forceinline__ void element_modal_f2(const f2 (&t)[21], const f2 (&h)[3][8], f2 (&f)[3][8], f2& w1, f2& w2,
                                                 f2& w3) {
  {
    const int idx[6] = {0, 1, 2, 3, 4, 5};
    const f2 e[6] = {h[0][HX_],
                     h[1][HY_],
                     h[2][HZ_],
                     f2_add(h[0][HZ_], h[2][HX_]),
                     f2_add(h[1][HZ_], h[2][HY_]),
                     f2_add(h[0][HY_], h[1][HX_])};
    f2 s[6];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      s[r] = f2_row<6>(t, r, idx, e);
      w1 = f2_fma(e[r], s[r], w1);
    }
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
    const f2 k3 = f2_pack(1.0f / 3.0f, 1.0f / 3.0f);
    const f2 uxy = f2_mul(h[0][HXY], k3), vxy = f2_mul(h[1][HXY], k3), wxy = f2_mul(h[2][HXY], k3);
    const f2 uxz = f2_mul(h[0][HXZ], k3), vxz = f2_mul(h[1][HXZ], k3), wxz = f2_mul(h[2][HXZ], k3);
    const f2 uyz = f2_mul(h[0][HYZ], k3), vyz = f2_mul(h[1][HYZ], k3), wyz = f2_mul(h[2][HYZ], k3);
    const int ix[5] = {1, 2, 3, 4, 5}, iy[5] = {0, 2, 3, 4, 5}, iz[5] = {0, 1, 3, 4, 5};
    const f2 ex[5] = {vxy, wxz, uxz, f2_add(vxz, wxy), uxy};
    const f2 ey[5] = {uxy, wyz, f2_add(uyz, wxy), vyz, vxy};
    const f2 ez[5] = {uxz, vyz, wxz, wyz, f2_add(uyz, vxz)};
    f[0][HXY] = f2_row_add<5>(t, 0, iy, ey, f2_row<5>(t, 5, ix, ex));
    f[1][HXY] = f2_row_add<5>(t, 5, iy, ey, f2_row<5>(t, 1, ix, ex));
    f[2][HXY] = f2_row_add<5>(t, 3, iy, ey, f2_row<5>(t, 4, ix, ex));
    f[0][HXZ] = f2_row_add<5>(t, 0, iz, ez, f2_row<5>(t, 3, ix, ex));
    f[1][HXZ] = f2_row_add<5>(t, 5, iz, ez, f2_row<5>(t, 4, ix, ex));
    f[2][HXZ] = f2_row_add<5>(t, 3, iz, ez, f2_row<5>(t, 2, ix, ex));
    f[0][HYZ] = f2_row_add<5>(t, 5, iz, ez, f2_row<5>(t, 3, iy, ey));
    f[1][HYZ] = f2_row_add<5>(t, 1, iz, ez, f2_row<5>(t, 4, iy, ey));
    f[2][HYZ] = f2_row_add<5>(t, 4, iz, ez, f2_row<5>(t, 2, iy, ey));
    const f2 in[9] = {uxy, vxy, wxy, uxz, vxz, wxz, uyz, vyz, wyz};
#pragma unroll
    for (int i = 0; i < 9; ++i) w2 = f2_fma(in[i], f[i % 3][i < 3 ? HXY : i < 6 ? HXZ : HYZ], w2);
  }
  {
    const f2 k9 = f2_pack(1.0f / 9.0f, 1.0f / 9.0f);
    const f2 u = f2_mul(h[0][HXYZ], k9), v = f2_mul(h[1][HXYZ], k9), w = f2_mul(h[2][HXYZ], k9);
    const int ixy[3] = {2, 3, 4}, ixz[3] = {1, 4, 5}, iyz[3] = {0, 3, 5};
    const f2 exy[3] = {w, u, v}, exz[3] = {v, w, u}, eyz[3] = {u, w, v};
    f[0][HXYZ] = f2_row_add<3>(t, 0, iyz, eyz, f2_row_add<3>(t, 5, ixz, exz, f2_row<3>(t, 3, ixy, exy)));
    f[1][HXYZ] = f2_row_add<3>(t, 5, iyz, eyz, f2_row_add<3>(t, 1, ixz, exz, f2_row<3>(t, 4, ixy, exy)));
    f[2][HXYZ] = f2_row_add<3>(t, 3, iyz, eyz, f2_row_add<3>(t, 4, ixz, exz, f2_row<3>(t, 2, ixy, exy)));
    w3 = f2_fma(u, f[0][HXYZ], f2_fma(v, f[1][HXYZ], f2_fma(w, f[2][HXYZ], w3)));
  }
}

}  // namespace e3d
