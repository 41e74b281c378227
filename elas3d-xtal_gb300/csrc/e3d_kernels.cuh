// Kernels of the sm_103a voxel-FE solver.  See e3d_device.cuh for the element
// arithmetic.  Layout in HBM (all component-major, node m = x + nx*(y + ny*z)):
//   u, g, b, z, h[2], Ah : 3*ns values each
//   minv                 : 6*ns (symmetric 3x3 block inverse: 00 11 22 01 02 12)
//   pix                  : ns int32, 0-based phase
//   cs                   : nphase*kCsStride FP64 stiffness tables (C/16 and the summed mode matrices)
//   cs32                 : nphase*24, FP32 upper triangle of C/16 (element_modal_f32)
//   dk                   : nphase*576, [p][a][i][b][j] (reference local order)
//   dkd                  : nphase*78: diagonal 3x3 blocks [a][i][j], then the inverse of their sum
//   hx, hy, hd           : tile-edge force halos (see apply_tile)
#pragma once
#include <cstdint>
#include <type_traits>

#include "e3d_bounds.cuh"
#include "e3d_device.cuh"
#include "e3d_f32x2.cuh"
#include "e3d_fixed.cuh"
#include "e3d_index.h"
#include "e3d_tma.cuh"

namespace e3d {

constexpr int TILE_X = 32;
constexpr int TILE_Y = 8;

// Tuning knobs of the persistent PCG kernel (set at build time).
#ifndef E3D_F32_BLOCKS_PER_SM
#define E3D_F32_BLOCKS_PER_SM 2  // resident 256-thread blocks per SM, FP32 form
#endif
// Planes per step of the ring-fed FP32 tile: each thread computes E3D_RING_ZS
// consecutive elements of its column between two barriers.  ZS = 1 runs two
// 128-register blocks per SM; ZS = 2 one 255-register block (two independent
// element computations per thread, no spills) -- measured slower at 500^3
// (13.3 vs 9.7 ms per inner iteration): occupancy matters more here.
#ifndef E3D_RING_ZS
#define E3D_RING_ZS 1
#endif
#ifndef E3D_TMA_STAGES
#define E3D_TMA_STAGES (E3D_RING_ZS + 4)  // ring stages per block (ZS + 1 in use, the rest in flight)
#endif
// FP32 tile state kept in shared memory instead of registers: the transformed
// lower node plane (rebuilt from the node buffer for each element) and the
// upper-plane forces carried to the next element (one slot per thread).  With
// the first, the FP32 persistent kernel no longer spills under its 128-register
// cap (500^3 inner iteration 6.9 ms, from 9.2); the second costs more shared
// memory traffic than it saves (6.9 ms either way) and stays off.
#ifndef E3D_F32_POLD_SMEM
#define E3D_F32_POLD_SMEM 1
#endif
#ifndef E3D_F32_CARRY_SMEM
#define E3D_F32_CARRY_SMEM 0
#endif
// FP64 stencil: node sums share the adjoint butterflies between neighbouring
// elements (9 instead of 11 additions per component and node).
#ifndef E3D_F64_SHARED_ADJ
#define E3D_F64_SHARED_ADJ 1
#endif
#ifndef E3D_PB_UNROLL_RING
#define E3D_PB_UNROLL_RING (E3D_RING_ZS == 2 ? 4 : 1)  // phase-B nodes in flight per thread, ring kernel
#endif
constexpr int NT = TILE_X * TILE_Y;  // threads per block of the tile kernels

// Device status codes (host maps them to E3D_*).
enum : int { DEV_OK = 0, DEV_TIMEOUT = 1, DEV_BAD_INDEX = 2 };
// PCG status.
enum : int {
  PCG_RUNNING = 0,
  PCG_CONVERGED = 1,
  PCG_HAH = 2,
  PCG_MAXITER = 3,
  PCG_BREAKDOWN = 4,
  PCG_TIMEOUT = 5,
  PCG_REPLACE = 6  // mixed form: the FP32 residual has dropped far enough for an FP64 replacement
};

struct GridDims {
  int nx, ny, nz;
  long long ns;
  int ntx, nty, ntz;  // tiles per direction
  int tz;             // element planes per tile
  long long ntiles;
};

// Length of one tile-edge halo buffer (hx, hy, hd) with w values per plane row.
__host__ __device__ inline long long halo_len(const GridDims& G, int w) { return 3LL * G.ntiles * G.tz * w; }

// Periodic wrap of v into [0, n); the callers pass neighbours (v in [-n, 2n)),
// handled without an integer division.
__host__ __device__ inline int wrapi(int v, int n) {
  if (v >= 0 && v < n) return v;
  if (v < 0 && v >= -n) return v + n;
  if (v >= n && v < 2 * n) return v - n;
  v %= n;
  return v < 0 ? v + n : v;
}

// Node index -> (x, y, z); 32-bit division when the grid allows it (every grid
// up to 2^32 nodes), far cheaper than the 64-bit one.
__device__ __forceinline__ void node_xyz(const GridDims& G, long long m, int& x, int& y, int& z) {
  if (G.ns <= 0xffffffffLL) {
    const unsigned mm = (unsigned)m, nx = (unsigned)G.nx, ny = (unsigned)G.ny;
    const unsigned q = mm / nx;
    x = (int)(mm - q * nx);
    const unsigned r = q / ny;
    y = (int)(q - r * ny);
    z = (int)r;
  } else {
    x = (int)(m % G.nx);
    y = (int)((m / G.nx) % G.ny);
    z = (int)(m / ((long long)G.nx * G.ny));
  }
}

template <typename T>
struct ApplyArgs {
  GridDims g;
  const int32_t* __restrict__ pix;  // 0-based phase per voxel
  const T* __restrict__ cs;         // scaled stiffness table
  int ncs;                          // rows of cs (every phase id is below it)
  const T* __restrict__ x;          // input (or h_old when fused)
  const T* __restrict__ zv;         // z (fused Fletcher-Reeves update only)
  T gamma;                          // FR coefficient
  int reset;                        // 1: h_new = z
  T* __restrict__ hnew;             // fused: h_new written for owned nodes
  T* __restrict__ y;                // in-tile part of K x
  T* __restrict__ hx;               // [3][ntiles][tz][TILE_Y]
  T* __restrict__ hy;               // [3][ntiles][tz][TILE_X]
  T* __restrict__ hd;               // [3][ntiles][tz]
  T* __restrict__ du;               // deferred correction update (DEFER_U): du -= lam_prev * x, own nodes
  T lam_prev;
};

template <typename T, bool CARRY, int TY = TILE_Y>
struct ApplySmemT {
  T node[2][3][(TILE_X + 1) * (TY + 1)];
  T r[9][TILE_X * TY];
};
template <typename T, int TY>
struct ApplySmemT<T, true, TY> {
  T node[2][3][(TILE_X + 1) * (TY + 1)];
  T r[9][TILE_X * TY];
  T carry[12][TILE_X * TY];
};
template <typename T, int TY = TILE_Y>
using ApplySmem = ApplySmemT<T, sizeof(T) == 4 && E3D_F32_CARRY_SMEM != 0, TY>;

// ---------------------------------------------------------------------------
// TMA plane ring of the fused FP32 stencil.  One stage holds one node plane of
// a tile: for h_old and z the main 32x8 box, the +x column box (4x8), the +y
// row box (32x1) and the corner box (4x1), three components each, then the
// tile's 32x8 phase ids.  Warp 0 keeps the ring full (one lane per box),
// running ahead across the block's tiles; a stage is refilled once every
// thread has read it (after the block barrier of the step that last reads it),
// and consumers wait on the stage's mbarrier with a wall-clock limit.
constexpr int kRingMain = 3 * 32 * 8 * 4;
constexpr int kRingCol = 3 * 4 * 8 * 4;
constexpr int kRingRow = 3 * 32 * 1 * 4;
constexpr int kRingCorner = 3 * 4 * 1 * 4;
constexpr int kRingVec = kRingMain + kRingCol + kRingRow + 128;  // corner box padded to 128 B
constexpr int kRingPix = 32 * 8 * 4;
constexpr int kStageBytes = 2 * kRingVec + kRingPix;
constexpr unsigned kPlaneTx = 2u * (kRingMain + kRingCol + kRingRow + kRingCorner) + kRingPix;
constexpr int kRingSmemBytes = E3D_TMA_STAGES * kStageBytes + 128;  // + alignment slack
static_assert(kRingVec % 128 == 0 && kStageBytes % 128 == 0, "TMA destinations must stay 128-byte aligned");

// Producer state, written by lane 0 of warp 0 and read by warp 0; kept in
// shared memory so it does not occupy registers of every thread.
struct RingCursor {
  long long ptile, tstride, tend;
  const CUtensorMap* hmap;  // the four maps of the buffer read as h_old
  int pzl, pzend;
  unsigned int issued;
};

struct PlaneRing {
  unsigned char* stage;   // E3D_TMA_STAGES * kStageBytes, 128-byte aligned
  uint64_t* full;         // one mbarrier per stage
  RingCursor* cur;        // shared memory
  const PlaneMaps* maps;  // tensor maps in global memory
  int* err;
  unsigned long long timeout_ns;
  unsigned int q;  // planes consumed by this block (same in every thread)
  int failed;      // a wait ran out or an error is flagged: stop waiting and issuing
};

__device__ __forceinline__ void ring_tile_span(const GridDims& G, long long t, int& zl0, int& zl1) {
  const int tiz = (int)(t / ((long long)G.ntx * G.nty));
  const int z0 = tiz * G.tz;
  zl0 = z0 - 1;
  zl1 = z0 + min(G.tz, G.nz - z0);
}

// Warp 0: start the loads of the cursor's next plane into its stage; lane 0
// sets the expected bytes, lanes 0-8 issue one box each, lane 0 advances the
// cursor.
__device__ __forceinline__ void ring_issue(PlaneRing& R, const GridDims& G) {
  RingCursor& C = *R.cur;
  const int lane = threadIdx.x;  // warp 0 only
  // warp-uniform decisions (the cursor was published by the last __syncwarp);
  // the error flag in global memory is read only on the slow path of a wait
  const bool bad = __any_sync(0xffffffffu, R.failed);
  if (bad) R.failed = 1;
  if (bad || C.ptile >= C.tend) return;
  const long long t = C.ptile;
  const int tix = (int)(t % G.ntx);
  const int tiy = (int)((t / G.ntx) % G.nty);
  const int x0 = tix * TILE_X, y0 = tiy * TILE_Y;
  const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0);
  // +x column / +y row of the tile, wrapped; x starts are multiples of 32 or 0
  const int xc = (x0 + wx == G.nx) ? 0 : x0 + wx;
  const int yr = (y0 + wy == G.ny) ? 0 : y0 + wy;
  const int zp = wrapi(C.pzl, G.nz);
  const unsigned s = C.issued % E3D_TMA_STAGES;
  unsigned char* st = R.stage + (size_t)s * kStageBytes;
  uint64_t* bar = R.full + s;
  if (lane == 0) mbar_arrive_expect_tx(bar, kPlaneTx);
  __syncwarp();
  if (lane < 8) {
    const int v = lane >> 2, kind = lane & 3;  // vector (h_old, z) and box kind
    const CUtensorMap* m = (v ? R.maps->z : C.hmap) + kind;
    const int off = v * kRingVec + (kind == BOX_MAIN ? 0 : kind == BOX_COL ? kRingMain
                                                   : kind == BOX_ROW ? kRingMain + kRingCol
                                                                     : kRingMain + kRingCol + kRingRow);
    const int bx = (kind == BOX_COL || kind == BOX_CORNER) ? xc : x0;
    const int by = (kind == BOX_ROW || kind == BOX_CORNER) ? yr : y0;
    tma_load_4d(st + off, m, bx, by, zp, 0, bar);
  } else if (lane == 8) {
    tma_load_3d(st + 2 * kRingVec, &R.maps->pix, x0, y0, zp, bar);
  }
  __syncwarp();
  if (lane == 0) {
    C.issued += 1;
    if (++C.pzl > C.pzend) {
      C.ptile += C.tstride;
      if (C.ptile < C.tend) ring_tile_span(G, C.ptile, C.pzl, C.pzend);
    }
  }
  __syncwarp();
}

// Once per kernel: barriers, from thread 0; followed by __syncthreads.
__device__ __forceinline__ void ring_setup(PlaneRing& R, unsigned char* dyn, uint64_t* bars, RingCursor* cur,
                                           const PlaneMaps* maps, int* err, unsigned long long timeout_ns) {
  const uint32_t a = smem_u32(dyn);
  R.stage = dyn + ((128u - (a & 127u)) & 127u);
  R.full = bars;
  R.cur = cur;
  R.maps = maps;
  R.err = err;
  R.timeout_ns = timeout_ns;
  R.q = 0;
  R.failed = 0;
  if (threadIdx.x == 0) {
    cur->ptile = cur->tend = 0;
    cur->tstride = 1;
    cur->hmap = maps->h0;
    cur->pzl = cur->pzend = 0;
    cur->issued = 0;
    for (int i = 0; i < E3D_TMA_STAGES; ++i) mbar_init(bars + i, 1);
    fence_mbar_init();
  }
  // (the caller's __syncthreads publishes the cursor and the barriers)
}

// Start of one stencil pass over tiles first, first+stride, ... < tend, reading
// h_old through hmap.  Every plane of the previous pass has been consumed.
__device__ __forceinline__ void ring_begin(PlaneRing& R, const GridDims& G, const CUtensorMap* hmap,
                                           long long first, long long stride, long long tend) {
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      fence_proxy_async_all();  // this block's and (after the grid barrier) the grid's writes before TMA reads
      RingCursor& C = *R.cur;
      C.hmap = hmap;
      C.ptile = first;
      C.tstride = stride;
      C.tend = tend;
      if (first < tend) ring_tile_span(G, first, C.pzl, C.pzend);
    }
    __syncwarp();
    for (int i = 0; i < E3D_TMA_STAGES; ++i) ring_issue(R, G);
  }
}

// All threads: wait until plane number n (n - R.q < E3D_TMA_STAGES) has
// landed; returns its stage.
__device__ __forceinline__ const unsigned char* ring_wait(PlaneRing& R, unsigned n) {
  const unsigned s = n % E3D_TMA_STAGES;
  // fast path: one probe; the slow path polls the error flag and the clock
  if (!R.failed && !mbar_try_wait(R.full + s, (n / E3D_TMA_STAGES) & 1u)) {
    if (!mbar_wait(R.full + s, (n / E3D_TMA_STAGES) & 1u, R.timeout_ns, R.err)) {
      if (*(volatile int*)R.err == DEV_OK) atomicExch(R.err, DEV_TIMEOUT);
      R.failed = 1;
    }
  }
  return R.stage + (size_t)s * kStageBytes;
}

// Stage address of plane number n (already waited for).
__device__ __forceinline__ const unsigned char* ring_stage(const PlaneRing& R, unsigned n) {
  return R.stage + (size_t)(n % E3D_TMA_STAGES) * kStageBytes;
}

// All threads, after a __syncthreads that follows every read of the oldest
// plane R.q: its stage is free (the barrier orders those reads before the
// refill); warp 0 refills it with the cursor's next plane.
__device__ __forceinline__ void ring_release(PlaneRing& R, const GridDims& G) {
  R.q += 1;
  if (threadIdx.x < 32) ring_issue(R, G);
}

// Thread 0, before the block exits: wait (bounded) for the last plane issued
// into each stage, so that no copy is still in flight after a failed pass.
// Phases complete in order, so the last one covers the earlier ones.
__device__ __forceinline__ void ring_drain(PlaneRing& R) {
  if (threadIdx.x != 0) return;
  const unsigned issued = R.cur->issued;
  for (unsigned s = 0; s < E3D_TMA_STAGES && s < issued; ++s) {
    const unsigned n = s + E3D_TMA_STAGES * ((issued - 1 - s) / E3D_TMA_STAGES);
    (void)mbar_wait(R.full + s, (n / E3D_TMA_STAGES) & 1u, 1000000000ull);
  }
}

// Barrier of the 128 threads that share a tile: the whole block, or, GROUPED,
// one of the groups of 128 that make up a larger block.
template <bool GROUPED>
__device__ __forceinline__ void tile_sync() {
  if constexpr (GROUPED)
    asm volatile("bar.sync %0, 128;" ::"r"(1 + (int)(threadIdx.x >> 7)) : "memory");
  else
    __syncthreads();
}

// One tile: TILE_X x TILE_Y element columns marching through tz element planes
// (plus one redundant plane below).  Each thread owns node column (x0+tx,
// y0+ty) and the element whose lower corner it is.  Element forces are summed
// into the nodes inside the tile through shared memory; the contributions to
// the nodes just past the tile's high-x / high-y edges go to the halo buffers
// and are added by the consumer (apply_finish / the PCG update), which keeps
// every sum in a fixed order.  FUSED: the input is h_new = z + gamma*h_old (or
// z on reset) formed on load -- the Fletcher-Reeves update of the previous
// iteration (src/elas3dxtal_pcg.f90:1988-1995) folded into this pass -- and
// h_new is stored for the tile's own nodes.  Returns this thread's share of
// h_new . (K h_new) through hAh.
//
// TY: rows of a tile (and warps of a block, or, GROUPED, of a group of 128 threads).
// from, planes: the part of the tile's planes to form.
template <typename T, bool FUSED, bool POLD_SMEM = (sizeof(T) == 4 && E3D_F32_POLD_SMEM != 0), bool DEFER_U = false,
          int TY = TILE_Y, bool GROUPED = false>
__device__ void apply_tile(const ApplyArgs<T>& A, long long tile, ApplySmem<T, TY>& sm, double& hAh, int from = 0,
                           int planes = 0x7fffffff) {
  constexpr int TILE_Y = TY;
  static_assert(!GROUPED || TILE_X * TY == 128, "a group is 128 threads");
  const GridDims& G = A.g;
  const int tid = GROUPED ? threadIdx.x % (TILE_X * TY) : threadIdx.x;
  const int tx = tid % TILE_X, ty = tid / TILE_X;
  const int tix = (int)(tile % G.ntx);
  const int tiy = (int)((tile / G.ntx) % G.nty);
  const int tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz + from;
  const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(planes, min(G.tz - from, G.nz - z0));
  const bool active = (tx < wx) && (ty < wy);
  const int xg = x0 + tx, yg = y0 + ty;
  const long long ns = G.ns;
  const long long nxy = (long long)G.nx * G.ny;
  const int nhalo = wx + wy + 1;
  // halo node (lx, ly) for loader thread q = tid < nhalo
  int hlx = 0, hly = 0;
  if (tid < wy) {
    hlx = wx;
    hly = tid;
  } else if (tid < wy + wx) {
    hlx = tid - wy;
    hly = wy;
  } else {
    hlx = wx;
    hly = wy;
  }
  const int hgx = wrapi(x0 + hlx, G.nx), hgy = wrapi(y0 + hly, G.ny);

  // Raw loads of one node plane are issued a step ahead (prefetch) so they are
  // in flight while the previous element computes; commit forms h_new and
  // stores the plane into shared memory.
  T pz_own[3], px_own[3], pz_h[3], px_h[3], pu_own[3];
  const bool need_x = !FUSED || !A.reset;
  auto prefetch = [&](int zl) {
    const int zp = wrapi(zl, G.nz);
    if (active) {
      const long long m = E3D_IDX((long long)xg + (long long)G.nx * yg + nxy * zp, ns);
      const bool own = zl >= z0 && zl < z0 + wz;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (need_x || (DEFER_U && own)) px_own[c] = __ldcg(A.x + m + c * ns);
        if (FUSED) pz_own[c] = __ldcg(A.zv + m + c * ns);
        if (DEFER_U && own) pu_own[c] = A.du[m + c * ns];
      }
    }
    if (tid < nhalo) {
      const long long m = E3D_IDX((long long)hgx + (long long)G.nx * hgy + nxy * zp, ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (need_x) px_h[c] = __ldcg(A.x + m + c * ns);
        if (FUSED) pz_h[c] = __ldcg(A.zv + m + c * ns);
      }
    }
  };
  auto combine = [&](const T (&zz)[3], const T (&xx)[3], T (&v)[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (FUSED)
        v[c] = A.reset ? zz[c] : fma_(A.gamma, xx[c], zz[c]);
      else
        v[c] = xx[c];
    }
  };
  auto commit = [&](int zl, bool own) {
    const int zp = wrapi(zl, G.nz);
    T* buf0 = sm.node[(zl + 2) & 1][0];
    const int stride = (TILE_X + 1) * (TILE_Y + 1);
    if (active) {
      T v[3];
      combine(pz_own, px_own, v);
      if (FUSED && own) {
        const long long m = E3D_IDX((long long)xg + (long long)G.nx * yg + nxy * zp, ns);
#pragma unroll
        for (int c = 0; c < 3; ++c) A.hnew[m + c * ns] = v[c];
        if constexpr (DEFER_U) {
          // nothing pending at the first step of a launch (lam_prev = 0): h_old
          // may then hold another solve's direction and is not used
          if (A.lam_prev != T(0)) {
#pragma unroll
            for (int c = 0; c < 3; ++c) A.du[m + c * ns] = pu_own[c] - A.lam_prev * px_own[c];
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) buf0[c * stride + ty * (TILE_X + 1) + tx] = v[c];
    }
    if (tid < nhalo) {
      T v[3];
      combine(pz_h, px_h, v);
#pragma unroll
      for (int c = 0; c < 3; ++c) buf0[E3D_IDX(c * stride + hly * (TILE_X + 1) + hlx, 3 * stride)] = v[c];
    }
  };
  auto read_corners = [&](int zl, T (&v)[3][4]) {
    const T* buf0 = sm.node[(zl + 2) & 1][0];
    const int stride = (TILE_X + 1) * (TILE_Y + 1);
    const int o = ty * (TILE_X + 1) + tx;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v[c][0] = buf0[c * stride + o];
      v[c][1] = buf0[c * stride + o + 1];
      v[c][2] = buf0[c * stride + o + TILE_X + 1];
      v[c][3] = buf0[c * stride + o + TILE_X + 2];
    }
  };

  constexpr bool kPoldSmem = POLD_SMEM;
  constexpr bool kCarrySmem = sizeof(T) == 4 && E3D_F32_CARRY_SMEM != 0;
  // FP64: the node sums share the adjoint's partial butterflies between
  // neighbouring elements (see the node-sum step below).
  constexpr bool kShareAdj = sizeof(T) == 8 && E3D_F64_SHARED_ADJ != 0;
  T Pold[3][4], carry[3][4];
  // FP32: the tile's share of h.Ah is summed in FP32 and added to the FP64
  // accumulator once per tile; FP64: every node's term goes straight into it.
  float dot32 = 0.f;
  auto add_dot = [&](T v) {
    if constexpr (sizeof(T) == 4)
      dot32 += v;
    else
      hAh += (double)v;
  };
  const long long ecol = (long long)xg + (long long)G.nx * yg;  // element column
  prefetch(z0 - 1);
  commit(z0 - 1, false);
  tile_sync<GROUPED>();
  if (!kPoldSmem && active) {
    T v0[3][4];
    read_corners(z0 - 1, v0);
#pragma unroll
    for (int c = 0; c < 3; ++c) had_xy(v0[c], Pold[c]);
  }
  prefetch(z0);
  int ph_cur = active ? __ldcs(A.pix + E3D_IDX(ecol + nxy * wrapi(z0 - 1, G.nz), ns)) : 0;
  const int htiles_stride = G.tz;  // per-tile plane stride in halo buffers
  for (int k = z0 - 1; k < z0 + wz; ++k) {
    const bool own_next = (k + 1 >= z0) && (k + 1 < z0 + wz);
    commit(k + 1, own_next);
    tile_sync<GROUPED>();
    if (k + 2 <= z0 + wz) prefetch(k + 2);
    const int ph_nxt =
        (active && k + 1 < z0 + wz) ? __ldcs(A.pix + E3D_IDX(ecol + nxy * wrapi(k + 1, G.nz), ns)) : 0;
    T rr[3][4];
    if (active) {
      T nxt[3][4];
      read_corners(k + 1, nxt);
      if constexpr (kPoldSmem) {  // plane k, intact until the barrier that ends this step
        T v0[3][4];
        read_corners(k, v0);
#pragma unroll
        for (int c = 0; c < 3; ++c) had_xy(v0[c], Pold[c]);
      }
      T Pn[3][4];
      T h[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        had_xy(nxt[c], Pn[c]);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          h[c][b] = Pn[c][b] + Pold[c][b];
          h[c][b + 4] = Pn[c][b] - Pold[c][b];
        }
      }
      T f[3][8];
      if constexpr (sizeof(T) == 4)
        element_modal_f32(A.cs + E3D_IDX(ph_cur, A.ncs) * kCs32Stride, h[0], h[1], h[2], f[0], f[1], f[2]);
      else
        element_modal<T>(A.cs + E3D_IDX(ph_cur, A.ncs) * kCsStride, h[0], h[1], h[2], f[0], f[1], f[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T lo[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          lo[b] = f[c][b] - f[c][b + 4];
          const T hi = f[c][b] + f[c][b + 4];
          if constexpr (kCarrySmem) {
            if (k >= z0) lo[b] += sm.carry[4 * c + b][tid];
            sm.carry[4 * c + b][tid] = hi;
          } else {
            if (k >= z0) lo[b] += carry[c][b];
            carry[c][b] = hi;
          }
        }
        if (k >= z0) {
          if constexpr (kShareAdj) {  // rr = e0, e1, g0, g1 of had_xy_adj; the butterfly's last step is shared
            rr[c][0] = lo[0] - lo[2];
            rr[c][1] = lo[0] + lo[2];
            rr[c][2] = lo[1] - lo[3];
            rr[c][3] = lo[1] + lo[3];
          } else {
            had_xy_adj(lo, rr[c]);
          }
        }
        if constexpr (!kPoldSmem) {
#pragma unroll
          for (int b = 0; b < 4; ++b) Pold[c][b] = Pn[c][b];
        }
      }
    }
    // plane k's values for the dot products, read before the barrier below
    // (after it, the next step may overwrite this buffer with plane k+2)
    T hk[3][4];
    if (k >= z0 && active) {
      const T* cb = sm.node[(k + 2) & 1][0];
      constexpr int cst = (TILE_X + 1) * (TILE_Y + 1);
      const int o = ty * (TILE_X + 1) + tx;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        hk[c][0] = cb[c * cst + o];
        hk[c][1] = tx == wx - 1 ? cb[c * cst + o + 1] : T(0);
        hk[c][2] = ty == wy - 1 ? cb[c * cst + o + TILE_X + 1] : T(0);
        hk[c][3] = (tx == wx - 1 && ty == wy - 1) ? cb[c * cst + o + TILE_X + 2] : T(0);
      }
    }
    if (kShareAdj && k >= z0) {
      // Node (x, y) collects r0(x,y) + r1(x-1,y) + r2(x,y-1) + r3(x-1,y-1) with
      // r0 = e0 - g0, r1 = e0 + g0, r2 = e1 - g1, r3 = e1 + g1.  Grouped as
      // E = e0(x,y) + e1(x,y-1), G = g0(x,y) + g1(x,y-1) (the element below
      // hands over e1, g1 through shared memory) and then
      // (E - G)(x,y) + (E + G)(x-1,y) (the lane to the left hands over E + G):
      // 9 additions per component and node instead of 11.  Contributions from
      // across the tile's low edges arrive through the halos, as before.
      if (active) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sm.r[2 * c + 0][tid] = rr[c][1];  // e1: to the element at y+1
          sm.r[2 * c + 1][tid] = rr[c][3];  // g1
        }
      }
      tile_sync<GROUPED>();
      if (ty < wy) {  // warp-uniform: every lane of the row takes part in the shuffles
        const int lz = k - z0 + from;
        T acc[3], pxv[3], hyv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          T E = T(0), Gs = T(0), e1 = T(0), g1 = T(0);
          if (active) {
            E = rr[c][0];
            Gs = rr[c][2];
            if (ty > 0) {
              E += sm.r[2 * c + 0][tid - TILE_X];
              Gs += sm.r[2 * c + 1][tid - TILE_X];
            }
            e1 = rr[c][1];
            g1 = rr[c][3];
          }
          const T P = E + Gs;  // r1 + r3 of this column: to node (x+1, y)
          const T R = e1 + g1;  // r3 alone: to node (x+1, y+1) of the next row
          const T Pl = __shfl_up_sync(0xffffffffu, P, 1);
          const T Rl = __shfl_up_sync(0xffffffffu, R, 1);
          acc[c] = tx > 0 ? (E - Gs) + Pl : (E - Gs);
          pxv[c] = P;
          hyv[c] = tx > 0 ? (e1 - g1) + Rl : (e1 - g1);
          rr[c][3] = R;
        }
        if (active) {
          const long long m = E3D_IDX((long long)xg + (long long)G.nx * yg + nxy * wrapi(k, G.nz), ns);
#pragma unroll
          for (int c = 0; c < 3; ++c) A.y[m + c * ns] = acc[c];
          add_dot(hk[0][0] * acc[0] + hk[1][0] * acc[1] + hk[2][0] * acc[2]);
          const long long hb = tile * htiles_stride + lz;
          if (tx == wx - 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) A.hx[E3D_IDX(((long long)c * G.ntiles * htiles_stride + hb) * TILE_Y + ty, halo_len(G, TILE_Y))] = pxv[c];
            add_dot(hk[0][1] * pxv[0] + hk[1][1] * pxv[1] + hk[2][1] * pxv[2]);
          }
          if (ty == wy - 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) A.hy[E3D_IDX(((long long)c * G.ntiles * htiles_stride + hb) * TILE_X + tx, halo_len(G, TILE_X))] = hyv[c];
            add_dot(hk[0][2] * hyv[0] + hk[1][2] * hyv[1] + hk[2][2] * hyv[2]);
          }
          if (tx == wx - 1 && ty == wy - 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) A.hd[E3D_IDX((long long)c * G.ntiles * htiles_stride + hb, halo_len(G, 1))] = rr[c][3];
            add_dot(hk[0][3] * rr[0][3] + hk[1][3] * rr[1][3] + hk[2][3] * rr[2][3]);
          }
        }
      }
    } else if (k >= z0) {
      if (active) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sm.r[3 * c + 0][tid] = rr[c][1];  // to node (x+1, y)
          sm.r[3 * c + 1][tid] = rr[c][2];  // to node (x, y+1)
          sm.r[3 * c + 2][tid] = rr[c][3];  // to node (x+1, y+1)
        }
      }
      tile_sync<GROUPED>();
      if (active) {
        const int lz = k - z0 + from;
        const long long m = E3D_IDX((long long)xg + (long long)G.nx * yg + nxy * wrapi(k, G.nz), ns);
        T hxv[3], hyv[3], acc[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[c] = rr[c][0];
          if (tx > 0) acc[c] += sm.r[3 * c + 0][tid - 1];
          if (ty > 0) acc[c] += sm.r[3 * c + 1][tid - TILE_X];
          if (tx > 0 && ty > 0) acc[c] += sm.r[3 * c + 2][tid - TILE_X - 1];
          A.y[m + c * ns] = acc[c];
          hxv[c] = rr[c][1] + (ty > 0 ? sm.r[3 * c + 2][tid - TILE_X] : T(0));
          hyv[c] = rr[c][2] + (tx > 0 ? sm.r[3 * c + 2][tid - 1] : T(0));
        }
        // per-node dot in T, accumulated in FP64
        add_dot(hk[0][0] * acc[0] + hk[1][0] * acc[1] + hk[2][0] * acc[2]);
        const long long hb = tile * htiles_stride + lz;
        if (tx == wx - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hx[E3D_IDX(((long long)c * G.ntiles * htiles_stride + hb) * TILE_Y + ty, halo_len(G, TILE_Y))] = hxv[c];
          add_dot(hk[0][1] * hxv[0] + hk[1][1] * hxv[1] + hk[2][1] * hxv[2]);
        }
        if (ty == wy - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hy[E3D_IDX(((long long)c * G.ntiles * htiles_stride + hb) * TILE_X + tx, halo_len(G, TILE_X))] = hyv[c];
          add_dot(hk[0][2] * hyv[0] + hk[1][2] * hyv[1] + hk[2][2] * hyv[2]);
        }
        if (tx == wx - 1 && ty == wy - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hd[E3D_IDX((long long)c * G.ntiles * htiles_stride + hb, halo_len(G, 1))] = rr[c][3];
          add_dot(hk[0][3] * rr[0][3] + hk[1][3] * rr[1][3] + hk[2][3] * rr[2][3]);
        }
      }
    } else if constexpr (kPoldSmem) {
      tile_sync<GROUPED>();  // plane z0-1 was re-read: the next step refills its buffer
    }
    ph_cur = ph_nxt;
  }
  if constexpr (sizeof(T) == 4) hAh += (double)dot32;
}

__device__ __forceinline__ void cp_async_4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------
// FP32 tile with two elements a thread (e3d_f32x2.cuh): 32 x 8 columns, 128
// threads; thread (tx, tr) has rows 2 tr and 2 tr + 1.
constexpr int kF2Threads = TILE_X * TILE_Y / 2;

// Planes in flight: with one, half of the stalls were waits for it (sixty solves of
// 32^3 to 88^3: 0.64 s; with two 0.60, with three the same).
constexpr int kF2Depth = 2;

struct F2Smem {
  float node[3][3][(TILE_Y + 1) * (TILE_X + 1)];  // plane k in one of three, rows of TILE_X + 1
  float r[2][6][kF2Threads];                      // forces to the row above, by plane parity
  // a thread's own slots: one plane's values in flight (z, h_old, du; rows a and
  // b; then the halo node's z and h_old), and what it carries up the column
  float raw[kF2Depth][18][kF2Threads];
  float raw_halo[kF2Depth][6][kF2Threads];
  f2 carry[12][kF2Threads];
  f2 pold[12][kF2Threads];
};

// The fused FP32 pass of apply_tile<float, true> over one tile: same results up
// to the order of sums, same halos.  One barrier a plane: between two of them the
// nodes of one plane are summed and the elements of the next formed, while the
// loads of the plane after that are in flight.  The dot product h . K h is the
// sum of the element energies, from values at hand in the element.  DEFER_U: du -=
// lam_prev * h_old for the own nodes on the way.  FULL: the tile has all its 32 x 8
// columns, so that nothing is masked.
__device__ __forceinline__ float* at_byte(float* p, unsigned long long o) {
  return reinterpret_cast<float*>(reinterpret_cast<char*>(p) + o);
}
__device__ __forceinline__ const float* at_byte(const float* p, unsigned long long o) {
  return reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + o);
}

// Whether a tile has all its 32 x 8 columns.
__device__ __forceinline__ bool tile_full(const GridDims& G, long long tile) {
  const long long txy = tile % ((long long)G.ntx * G.nty);
  return (txy % G.ntx + 1) * TILE_X <= G.nx && (txy / G.ntx + 1) * TILE_Y <= G.ny;
}

template <bool DEFER_U, bool FULL, bool GROUPED>
static __device__ __forceinline__ void apply_tile_f2(const ApplyArgs<float>& A, long long tile, F2Smem& sm,
                                                     double& hAh) {
  const GridDims& G = A.g;
  const int tid = threadIdx.x % kF2Threads;
  const int tx = tid % TILE_X, tr = tid / TILE_X, ya = 2 * tr;
  const int tix = (int)(tile % G.ntx);
  const int tiy = (int)((tile / G.ntx) % G.nty);
  const int tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
  const int wx = FULL ? TILE_X : min(TILE_X, G.nx - x0), wy = FULL ? TILE_Y : min(TILE_Y, G.ny - y0);
  const int wz = min(G.tz, G.nz - z0);
  const bool act_a = FULL || (tx < wx && ya < wy), act_b = FULL || (tx < wx && ya + 1 < wy);
  const unsigned nx = (unsigned)G.nx, nxy = nx * (unsigned)G.ny;
  const long long ns = G.ns;
  constexpr int kRow = TILE_X + 1;
  const unsigned own = (unsigned)(x0 + tx) + nx * (unsigned)(y0 + ya);
  // halo node of loader thread tid < wx + wy + 1
  const int nhalo = wx + wy + 1;
  int hlx = wx, hly = wy;
  if (tid < wy)
    hly = tid;
  else if (tid < wy + wx)
    hlx = tid - wy;
  const unsigned halo = (unsigned)wrapi(x0 + hlx, G.nx) + nx * (unsigned)wrapi(y0 + hly, G.ny);
  const bool reset = A.reset != 0, owe = DEFER_U && A.lam_prev != 0.f;
  const int zend = z0 + wz;

  // raw slot of field f (z 0, h_old 1, du 2), component c, row q
  auto slot = [](int f, int c, int q) { return 6 * f + 2 * c + q; };
  auto load = [&](int zl) {
    const int d = (zl - z0 + 1) % kF2Depth;
    if (zl <= zend) {
    const int zw = wrapi(zl, G.nz);
    const bool mine = DEFER_U && zl >= z0 && zl < zend, need_x = !reset || mine;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (q ? act_b : act_a) {
        const unsigned long long o = node_bytes4(E3D_IDX(node_of(own + (q ? nx : 0u), nxy, zw), ns));
#pragma unroll
        for (int c = 0; c < 3; ++c) cp_async_4(&sm.raw[d][slot(0, c, q)][tid], at_byte(A.zv + c * ns, o));
        if (need_x)
#pragma unroll
          for (int c = 0; c < 3; ++c) cp_async_4(&sm.raw[d][slot(1, c, q)][tid], at_byte(A.x + c * ns, o));
        if (mine)
#pragma unroll
          for (int c = 0; c < 3; ++c) cp_async_4(&sm.raw[d][slot(2, c, q)][tid], at_byte(A.du + c * ns, o));
      }
    if (tid < nhalo) {
      const unsigned long long o = node_bytes4(E3D_IDX(node_of(halo, nxy, zw), ns));
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async_4(&sm.raw_halo[d][c][tid], at_byte(A.zv + c * ns, o));
      if (!reset)
#pragma unroll
        for (int c = 0; c < 3; ++c) cp_async_4(&sm.raw_halo[d][3 + c][tid], at_byte(A.x + c * ns, o));
    }
    }
    cp_async_commit();
  };
  auto commit = [&](int zl, float (&buf)[3][(TILE_Y + 1) * kRow]) {
    const int d = (zl - z0 + 1) % kF2Depth;
    cp_async_wait<kF2Depth - 1>();
    const bool mine = zl >= z0 && zl < zend;
    // every slot is read before anything is stored: a store in between would
    // hold back the reads behind it
    float z[6], x[6], du[6], zh[3], xh[3];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      z[i] = sm.raw[d][i][tid];
      x[i] = sm.raw[d][6 + i][tid];
      du[i] = DEFER_U ? sm.raw[d][12 + i][tid] : 0.f;
    }
    const bool halo_thread = tid < nhalo;
    if (halo_thread) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        zh[c] = sm.raw_halo[d][c][tid];
        xh[c] = sm.raw_halo[d][3 + c][tid];
      }
    }
    float v[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) v[i] = reset ? z[i] : fmaf(A.gamma, x[i], z[i]);
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (q ? act_b : act_a) {
#pragma unroll
        for (int c = 0; c < 3; ++c) buf[c][(ya + q) * kRow + tx] = v[2 * c + q];
      }
    if (halo_thread) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        buf[c][E3D_IDX(hly * kRow + hlx, (TILE_Y + 1) * kRow)] = reset ? zh[c] : fmaf(A.gamma, xh[c], zh[c]);
    }
    if (mine) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (q ? act_b : act_a) {
          const unsigned long long o = node_bytes4(E3D_IDX(node_of(own + (q ? nx : 0u), nxy, zl), ns));
#pragma unroll
          for (int c = 0; c < 3; ++c) *at_byte(A.hnew + c * ns, o) = v[2 * c + q];
          // nothing pending at the first step of a launch (lam_prev = 0): h_old
          // may then hold another solve's direction and is not used
          if (owe)
#pragma unroll
            for (int c = 0; c < 3; ++c) *at_byte(A.du + c * ns, o) = du[2 * c + q] - A.lam_prev * x[2 * c + q];
        }
    }
  };
  // xy transform of a plane for both elements: P[by * 2 + bx]
  auto plane_transform = [&](const float (&buf)[3][(TILE_Y + 1) * kRow], f2 (&P)[3][4]) {
    float w[3][6];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 6; ++i) w[c][i] = buf[c][(ya + i / 2) * kRow + tx + (i & 1)];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const f2 l = f2_pack(w[c][0], w[c][2]), r = f2_pack(w[c][1], w[c][3]);
      const f2 s = f2_add(r, l), d = f2_sub(r, l);
      const float s2 = w[c][5] + w[c][4], d2 = w[c][5] - w[c][4];
      const f2 su = f2_pack(f2_hi(s), s2), du = f2_pack(f2_hi(d), d2);  // of the rows above
      P[c][0] = f2_add(su, s);
      P[c][2] = f2_sub(su, s);
      P[c][1] = f2_add(du, d);
      P[c][3] = f2_sub(du, d);
    }
  };
  // sums of the last element plane that wait for the rows below and the lanes to the left
  float e_a[3], g_a[3], e_b[3], g_b[3];  // (those of plane z0 - 1 are not used)
  const bool top = tr == (wy - 1) / 2, odd = !FULL && (wy & 1) != 0;
  const long long per_c = G.ntiles * (long long)G.tz;
  auto node_sums = [&](int k) {
    const float(*r)[kF2Threads] = sm.r[k & 1];
    const unsigned long long o = node_bytes4(node_of(own, nxy, k));
    const long long hb = tile * G.tz + (k - z0);
    float ea[3], ga[3], rb[6], na[3], nb[3];
#pragma unroll
    for (int i = 0; i < 6; ++i) rb[i] = tr > 0 ? r[i][tid - TILE_X] : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ea[c] = e_a[c] + rb[c];
      ga[c] = g_a[c] + rb[3 + c];
      const float gl = __shfl_up_sync(0xffffffffu, ga[c], 1), hl = __shfl_up_sync(0xffffffffu, g_b[c], 1);
      na[c] = tx > 0 ? ea[c] + gl : ea[c];
      nb[c] = tx > 0 ? e_b[c] + hl : e_b[c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (act_a) *at_byte(A.y + E3D_IDX(c * ns, 3 * ns), o) = na[c];
      if (act_b) *at_byte(A.y + E3D_IDX(c * ns, 3 * ns), o + node_bytes4(nx)) = nb[c];
    }
    if (tx == wx - 1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float* hx = A.hx + E3D_IDX((c * per_c + hb) * TILE_Y + ya, 3 * per_c * TILE_Y);
        if (act_a) hx[0] = ga[c];
        if (act_b) hx[1] = g_b[c];
      }
    }
    if (top) {  // warp-uniform: the row past the tile, element b's rows above or, of an odd tile, b's own
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float gt = odd ? g_b[c] : r[3 + c][tid], et = odd ? e_b[c] : r[c][tid];
        const float gtl = __shfl_up_sync(0xffffffffu, gt, 1);
        if (tx < wx) A.hy[E3D_IDX((c * per_c + hb) * TILE_X + tx, 3 * per_c * TILE_X)] = tx > 0 ? et + gtl : et;
        if (tx == wx - 1) A.hd[E3D_IDX(c * per_c + hb, 3 * per_c)] = gt;
      }
    }
  };

  f2 w1 = 0, w2 = 0, w3 = 0;  // element energies by Hadamard order
#pragma unroll
  for (int i = 0; i < kF2Depth; ++i) load(z0 - 1 + i);
  commit(z0 - 1, sm.node[0]);
  load(z0 - 1 + kF2Depth);
  commit(z0, sm.node[1]);
  load(z0 + kF2Depth);
  tile_sync<GROUPED>();
  {
    f2 P[3][4];
    plane_transform(sm.node[0], P);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int b = 0; b < 4; ++b) sm.pold[4 * c + b][tid] = P[c][b];
  }
  int b0 = 0;  // buffer of plane k
  const int32_t* pix = A.pix;
  auto phase = [&](int z, int& pa, int& pb) {
    const unsigned m = node_of(own, nxy, wrapi(z, G.nz));
    pa = act_a ? __ldcs(pix + E3D_IDX(m, ns)) : 0;
    pb = act_b ? __ldcs(pix + E3D_IDX(m + nx, ns)) : 0;
  };
  int pa, pb;
  phase(z0 - 1, pa, pb);
  for (int k = z0 - 1; k < zend; ++k) {
    const int b1 = b0 == 2 ? 0 : b0 + 1, b2 = b1 == 2 ? 0 : b1 + 1;  // of planes k + 1 and k + 2
    float4 qa[6], qb[6];
    {
      const float4* ra = reinterpret_cast<const float4*>(A.cs + E3D_IDX(pa, A.ncs) * kCs32Stride);
      const float4* rb = reinterpret_cast<const float4*>(A.cs + E3D_IDX(pb, A.ncs) * kCs32Stride);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        qa[i] = __ldg(ra + i);
        qb[i] = __ldg(rb + i);
      }
    }
    if (k + 2 <= zend) commit(k + 2, sm.node[b2]);
    load(k + 2 + kF2Depth);
    int na = 0, nb = 0;
    if (k + 1 < zend) phase(k + 1, na, nb);
    if (k > z0) node_sums(k - 1);
    {
      f2 h[3][8];
      {
        f2 Pn[3][4], Po[3][4];
#pragma unroll
        for (int i = 0; i < 12; ++i) Po[i / 4][i % 4] = sm.pold[i][tid];
        plane_transform(sm.node[b1], Pn);
#pragma unroll
        for (int i = 0; i < 12; ++i) sm.pold[i][tid] = Pn[i / 4][i % 4];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            h[c][b] = f2_add(Pn[c][b], Po[c][b]);
            h[c][b + 4] = f2_sub(Pn[c][b], Po[c][b]);
          }
      }
      f2 t[21];
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        t[4 * i] = f2_pack(qa[i].x, qb[i].x);
        if (i < 5) {
          t[4 * i + 1] = f2_pack(qa[i].y, qb[i].y);
          t[4 * i + 2] = f2_pack(qa[i].z, qb[i].z);
          t[4 * i + 3] = f2_pack(qa[i].w, qb[i].w);
        }
      }
      f2 f[3][8];
      element_modal_f2(t, h, f, w1, w2, w3);
      if (k < z0) w1 = w2 = w3 = 0;  // the redundant plane below the tile: its elements are another tile's
      f2 cy[12];
#pragma unroll
      for (int i = 0; i < 12; ++i) cy[i] = sm.carry[i][tid];
      float top_r[6];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        f2 lo[4];
        lo[0] = f2_sub(cy[4 * c], f[c][4]);
#pragma unroll
        for (int b = 1; b < 4; ++b) lo[b] = f2_add(f2_sub(f[c][b], f[c][b + 4]), cy[4 * c + b]);
        const f2 p0 = f2_sub(lo[0], lo[2]), p1 = f2_add(lo[0], lo[2]);
        const f2 q0 = f2_sub(lo[1], lo[3]), q1 = f2_add(lo[1], lo[3]);
        const f2 r0 = f2_sub(p0, q0), r1 = f2_add(p0, q0), r2 = f2_sub(p1, q1), r3 = f2_add(p1, q1);
        e_a[c] = f2_lo(r0);
        g_a[c] = f2_lo(r1);
        e_b[c] = act_b ? f2_hi(r0) + f2_lo(r2) : f2_lo(r2);
        g_b[c] = act_b ? f2_hi(r1) + f2_lo(r3) : f2_lo(r3);
        top_r[c] = act_b ? f2_hi(r2) : 0.f;
        top_r[3 + c] = act_b ? f2_hi(r3) : 0.f;
        cy[4 * c] = f[c][4];
#pragma unroll
        for (int b = 1; b < 4; ++b) cy[4 * c + b] = f2_add(f[c][b], f[c][b + 4]);
      }
#pragma unroll
      for (int i = 0; i < 12; ++i) sm.carry[i][tid] = cy[i];
#pragma unroll
      for (int i = 0; i < 6; ++i) sm.r[k & 1][i][tid] = top_r[i];
    }
    tile_sync<GROUPED>();
    pa = na;
    pb = nb;
    b0 = b1;
  }
  node_sums(zend - 1);
  const float ea = f2_lo(w1) + 3.f * f2_lo(w2) + 9.f * f2_lo(w3), eb = f2_hi(w1) + 3.f * f2_hi(w2) + 9.f * f2_hi(w3);
  if (act_a) hAh += (double)ea;
  if (act_b) hAh += (double)eb;
}

// ---------------------------------------------------------------------------
// FP64 tile in fixed point (e3d_fixed.cuh).

// Rows of a fixed-point tile, and blocks per SM.  What bounds the tile is integer
// issue: 378 wide multiply-adds an element at two cycles of a scheduler each, which
// its other integer instructions (some 1200 a warp and plane) do not overlap, and
// the latency of their chains with two warps a scheduler.  Two blocks of 4 warps
// with 255 registers run their FP64 and load phases beside each other's products.
// FP64 iteration at 300^3 as first built: 4.67 ms; one block of 8 warps 4.89, two of
// 6 (168 registers) 5.04, one of 12 5.01, three of 4 5.08; the FP64 element form 14.5.
// Now 4.52.
constexpr int kFxRows = 4;
constexpr int kFxThreads = TILE_X * kFxRows;
constexpr int kFxBlocks = 2;

struct FxArgs {
  const int4* __restrict__ tab;  // kFxStride int4 per phase
  int kc;                        // table exponent
  unsigned* mx;                  // fused: row maxima of h_new, written here
};

template <bool FUSED>
struct FxSmem {
  static constexpr int kHalo = TILE_X + kFxRows + 1;
  long long node[3][3][(TILE_X + 1) * (kFxRows + 1)];  // plane k in one of three
  long long r[2][9][kFxThreads];                       // by plane parity
  // forces on the nodes past the tile's high edges (y row 0..31, x column
  // 32.., corner last) by plane parity, and those nodes' values, plane k in k % 4
  long long edge[2][3][kHalo];
  long long edge_x[FUSED ? 4 : 1][3][kHalo];
  // a thread's own slots: upper-plane forces of its last element, raw values of
  // one plane in flight (x, then z; own node, halo node)
  long long carry[12][kFxThreads];
  double raw[FUSED ? 6 : 3][kFxThreads + kHalo];
};

// Larger of the two, or a NaN where either is one: in a reduction, which meets its
// values in any order, a NaN must reach the result.
__host__ __device__ __forceinline__ double fx_max(double a, double b) { return a != a || b <= a ? a : b; }
__device__ __forceinline__ unsigned abs_hi(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }

constexpr int kFxGeneral = 0x7fffffff;

// Exponent kx with 2^kx * b < 2^kFxNodeBits (b >= 0), or kFxGeneral where that
// leaves the range of exponent arithmetic.
__device__ __forceinline__ int fx_exponent_below(double b) {
  if (b == 0.0) return 0;
  const int e = __double2hiint(b) >> 20;  // b < 2^(e - 1022)
  if (e < 1023 - 400 || e > 1023 + 400) return kFxGeneral;
  return kFxNodeBits - (e - 1022);
}
// The same for values whose high words are at most hi.
__device__ __forceinline__ int fx_exponent(unsigned hi) {
  if (hi >= 0x7ff00000u) return kFxGeneral;
  return fx_exponent_below(hi ? __hiloint2double((int)hi + 1, 0) : 0.0);
}

// How much smaller than the largest value that a tile reads its parts may be, in
// powers of two.  A tile's values share one exponent, so that a part 2^s smaller is
// held to 2^-(56 - s) of itself.  Error of K.x there over that of the FP64 form,
// measured with s from the typical size to the peak: 0.6 at s = 2, 1 at 4, 7 at 7, 57
// at 10 (1.6e-15 of the part's own size).  Random vectors, the directions of a
// solve from its third to twelfth iteration on and displacements stay within these; a few
// entries far above the rest, a direction that has not reached all of the grid
// yet, and a rigid offset of one component do not: such a tile takes the FP64 form.
constexpr unsigned kFxRow = 5;         // a row of the tile over all its planes
constexpr unsigned kFxSegment = 8;     // a row of one plane (stand-alone pass only)
constexpr unsigned kFxComponent = 10;  // one component of a row (stand-alone pass only)

// What fx_tile_exponent asks of the rows of a tile, per row of 32 nodes over all
// planes, words tile * kFxRows + row: m, the largest |value| as the high word of the
// double; lim, the largest exponent that the tile's scale may have by the
// limits above.
struct FxRowMax {
  const unsigned* m;
  const unsigned* lim;
};
// The same of h_new = z + gamma h_old before it is formed: the largest |h_old| (null: a
// reset) and |z| (two words a row, tile * 2 * kFxRows + row and + kFxRows).
struct FxRowMaxFused {
  const unsigned* h;
  const unsigned* z;
  double gamma;
};

// Exponent kx of a tile: 2^kx * |value| < 2^kFxNodeBits for every node that the tile
// reads: its own rows, those of the next tile in x, the first of the next in y, and
// of all these the planes above and below.  kFxGeneral where a value is not finite,
// the exponent leaves the range of exponent arithmetic or the values are uneven.
// Every warp finds it by itself, a row a lane.
template <typename Rows>
static __device__ __forceinline__ int fx_tile_exponent(const GridDims& G, long long tile, const Rows& R) {
  const int lane = threadIdx.x & 31;
  unsigned w = 0, limit = 0xffffffffu;  // bound of the row's values, and the largest exponent it allows
  if (lane < 30) {
    const int row = lane % 5, nb = lane / 5;
    const int tix = (int)(tile % G.ntx), tiy = (int)((tile / G.ntx) % G.nty),
              tiz = (int)(tile / ((long long)G.ntx * G.nty));
    const int ax = wrapi(tix + nb / 3, G.ntx), ay = wrapi(tiy + row / 4, G.nty), az = wrapi(tiz + nb % 3 - 1, G.ntz);
    const long long t = E3D_IDX(ax + (long long)G.ntx * (ay + (long long)G.nty * az), G.ntiles);
    const int r = row % 4;
    if constexpr (std::is_same_v<Rows, FxRowMaxFused>) {
      const unsigned bx = R.h ? __ldcg(R.h + t * kFxRows + r) : 0u;
      const unsigned bz = max(__ldcg(R.z + t * 2 * kFxRows + r), __ldcg(R.z + t * 2 * kFxRows + kFxRows + r));
      const double vx = bx ? __hiloint2double((int)bx + 1, 0) : 0.0, vz = bz ? __hiloint2double((int)bz + 1, 0) : 0.0;
      w = max(bx, bz) >= 0x7ff00000u ? 0x7ff00000u : abs_hi(fma(fabs(R.gamma), vx, vz));
      if (w) limit = (w >> 20) + kFxRow;
    } else {
      w = __ldcg(R.m + t * kFxRows + r);
      limit = __ldcg(R.lim + t * kFxRows + r);
    }
  }
  static_assert(kFxRows == 4, "30 rows: a tile's, times two in x and three in z, and the next one's first");
  w = __reduce_max_sync(0xffffffffu, w);
  limit = __reduce_min_sync(0xffffffffu, limit);
  if ((w + 1) >> 20 > limit) return kFxGeneral;
  return fx_exponent(w);
}

// apply_tile<double, FUSED> with the element products in fixed point: the same
// march, halos and results; loads, h_new, the halos and K x are doubles.  One
// block barrier a plane: between two of them a block sums the nodes of one
// plane, forms the elements of the next, and converts the plane after that, so
// that its warps need not be in the same phase.  Loads are in flight one plane
// ahead without holding registers.  FP64 is left with the direction update, the
// conversions of K x and the dot product.
template <bool FUSED, bool GROUPED = false>
static __device__ __forceinline__ void apply_tile_fx(const ApplyArgs<double>& A, const FxArgs& F, int kx, long long tile,
                                                     FxSmem<FUSED>& sm, double& hAh) {
  constexpr int TILE_Y = kFxRows, NT = kFxThreads;
  const GridDims& G = A.g;
  const int tid = threadIdx.x % kFxThreads;
  const int tx = tid % TILE_X, ty = tid / TILE_X;
  const int tix = (int)(tile % G.ntx);
  const int tiy = (int)((tile / G.ntx) % G.nty);
  const int tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
  const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(G.tz, G.nz - z0);
  const bool active = (tx < wx) && (ty < wy);
  const bool xedge = active && tx == wx - 1, yedge = active && ty == wy - 1;
  const long long ns = G.ns;
  const long long nxy = (long long)G.nx * G.ny;
  const int nhalo = wx + wy + 1;
  constexpr int cst = (TILE_X + 1) * (TILE_Y + 1);
  constexpr int ed = TILE_X + TILE_Y + 1;
  int hlx = wx, hly = wy;  // halo node of loader thread tid < nhalo
  if (tid < wy)
    hly = tid;
  else if (tid < wy + wx)
    hlx = tid - wy;
  const long long own_col = (long long)(x0 + tx) + (long long)G.nx * (y0 + ty);
  const long long halo_col = (long long)wrapi(x0 + hlx, G.nx) + (long long)G.nx * wrapi(y0 + hly, G.ny);
  const int ko = 64 - kx - F.kc, ko20 = ko * (1 << 20);  // force unit 2^ko

  // One node plane's loads are in flight while the previous element computes, in
  // slots that the loading thread alone reads back: they hold no registers.
  const bool need_x = !FUSED || !A.reset;
  auto prefetch = [&](int zl) {
    const long long zo = nxy * wrapi(zl, G.nz);
    if (active) {
      const long long m = E3D_IDX(own_col + zo, ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (need_x) cp_async_8(&sm.raw[c][tid], A.x + m + c * ns);
        if (FUSED) cp_async_8(&sm.raw[FUSED ? 3 + c : c][tid], A.zv + m + c * ns);
      }
    }
    if (tid < nhalo) {
      const long long m = E3D_IDX(halo_col + zo, ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (need_x) cp_async_8(&sm.raw[c][NT + tid], A.x + m + c * ns);
        if (FUSED) cp_async_8(&sm.raw[FUSED ? 3 + c : c][NT + tid], A.zv + m + c * ns);
      }
    }
    cp_async_commit();
  };
  auto loaded = [&](int i, int c) {
    if (!FUSED) return sm.raw[c][i];
    const double z = sm.raw[FUSED ? 3 + c : c][i];
    return A.reset ? z : fma(A.gamma, sm.raw[c][i], z);
  };
  unsigned hmax = 0;
  // Plane zl's values from their slots: the node's own in X (stored to its plane
  // buffer by commit), the halo's at once.
  long long X[3];
  int nb = (z0 + 2) % 3;  // z0 - 1 mod 3
  auto convert = [&](int zl, int buf, bool own) {
    cp_async_wait<0>();
    if (active) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double v = loaded(tid, c);
        if (FUSED) {
          if (own) {
            A.hnew[E3D_IDX(own_col + nxy * zl, ns) + c * ns] = v;
            hmax = max(hmax, abs_hi(v));
          }
        }
        X[c] = fx_from_double(v, kx);
      }
    }
    if (tid < nhalo) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        sm.node[buf][c][E3D_IDX(hly * (TILE_X + 1) + hlx, cst)] = fx_from_double(loaded(NT + tid, c), kx);
    }
  };
  auto commit = [&](int buf) {
    if (active) {
#pragma unroll
      for (int c = 0; c < 3; ++c) sm.node[buf][c][ty * (TILE_X + 1) + tx] = X[c];
    }
  };
  auto plane_transform = [&](int buf, long long (&P)[3][4]) {
    const long long* b = sm.node[buf][0] + ty * (TILE_X + 1) + tx;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long v[4] = {b[c * cst], b[c * cst + 1], b[c * cst + TILE_X + 1], b[c * cst + TILE_X + 2]};
      had_xy(v, P[c]);
    }
  };
  double dot = 0.0, dot_edge = 0.0;
  // Edge forces of plane k to the halo buffers, and their share of the dot
  // product: the 3 * ed values in kFlush shares of 32, one a warp, rotating.
  auto edge_flush = [&](int k, int share) {
    const int v = share * 32 + (tid & 31);
    if (v < 3 * ed) {
      const int c = v / ed, e = v - c * ed;
      const long long hb = tile * G.tz + (k - z0);
      const long long per_c = G.ntiles * (long long)G.tz;
      double* out = nullptr;
      if (e < TILE_X) {
        if (e < wx) out = A.hy + E3D_IDX((c * per_c + hb) * TILE_X + e, 3 * per_c * TILE_X);
      } else if (e < ed - 1) {
        if (e - TILE_X < wy) out = A.hx + E3D_IDX((c * per_c + hb) * TILE_Y + (e - TILE_X), 3 * per_c * TILE_Y);
      } else {
        out = A.hd + E3D_IDX(c * per_c + hb, 3 * per_c);
      }
      if (out) {
        const double d = __ll2double_rn(sm.edge[k & 1][c][e]);
        if (FUSED) dot_edge = fma(__ll2double_rn(sm.edge_x[FUSED ? k & 3 : 0][c][e]), d, dot_edge);
        *out = fx_scale(d, ko20);
      }
    }
  };
  constexpr int kFlush = (3 * ed + 31) / 32;
  static_assert(kFlush <= kFxRows, "a share for each of some of the warps");
  long long acc0[3] = {0, 0, 0};  // own corner force of the last element
  // node sums of plane k from the forces its elements left in sm.r; buf: the
  // buffer whose own slot still holds the node's value there
  auto node_sums = [&](int k, int buf) {
    if (active) {
      const long long m = E3D_IDX(own_col + nxy * k, ns);
      const long long(*r)[NT] = sm.r[k & 1];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const long long left3 = tx > 0 ? r[3 * c + 2][tid - 1] : 0;
        const long long below3 = ty > 0 ? r[3 * c + 2][tid - TILE_X] : 0;
        long long acc = acc0[c];
        if (tx > 0) acc += r[3 * c + 0][tid - 1];
        if (ty > 0) acc += r[3 * c + 1][tid - TILE_X];
        if (tx > 0 && ty > 0) acc += r[3 * c + 2][tid - TILE_X - 1];
        const double d = __ll2double_rn(acc);
        if (FUSED) dot = fma(__ll2double_rn(sm.node[buf][c][ty * (TILE_X + 1) + tx]), d, dot);
        A.y[m + c * ns] = fx_scale(d, ko20);
        if (xedge) sm.edge[k & 1][c][TILE_X + ty] = r[3 * c + 0][tid] + below3;
        if (yedge) sm.edge[k & 1][c][tx] = r[3 * c + 1][tid] + left3;
        if (xedge && yedge) sm.edge[k & 1][c][ed - 1] = r[3 * c + 2][tid];
      }
    }
  };

  // One barrier a plane.  Between barriers k-1 and k: node sums of plane k-1,
  // the element of plane k (from plane k+1's buffer and the transform kept of
  // plane k), conversion of plane k+2 into the buffer that held plane k-1, edge
  // forces of plane k-2.
  // (set here, or the threads outside the grid would carry them from tile to tile)
  long long Pold[3][4] = {};
  auto edge_share = [&](int k) { return ((tid >> 5) + k) % kFxRows; };
  auto next = [](int b) { return b == 2 ? 0 : b + 1; };
  prefetch(z0 - 1);
  convert(z0 - 1, nb, false);
  commit(nb);
  prefetch(z0);
  const int nb1 = next(nb);
  convert(z0, nb1, true);
  commit(nb1);
  tile_sync<GROUPED>();
  if (active) plane_transform(nb, Pold);
  prefetch(z0 + 1);
  int b0 = nb;  // buffer of plane k
  int ph_cur = active ? __ldcs(A.pix + E3D_IDX(own_col + nxy * wrapi(z0 - 1, G.nz), ns)) : 0;
  for (int k = z0 - 1; k < z0 + wz; ++k) {
    const int b1 = next(b0), b2 = next(b1);  // of planes k + 1 and k + 2
    const bool more = k + 2 <= z0 + wz;
    if (more) convert(k + 2, b2, k + 2 < z0 + wz);
    if (k + 3 <= z0 + wz) prefetch(k + 3);
    const int ph_nxt = (active && k + 1 < z0 + wz) ? __ldcs(A.pix + E3D_IDX(own_col + nxy * (k + 1), ns)) : 0;
    if (k > z0) node_sums(k - 1, b2);
    if (k > z0 + 1 && edge_share(k) < kFlush) edge_flush(k - 2, edge_share(k));
    if (active) {
      long long h[3][8];
      {
        long long Pn[3][4];
        plane_transform(b1, Pn);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            h[c][b] = Pn[c][b] + Pold[c][b];
            h[c][b + 4] = Pn[c][b] - Pold[c][b];
            Pold[c][b] = Pn[c][b];
          }
      }
      long long f[3][8];
      element_modal_fx(F.tab + E3D_IDX(ph_cur, A.ncs) * kFxStride, h, f);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (k >= z0) {
          long long lo[4], rr[4];
          lo[0] = sm.carry[4 * c][tid] - f[c][4];
#pragma unroll
          for (int b = 1; b < 4; ++b) lo[b] = (f[c][b] - f[c][b + 4]) + sm.carry[4 * c + b][tid];
          had_xy_adj(lo, rr);
          acc0[c] = rr[0];
          sm.r[k & 1][3 * c + 0][tid] = rr[1];  // to node (x+1, y)
          sm.r[k & 1][3 * c + 1][tid] = rr[2];  // to node (x, y+1)
          sm.r[k & 1][3 * c + 2][tid] = rr[3];  // to node (x+1, y+1)
        }
        sm.carry[4 * c][tid] = f[c][4];
#pragma unroll
        for (int b = 1; b < 4; ++b) sm.carry[4 * c + b][tid] = f[c][b] + f[c][b + 4];
      }
      if (FUSED && k >= z0 && (xedge || yedge)) {  // plane k's values past the edges
        const long long* b = sm.node[b0][0] + ty * (TILE_X + 1) + tx;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (yedge) sm.edge_x[FUSED ? k & 3 : 0][c][tx] = b[c * cst + TILE_X + 1];
          if (xedge) sm.edge_x[FUSED ? k & 3 : 0][c][TILE_X + ty] = b[c * cst + 1];
          if (xedge && yedge) sm.edge_x[FUSED ? k & 3 : 0][c][ed - 1] = b[c * cst + TILE_X + 2];
        }
      }
    }
    if (more) commit(b2);
    tile_sync<GROUPED>();
    ph_cur = ph_nxt;
    b0 = b1;
  }
  const int kl = z0 + wz - 1;
  node_sums(kl, b0 == 0 ? 2 : b0 - 1);
  if (wz > 1 && edge_share(kl + 1) < kFlush) edge_flush(kl - 1, edge_share(kl + 1));
  tile_sync<GROUPED>();
  if (edge_share(kl + 2) < kFlush) edge_flush(kl, edge_share(kl + 2));
  if (FUSED) {
    hmax = __reduce_max_sync(0xffffffffu, hmax);
    if ((tid & 31) == 0) F.mx[E3D_IDX(tile * kFxRows + ty, G.ntiles * kFxRows)] = hmax;
    // ldexp, not exponent arithmetic: the sums may be zero or span any range
    hAh += ldexp(dot + dot_edge, ko - kx);
  }
}

// A tile that the fixed-point form does not take: the FP64 form, out of line.
template <bool GROUPED>
static __device__ __noinline__ void apply_tile_general(const ApplyArgs<double>& A, long long tile,
                                                       ApplySmem<double, kFxRows>& sm) {
  double dot = 0.0;
  apply_tile<double, false, false, false, kFxRows, GROUPED>(A, tile, sm, dot);
}

// Shared memory of apply_tile_ring: the in-plane force exchange of the ZS
// planes of a step, double-buffered by step parity so one barrier per step
// suffices.
template <int ZS>
struct RingApplySmem {
  float r[2][9 * ZS][NT];
};

// The fused FP32 tile fed by the plane ring (TMA).  Same element arithmetic,
// values and summation order as apply_tile<float, true>, but every thread reads
// its element's four corners of the next plane straight from the ring stage
// (main box, or the +x column / +y row / corner box at the tile edge) and forms
// h_new = z + gamma*h_old there, so no node buffer and no copy barrier are
// needed.  A step computes ZS consecutive elements of the thread's column
// (ZS = 2: two independent element computations between barriers, the shared
// middle plane transformed once); with the force exchange double-buffered one
// __syncthreads per step orders the steps, and the step's oldest stages are
// refilled right after it.  At a step for element planes k .. k+ZS-1 the ring
// holds plane k at R.q.
template <int ZS>
static __device__ void apply_tile_ring(const ApplyArgs<float>& A, long long tile, RingApplySmem<ZS>& sm, double& hAh,
                                       PlaneRing& R) {
  const GridDims& G = A.g;
  const int tid = threadIdx.x;
  const int tx = tid % TILE_X, ty = tid / TILE_X;
  const int tix = (int)(tile % G.ntx);
  const int tiy = (int)((tile / G.ntx) % G.nty);
  const int tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
  const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(G.tz, G.nz - z0);
  const bool active = (tx < wx) && (ty < wy);
  const long long ns = G.ns;
  const long long nxy = (long long)G.nx * G.ny;
  const long long ncol = (long long)(x0 + tx) + (long long)G.nx * (y0 + ty);
  // stage offset (floats within one vector) and component stride of corner d
  // = dx + 2*dy of this thread's element
  auto corner_at = [&](int d, int& off, int& str) {
    const int lx = tx + (d & 1), ly = ty + (d >> 1);
    if (lx < wx) {
      if (ly < wy) {
        off = ly * TILE_X + lx;
        str = NT;
      } else {
        off = (kRingMain + kRingCol) / 4 + lx;
        str = TILE_X;
      }
    } else {
      if (ly < wy) {
        off = kRingMain / 4 + ly * 4;
        str = TILE_X;
      } else {
        off = (kRingMain + kRingCol + kRingRow) / 4;
        str = 4;
      }
    }
  };
  auto hval = [&](const unsigned char* st, int off) -> float {
    const float x = reinterpret_cast<const float*>(st)[E3D_IDX(off, kRingVec / 4)];
    const float z = reinterpret_cast<const float*>(st + kRingVec)[E3D_IDX(off, kRingVec / 4)];
    return A.reset ? z : fmaf(A.gamma, x, z);
  };
  auto corners = [&](const unsigned char* st, float (&v)[3][4]) {
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      int off, str;
      corner_at(d, off, str);
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c][d] = hval(st, off + c * str);
    }
  };
  auto phase_of = [&](const unsigned char* st) { return reinterpret_cast<const int*>(st + 2 * kRingVec)[tid]; };

  float Pold[3][4], carry[3][4];
  float dot32 = 0.f;
  int ph_cur = 0;
  {
    const unsigned char* st = ring_wait(R, R.q);  // plane z0-1
    if (active) {
      float v0[3][4];
      corners(st, v0);
#pragma unroll
      for (int c = 0; c < 3; ++c) had_xy(v0[c], Pold[c]);
      ph_cur = phase_of(st);
    }
  }
  const int hstride = G.tz;
  int step = 0;
  for (int k = z0 - 1; k < z0 + wz; k += ZS, ++step) {
    const int ne = min(ZS, z0 + wz - k);  // elements k .. k+ne-1 in this step
    float rr[ZS][3][4];
    float hk[ZS][3][4];
#pragma unroll
    for (int j = 0; j < ZS; ++j) {
      if (j < ne) {
        const int kk = k + j;
        const unsigned char* st1 = ring_wait(R, R.q + 1 + j);  // plane kk+1
        int ph_nxt = 0;
        if (active) {
          float nxt[3][4];
          corners(st1, nxt);
          if (kk + 1 >= z0 && kk + 1 < z0 + wz) {
            const long long m = E3D_IDX(ncol + nxy * (kk + 1), ns);
#pragma unroll
            for (int c = 0; c < 3; ++c) A.hnew[m + c * ns] = nxt[c][0];
          }
          ph_nxt = phase_of(st1);
          float Pn[3][4], h[3][8];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            had_xy(nxt[c], Pn[c]);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              h[c][b] = Pn[c][b] + Pold[c][b];
              h[c][b + 4] = Pn[c][b] - Pold[c][b];
            }
          }
          float f[3][8];
          element_modal_f32(A.cs + E3D_IDX(ph_cur, A.ncs) * kCs32Stride, h[0], h[1], h[2], f[0], f[1], f[2]);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            float lo[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              lo[b] = f[c][b] - f[c][b + 4];
              const float hi = f[c][b] + f[c][b + 4];
              if (kk >= z0) lo[b] += carry[c][b];
              carry[c][b] = hi;
            }
            if (kk >= z0) had_xy_adj(lo, rr[j][c]);
#pragma unroll
            for (int b = 0; b < 4; ++b) Pold[c][b] = Pn[c][b];
          }
        }
        // plane kk's h_new for the dot products, read before the barrier (the
        // stage is refilled after it)
        if (kk >= z0 && active) {
          const unsigned char* st0 = ring_stage(R, R.q + j);
#pragma unroll
          for (int d = 0; d < 4; ++d) {
            const bool need = d == 0 || (d == 1 && tx == wx - 1) || (d == 2 && ty == wy - 1) ||
                              (d == 3 && tx == wx - 1 && ty == wy - 1);
            int off, str;
            corner_at(d, off, str);
#pragma unroll
            for (int c = 0; c < 3; ++c) hk[j][c][d] = need ? hval(st0, off + c * str) : 0.f;
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            sm.r[step & 1][9 * j + 3 * c + 0][tid] = rr[j][c][1];  // to node (x+1, y)
            sm.r[step & 1][9 * j + 3 * c + 1][tid] = rr[j][c][2];  // to node (x, y+1)
            sm.r[step & 1][9 * j + 3 * c + 2][tid] = rr[j][c][3];  // to node (x+1, y+1)
          }
        }
        ph_cur = ph_nxt;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ZS; ++j)
      if (j < ne) ring_release(R, G);  // planes k .. k+ne-1
#pragma unroll
    for (int j = 0; j < ZS; ++j) {
      const int kk = k + j;
      if (j < ne && kk >= z0 && active) {
        const float(*r)[NT] = sm.r[step & 1] + 9 * j;
        const int lz = kk - z0;
        const long long m = E3D_IDX(ncol + nxy * kk, ns);
        float hxv[3], hyv[3], acc[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[c] = rr[j][c][0];
          if (tx > 0) acc[c] += r[3 * c + 0][tid - 1];
          if (ty > 0) acc[c] += r[3 * c + 1][tid - TILE_X];
          if (tx > 0 && ty > 0) acc[c] += r[3 * c + 2][tid - TILE_X - 1];
          A.y[m + c * ns] = acc[c];
          hxv[c] = rr[j][c][1] + (ty > 0 ? r[3 * c + 2][tid - TILE_X] : 0.f);
          hyv[c] = rr[j][c][2] + (tx > 0 ? r[3 * c + 2][tid - 1] : 0.f);
        }
        dot32 += hk[j][0][0] * acc[0] + hk[j][1][0] * acc[1] + hk[j][2][0] * acc[2];
        const long long hb = tile * hstride + lz;
        if (tx == wx - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hx[E3D_IDX(((long long)c * G.ntiles * hstride + hb) * TILE_Y + ty, halo_len(G, TILE_Y))] = hxv[c];
          dot32 += hk[j][0][1] * hxv[0] + hk[j][1][1] * hxv[1] + hk[j][2][1] * hxv[2];
        }
        if (ty == wy - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hy[E3D_IDX(((long long)c * G.ntiles * hstride + hb) * TILE_X + tx, halo_len(G, TILE_X))] = hyv[c];
          dot32 += hk[j][0][2] * hyv[0] + hk[j][1][2] * hyv[1] + hk[j][2][2] * hyv[2];
        }
        if (tx == wx - 1 && ty == wy - 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.hd[E3D_IDX((long long)c * G.ntiles * hstride + hb, halo_len(G, 1))] = rr[j][c][3];
          dot32 += hk[j][0][3] * rr[j][0][3] + hk[j][1][3] * rr[j][1][3] + hk[j][2][3] * rr[j][2][3];
        }
      }
    }
  }
  ring_release(R, G);  // plane z0+wz, last read before the final step's barrier
  hAh += (double)dot32;
}

// Halo contribution for node (x, y, z) from the neighbouring tiles.
template <typename T, int TY = TILE_Y>
__device__ __forceinline__ void halo_add(const GridDims& G, const T* __restrict__ hx,
                                         const T* __restrict__ hy, const T* __restrict__ hd,
                                         int x, int y, int z, T (&v)[3]) {
  constexpr int TILE_Y = TY;
  const int tix = x / TILE_X, lx = x - tix * TILE_X;
  const int tiy = y / TILE_Y, ly = y - tiy * TILE_Y;
  const int tiz = z / G.tz, lz = z - tiz * G.tz;
  if (lx != 0 && ly != 0) return;
  const int txl = tix == 0 ? G.ntx - 1 : tix - 1;
  const int tyd = tiy == 0 ? G.nty - 1 : tiy - 1;
  const long long plane = (long long)tiz * G.nty;
  const long long per_c = G.ntiles * G.tz;
  if (lx == 0) {
    const long long t = (long long)txl + (long long)G.ntx * (tiy + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hx + E3D_IDX((c * per_c + t * G.tz + lz) * TILE_Y + ly, 3 * per_c * TILE_Y));
  }
  if (ly == 0) {
    const long long t = (long long)tix + (long long)G.ntx * (tyd + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hy + E3D_IDX((c * per_c + t * G.tz + lz) * TILE_X + lx, 3 * per_c * TILE_X));
  }
  if (lx == 0 && ly == 0) {
    const long long t = (long long)txl + (long long)G.ntx * (tyd + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hd + E3D_IDX(c * per_c + t * G.tz + lz, 3 * per_c));
  }
}

// halo_add for a node whose tile coordinates are known (no integer division);
// same additions in the same order.
template <typename T, int TY = TILE_Y>
__device__ __forceinline__ void halo_add_tile(const GridDims& G, const T* __restrict__ hx,
                                              const T* __restrict__ hy, const T* __restrict__ hd,
                                              int tix, int tiy, int tiz, int lx, int ly, int lz, T (&v)[3]) {
  constexpr int TILE_Y = TY;
  if (lx != 0 && ly != 0) return;
  const int txl = tix == 0 ? G.ntx - 1 : tix - 1;
  const int tyd = tiy == 0 ? G.nty - 1 : tiy - 1;
  const long long plane = (long long)tiz * G.nty;
  const long long per_c = G.ntiles * G.tz;
  if (lx == 0) {
    const long long t = (long long)txl + (long long)G.ntx * (tiy + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hx + E3D_IDX((c * per_c + t * G.tz + lz) * TILE_Y + ly, 3 * per_c * TILE_Y));
  }
  if (ly == 0) {
    const long long t = (long long)tix + (long long)G.ntx * (tyd + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hy + E3D_IDX((c * per_c + t * G.tz + lz) * TILE_X + lx, 3 * per_c * TILE_X));
  }
  if (lx == 0 && ly == 0) {
    const long long t = (long long)txl + (long long)G.ntx * (tyd + plane);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] += __ldcg(hd + E3D_IDX(c * per_c + t * G.tz + lz, 3 * per_c));
  }
}

// ---------------------------------------------------------------------------
// Stand-alone apply: one tile per block, then apply_finish adds the halos.
template <typename T>
__global__ void __launch_bounds__(NT, 1) apply_tiles_kernel(ApplyArgs<T> A, double* partial) {
  __shared__ ApplySmem<T> sm;
  __shared__ double red[NT / 32];
  double hAh = 0.0;
  apply_tile<T, false>(A, blockIdx.x, sm, hAh);
  const double s = block_sum<NT>(hAh, red);
  if (partial && threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Bound of |v| as FxRowMax keeps it: zero for zero alone.
__device__ __forceinline__ unsigned size_word(double v) { return abs_hi(v) | (__double2loint(v) != 0 ? 1u : 0u); }

// Row maxima of a warp's row of nodes, plane by plane (FxRowMax); all lanes take part.
struct FxRowScan {
  unsigned comp[3] = {0, 0, 0}, segment = 0xffffffffu;
  __device__ __forceinline__ void plane(unsigned a, unsigned b, unsigned c) {
    comp[0] = max(comp[0], a);
    comp[1] = max(comp[1], b);
    comp[2] = max(comp[2], c);
    const unsigned seg = __reduce_max_sync(0xffffffffu, max(a, max(b, c)));
    if (seg) segment = min(segment, seg);
  }
  // The row's words, the same in every lane.
  __device__ __forceinline__ void finish(unsigned& m, unsigned& lim) {
    m = 0;
    lim = segment == 0xffffffffu ? segment : (segment >> 20) + kFxSegment;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const unsigned v = __reduce_max_sync(0xffffffffu, comp[c]);
      m = max(m, v);
      if (v) lim = min(lim, (v >> 20) + kFxComponent);
    }
    if (m) lim = min(lim, (m >> 20) + kFxRow);
  }
};

// Row maxima of a tile of a nodal vector, one block a tile: the largest |value|
// alone, for a solve's own vectors.
__device__ __forceinline__ unsigned tile_row_max(const GridDims& G, long long tile, const double* x, int from = 0,
                                                 int planes = 0x7fffffff) {
  const int tx = threadIdx.x % TILE_X, ty = threadIdx.x / TILE_X;
  const int tix = (int)(tile % G.ntx), tiy = (int)((tile / G.ntx) % G.nty),
            tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int xg = tix * TILE_X + tx, yg = tiy * kFxRows + ty, z0 = tiz * G.tz + from;
  const int z1 = min(G.nz, z0 + min(planes, G.tz - from));
  unsigned v = 0;
  if (xg < G.nx && yg < G.ny) {
    const long long nxy = (long long)G.nx * G.ny;
    const double* col = x + E3D_IDX(xg + (long long)G.nx * yg + nxy * z0, G.ns);
#pragma unroll 4
    for (int z = z0; z < z1; ++z, col += nxy) {
      const unsigned a = abs_hi(__ldcg(col)), b = abs_hi(__ldcg(col + G.ns)), c = abs_hi(__ldcg(col + 2 * G.ns));
      v = max(v, max(a, max(b, c)));
    }
  }
  return __reduce_max_sync(0xffffffffu, v);
}

static __global__ void __launch_bounds__(kFxThreads) tile_max_kernel(GridDims G, const double* __restrict__ x,
                                                                     unsigned* __restrict__ m, unsigned* __restrict__ lim) {
  const long long tile = blockIdx.x;
  const int tx = threadIdx.x % TILE_X, ty = threadIdx.x / TILE_X;
  const int tix = (int)(tile % G.ntx), tiy = (int)((tile / G.ntx) % G.nty),
            tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int xg = tix * TILE_X + tx, yg = tiy * kFxRows + ty, z0 = tiz * G.tz, z1 = min(G.nz, z0 + G.tz);
  const bool active = xg < G.nx && yg < G.ny;
  const long long nxy = (long long)G.nx * G.ny;
  const double* col = x + E3D_IDX(active ? xg + (long long)G.nx * yg + nxy * z0 : 0, G.ns);
  FxRowScan scan;
  constexpr int kAhead = 4;  // planes loaded before the first is scanned: the scan holds loads behind it back
  for (int z = z0; z < z1; z += kAhead) {
    double v[kAhead][3];
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[j][c] = active && z + j < z1 ? __ldcg(col + j * nxy + c * G.ns) : 0.0;
    col += kAhead * nxy;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) scan.plane(size_word(v[j][0]), size_word(v[j][1]), size_word(v[j][2]));
  }
  unsigned vm, vl;
  scan.finish(vm, vl);
  if (tx == 0) {
    m[E3D_IDX(tile * kFxRows + ty, G.ntiles * kFxRows)] = vm;
    lim[E3D_IDX(tile * kFxRows + ty, G.ntiles * kFxRows)] = vl;
  }
}

// The stand-alone FP64 apply in fixed point, one tile a block; R: of A.x.
static __global__ void __launch_bounds__(kFxThreads, kFxBlocks) apply_tiles_fx_kernel(ApplyArgs<double> A, FxArgs F,
                                                                                      FxRowMax R) {
  extern __shared__ __align__(128) unsigned char e3d_fx_dyn[];  // sizeof(FxSmem<false>)
  FxSmem<false>& sm = *reinterpret_cast<FxSmem<false>*>(e3d_fx_dyn);
  static_assert(sizeof(ApplySmem<double, kFxRows>) <= sizeof(FxSmem<false>), "the FP64 form shares the memory");
  __shared__ ApplyArgs<double> sA;
  double dummy = 0.0;
  const int kx = fx_tile_exponent(A.g, blockIdx.x, R);
  if (kx != kFxGeneral) {
    apply_tile_fx<false>(A, F, kx, blockIdx.x, sm, dummy);
  } else {
    if (threadIdx.x == 0) sA = A;
    __syncthreads();
    apply_tile_general<false>(sA, blockIdx.x, *reinterpret_cast<ApplySmem<double, kFxRows>*>(e3d_fx_dyn));
  }
}

template <typename T, int TY = TILE_Y>
__global__ void apply_finish_kernel(GridDims G, const T* __restrict__ yin, const T* __restrict__ hx,
                                    const T* __restrict__ hy, const T* __restrict__ hd,
                                    T* __restrict__ yout) {
  const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= G.ns) return;
  int x, y, z;
  node_xyz(G, m, x, y, z);
  T v[3] = {yin[m], yin[m + G.ns], yin[m + 2 * G.ns]};
  halo_add<T, TY>(G, hx, hy, hd, x, y, z, v);
  yout[m] = v[0];
  yout[m + G.ns] = v[1];
  yout[m + 2 * G.ns] = v[2];
}

// energy_OpenMP tail (src/elas3dxtal_pcg.f90:1332-1340): g = Ku + b,
// partial sums of (u.Ku/2 + b.u) and of g.g (gg0, :452).
template <int TY>
static __global__ void __launch_bounds__(256) energy_finish_kernel(GridDims G, const double* __restrict__ ku,
                                                            const double* __restrict__ hx,
                                                            const double* __restrict__ hy,
                                                            const double* __restrict__ hd,
                                                            const double* __restrict__ u,
                                                            const double* __restrict__ b,
                                                            double* __restrict__ g, double* partial) {
  __shared__ double red[8];
  double eu = 0.0, gg = 0.0;
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < G.ns;
       m += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    node_xyz(G, m, x, y, z);
    double v[3] = {ku[m], ku[m + G.ns], ku[m + 2 * G.ns]};
    halo_add<double, TY>(G, hx, hy, hd, x, y, z, v);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long i = m + c * G.ns;
      eu += 0.5 * u[i] * v[c] + b[i] * u[i];
      const double gv = v[c] + b[i];
      g[i] = gv;
      gg += gv * gv;
    }
  }
  const double s1 = block_sum<256>(eu, red);
  const double s2 = block_sum<256>(gg, red);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = s1;
    partial[2 * blockIdx.x + 1] = s2;
  }
}

// Sums n partials of stride `stride` in a fixed order (single block).
static __global__ void reduce_partials_kernel(const double* __restrict__ partial, int n, int stride,
                                       int nfields, double* __restrict__ out) {
  __shared__ double red[8];
  for (int f = 0; f < nfields; ++f) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[(long long)i * stride + f];
    const double t = block_sum<256>(s, red);
    if (threadIdx.x == 0) out[f] = t;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// femat.  One block of 32 threads per phase.
struct FematParams {
  int nphase, flag_m;
  double c11, c12, c44, K1, G1, Km, Gm;
};

// rotatestiffnessby (src/elas3dxtal_pcg.f90:2535-2633) for one grain: the Bond matrix.
static __device__ void bond_matrix(const double (&r)[3], double (&N)[6][6]) {
  const double rdotr = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
  const double term1 = 1.0 - rdotr;
  double term2 = 1.0 + rdotr;
  double Q[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) Q[i][j] = (i == j ? term1 : 0.0) + 2.0 * r[i] * r[j];
  Q[0][1] -= 2.0 * r[2];
  Q[0][2] += 2.0 * r[1];
  Q[1][2] -= 2.0 * r[0];
  Q[1][0] += 2.0 * r[2];
  Q[2][0] -= 2.0 * r[1];
  Q[2][1] += 2.0 * r[0];
  if (term2 > 1.0e-12) {
    term2 = 1.0 / term2;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) Q[i][j] *= term2;
  } else {
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) Q[i][j] = (i == j) ? 1.0 : 0.0;
  }
  for (int row = 0; row < 3; ++row) {
    N[row][0] = Q[row][0] * Q[row][0];
    N[row][1] = Q[row][1] * Q[row][1];
    N[row][2] = Q[row][2] * Q[row][2];
    N[row][3] = Q[row][1] * Q[row][2];
    N[row][4] = Q[row][2] * Q[row][0];
    N[row][5] = Q[row][0] * Q[row][1];
  }
  N[3][0] = 2.0 * Q[2][0] * Q[0][0];
  N[3][1] = 2.0 * Q[2][1] * Q[0][1];
  N[3][2] = 2.0 * Q[2][2] * Q[0][2];
  N[3][3] = Q[0][1] * Q[2][2] + Q[0][2] * Q[2][1];
  N[3][4] = Q[0][2] * Q[2][0] + Q[0][0] * Q[2][2];
  N[3][5] = Q[0][0] * Q[2][1] + Q[0][1] * Q[2][0];
  N[4][0] = 2.0 * Q[1][0] * Q[2][0];
  N[4][1] = 2.0 * Q[1][1] * Q[2][1];
  N[4][2] = 2.0 * Q[1][2] * Q[2][2];
  N[4][3] = Q[1][1] * Q[2][2] + Q[1][2] * Q[2][1];
  N[4][4] = Q[1][0] * Q[2][2] + Q[1][2] * Q[2][0];
  N[4][5] = Q[1][1] * Q[2][0] + Q[1][0] * Q[2][1];
  N[5][0] = 2.0 * Q[0][0] * Q[1][0];
  N[5][1] = 2.0 * Q[0][1] * Q[1][1];
  N[5][2] = 2.0 * Q[0][2] * Q[1][2];
  N[5][3] = Q[0][1] * Q[1][2] + Q[0][2] * Q[1][1];
  N[5][4] = Q[0][2] * Q[1][0] + Q[0][0] * Q[1][2];
  N[5][5] = Q[0][0] * Q[1][1] + Q[0][1] * Q[1][0];
}

// N^T C N for the cubic C, by the 32 threads of a warp, an entry of the 6 x 6 products
// each; every array is in shared memory.  A lane's FP64 instructions cost as much as
// a warp's: with one thread at work here and in modal_table_warp (72 divisions) the
// tables of seven phases took 97 us, so 31; those of 300^3's phases 331, so 89.
static __device__ void bond_rotate_warp(const double (&r)[3], double c11, double c12, double c44, double (&N)[6][6],
                                        double (&Tm)[6][6], double (&out)[6][6]) {
  const int lane = threadIdx.x;
  if (lane == 0) bond_matrix(r, N);
  __syncwarp();
  for (int e = lane; e < 36; e += 32) {
    const int i = e / 6, j = e % 6;
    double s = 0.0;
    for (int k = 0; k < 6; ++k) s += N[k][i] * (k < 3 && j < 3 ? (k == j ? c11 : c12) : k == j ? c44 : 0.0);
    Tm[i][j] = s;
  }
  __syncwarp();
  for (int e = lane; e < 36; e += 32) {
    const int i = e / 6, j = e % 6;
    double s = 0.0;
    for (int k = 0; k < 6; ++k) s += Tm[i][k] * N[k][j];
    out[i][j] = s;
  }
  __syncwarp();
}

// modal_table by the threads of a warp; C1 and C2: scratch, in shared memory as the rest.
static __device__ void modal_table_warp(const double (&C6)[6][6], double* tab, double (&C1)[6][6], double (&C2)[6][6]) {
  const int lane = threadIdx.x;
  for (int e = lane; e < 36; e += 32) {
    const double v = C6[e / 6][e % 6];
    tab[e] = v / 16.0;
    C1[e / 6][e % 6] = v / 48.0;
    C2[e / 6][e % 6] = v / 144.0;
  }
  __syncwarp();
  if (lane < 9) {  // column of M2: the response to a unit component
    double in[9], out[9];
    for (int r = 0; r < 9; ++r) in[r] = r == lane ? 1.0 : 0.0;
    second_order_modes(&C1[0][0], in, out);
    for (int r = 0; r < 9; ++r) tab[kM2 + 9 * r + lane] = out[r];
  } else if (lane < 12) {
    double in[3], out[3];
    for (int r = 0; r < 3; ++r) in[r] = r == lane - 9 ? 1.0 : 0.0;
    third_order_modes(&C2[0][0], in, out);
    for (int r = 0; r < 3; ++r) tab[kM3 + 3 * r + lane - 9] = out[r];
  }
  __syncwarp();
}

// K ck + G cmu of an isotropic phase (src/elas3dxtal_pcg.f90:655-664, 680-682, 701-705).
static __device__ void isotropic_warp(double K, double G, double (&C6)[6][6]) {
  for (int e = threadIdx.x; e < 36; e += 32) {
    const int i = e / 6, j = e % 6;
    const double ck = (i < 3 && j < 3) ? 1.0 : 0.0;
    double cmu = 0.0;
    if (i < 3 && j < 3) cmu = (i == j) ? 4.0 / 3.0 : -2.0 / 3.0;
    if (i >= 3 && i == j) cmu = 1.0;
    C6[i][j] = K * ck + G * cmu;
  }
  __syncwarp();
}

// Phase ids from device memory: 1-based with the range check of ppixel_hdf5
// (src/elas3dxtal_pcg.f90:2986-2989) -> 0-based; flags DEV_BAD_INDEX.
static __global__ void pix_from_device_kernel(long long ns, const int32_t* __restrict__ in, int nphase,
                                              int32_t* __restrict__ out, int* err) {
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < ns; m += (long long)gridDim.x * blockDim.x) {
    const int32_t v = in[m];
    if (v < 1 || v > nphase) {
      atomicExch(err, DEV_BAD_INDEX);
      out[m] = 0;
    } else {
      out[m] = v - 1;
    }
  }
}

// The same check and conversion in place: the 1-based ids were copied into
// the phase map as they came from the host (err may be null when the host has
// checked the ids already).
static __global__ void pix_to_zero_based_kernel(long long ns, int nphase, int32_t* pix, int* err) {
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < ns; m += (long long)gridDim.x * blockDim.x) {
    const int32_t v = pix[m];
    if (v < 1 || v > nphase) {
      if (err) atomicExch(err, DEV_BAD_INDEX);
      pix[m] = 0;
    } else {
      pix[m] = v - 1;
    }
  }
}

// Reference local node r (1..8 -> 0..7) to corner index a = ox + 2oy + 4oz.
static __constant__ int kRefToCorner[8] = {0, 1, 3, 2, 4, 5, 7, 6};

// Norms of a phase (see fx_info) from its element matrix in shared memory, one warp.
static __device__ __forceinline__ void fx_store_norms(const double (&col)[24][24], const double* csh, double* out) {
  const int lane = threadIdx.x;
  double d = 0.0, rows = 0.0, entry = 0.0;
  if (lane < 24)
    for (int c = 0; c < 24; ++c) d += fabs(lane <= c ? col[c][lane] : col[lane][c]);
  if (lane < 18) {
    const int n = lane < 6 ? 6 : lane < 15 ? 9 : 3, r = lane < 6 ? lane : lane < 15 ? lane - 6 : lane - 15;
    const double* m = csh + (lane < 6 ? 0 : lane < 15 ? kM2 : kM3) + n * r;
    for (int c = 0; c < n; ++c) {
      rows += fabs(m[c]);
      entry = fx_max(entry, fabs(m[c]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d = fx_max(d, __shfl_xor_sync(0xffffffffu, d, o));
    rows = fx_max(rows, __shfl_xor_sync(0xffffffffu, rows, o));
    entry = fx_max(entry, __shfl_xor_sync(0xffffffffu, entry, o));
  }
  if (lane == 0) {
    out[0] = d;
    out[1] = rows;
    out[2] = entry;
  }
}

// invert3x3 (src/elas3dxtal_pcg.f90:2046-2147) of a symmetric block: a and ai hold
// 00 11 22 01 02 12.  Same products as there; the cofactors that symmetry makes
// equal are formed once.
__device__ __forceinline__ void invert3x3(const double (&a)[6], double (&ai)[6]) {
  const double c00 = a[1] * a[2] - a[5] * a[5];
  const double c01 = -a[3] * a[2] + a[5] * a[4];
  const double c02 = a[3] * a[5] - a[1] * a[4];
  const double det = a[0] * c00 + a[3] * c01 + a[4] * c02;
  if (fabs(det) < 1e-14) {
    for (int i = 0; i < 6; ++i) ai[i] = 0.0;
    return;
  }
  const double inv_det = 1.0 / det;
  ai[0] = c00 * inv_det;
  ai[1] = (a[0] * a[2] - a[4] * a[4]) * inv_det;
  ai[2] = (a[0] * a[1] - a[3] * a[3]) * inv_det;
  ai[3] = c01 * inv_det;
  ai[4] = c02 * inv_det;
  ai[5] = (-a[0] * a[5] + a[4] * a[3]) * inv_det;
}

// The diagonal blocks of a phase, and the inverse of their sum: the block of a node
// whose eight elements are all of this phase (as bjacobi_kernel forms it).
constexpr int kDkdStride = 78;
static __device__ __forceinline__ void store_uniform_inverse(const double (&col)[24][24], double* __restrict__ dkd) {
  if (threadIdx.x != 0) return;
  double M[6], s[6];
  for (int ra = 0; ra < 8; ++ra) {
    const double(*b)[24] = col + 3 * ra;
    const int o = 3 * ra;
    const double d[6] = {b[0][o], b[1][o + 1], b[2][o + 2], b[1][o], b[2][o], b[2][o + 1]};
    for (int i = 0; i < 6; ++i) M[i] = ra == 0 ? d[i] : M[i] + d[i];
  }
  invert3x3(M, s);
  for (int q = 0; q < 6; ++q) dkd[72 + q] = s[q];
}

static __global__ void femat_phase_kernel(FematParams P, const double* __restrict__ rod, double* __restrict__ cmod,
                                   double* __restrict__ cs, float* __restrict__ cs32,
                                   double* __restrict__ dk, double* __restrict__ dkd, double* __restrict__ norms) {
  const int p = blockIdx.x;
  __shared__ double csh[kCsStride];
  __shared__ double col[24][24];  // col[c][r] = (K e_c)[r], c/r = refnode*3 + dof
  __shared__ double C6[6][6], w1[6][6], w2[6][6];
  if (p == P.nphase - 1) {
    isotropic_warp(P.K1, P.G1, C6);
  } else if (P.flag_m == 0) {
    isotropic_warp(P.Km, P.Gm, C6);
  } else {
    const double r[3] = {rod[3 * p], rod[3 * p + 1], rod[3 * p + 2]};
    bond_rotate_warp(r, P.c11, P.c12, P.c44, w1, w2, C6);
  }
  for (int e = threadIdx.x; e < 36; e += 32) cmod[p + (long long)P.nphase * (e / 6 + 6 * (e % 6))] = C6[e / 6][e % 6];
  modal_table_warp(C6, csh, w1, w2);
  __syncthreads();
  for (int i = threadIdx.x; i < kCsStride; i += blockDim.x) cs[(long long)p * kCsStride + i] = csh[i];
  for (int r = threadIdx.x; r < 6; r += blockDim.x)  // FP32: upper triangle of C/16
    for (int c = r; c < 6; ++c) cs32[(long long)p * kCs32Stride + sym6(r, c)] = (float)csh[6 * r + c];
  for (int i = 21 + threadIdx.x; i < kCs32Stride; i += blockDim.x) cs32[(long long)p * kCs32Stride + i] = 0.f;
  // dk columns: K applied to unit nodal vectors with the same element routine
  // as the stencil, so the preconditioner and b see exactly that matrix.
  if (threadIdx.x < 24) {
    const int cidx = threadIdx.x;
    const int rb = cidx / 3, j = cidx % 3;
    double u[3][8], r[3][8];
    for (int c = 0; c < 3; ++c)
      for (int a = 0; a < 8; ++a) u[c][a] = 0.0;
    u[j][kRefToCorner[rb]] = 1.0;
    element_apply<double>(csh, u, r);
    for (int ra = 0; ra < 8; ++ra)
      for (int i = 0; i < 3; ++i) col[cidx][ra * 3 + i] = r[i][kRefToCorner[ra]];
  }
  __syncthreads();
  // symmetric dk: entry (r, c) taken from the column with the larger index
  for (int e = threadIdx.x; e < 576; e += blockDim.x) {
    const int r = e / 24, c = e % 24;
    const double v = (r <= c) ? col[c][r] : col[r][c];
    dk[(long long)p * 576 + e] = v;
    const int ra = r / 3, i = r % 3, cb = c / 3, j = c % 3;
    if (ra == cb) dkd[(long long)p * kDkdStride + ra * 9 + i * 3 + j] = v;
  }
  store_uniform_inverse(col, dkd + (long long)p * kDkdStride);
  fx_store_norms(col, csh, norms + 3 * p);
}

// Integer tables of the fixed-point stencil and their exponent, from all phases'
// norms; every block reduces them itself.
static __global__ void __launch_bounds__(96) fx_table_kernel(int nphase, const double* __restrict__ norms,
                                                             const double* __restrict__ cs, int4* __restrict__ tab,
                                                             double* __restrict__ info) {
  __shared__ double red[4][3];
  __shared__ FxInfo f;
  double d = 0.0, dmin = 1e300, rows = 0.0, entry = 0.0;
  for (int p = threadIdx.x; p < nphase; p += blockDim.x) {
    const double a = norms[3 * p];
    d = fx_max(d, a);
    if (a > 0.0) dmin = fmin(dmin, a);
    rows = fx_max(rows, norms[3 * p + 1]);
    entry = fx_max(entry, norms[3 * p + 2]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d = fx_max(d, __shfl_xor_sync(0xffffffffu, d, o));
    dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    rows = fx_max(rows, __shfl_xor_sync(0xffffffffu, rows, o));
    entry = fx_max(entry, __shfl_xor_sync(0xffffffffu, entry, o));
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = d;
    red[1][w] = dmin;
    red[2][w] = rows;
    red[3][w] = entry;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 3; ++i) {
      d = fx_max(d, red[0][i]);
      dmin = fmin(dmin, red[1][i]);
      rows = fx_max(rows, red[2][i]);
      entry = fx_max(entry, red[3][i]);
    }
    f = fx_info(d, dmin, rows, entry);
    if (blockIdx.x == 0) {
      info[0] = f.kc;
      info[1] = f.ok;
    }
  }
  __syncthreads();
  if (!f.ok) return;
  for (int p = blockIdx.x; p < nphase; p += gridDim.x)
    for (int e = threadIdx.x; e < kFxEntries; e += blockDim.x) {
      int h, l;
      fx_split(fx_source(cs + (long long)p * kCsStride, e), f.kc, h, l);
      reinterpret_cast<int2*>(tab + (long long)p * kFxStride)[e] = make_int2(h, l);
    }
}

// Periodic-jump force b (src/elas3dxtal_pcg.f90:815-1100), node-centric so
// the sum over a node's boundary elements has a fixed order.  An element with
// lower corner (i,j,k) on the high face of any direction d has nodal jumps
// delta(a, :) = sum_d [wrap_d] [o_d(a)] E(:, d) n_d.
struct JumpParams {
  double E[3][3];  // symmetric strain tensor
};

struct ElementJump {
  double T[8][3];  // jump of a corner by the directions in which it crosses (bits x, y, z)
  __device__ __forceinline__ void fill(const GridDims& G, const JumpParams& J, int m) {
    const double n[3] = {(double)G.nx, (double)G.ny, (double)G.nz};
    for (int c = 0; c < 3; ++c) {
      double v = 0.0;
      for (int d = 0; d < 3; ++d)
        if (m >> d & 1) v += J.E[c][d] * n[d];
      T[m][c] = v;
    }
  }
  // directions in which element (x, y, z) crosses a high face
  static __device__ __forceinline__ int crossing(const GridDims& G, int x, int y, int z) {
    return (x == G.nx - 1 ? 1 : 0) | (y == G.ny - 1 ? 2 : 0) | (z == G.nz - 1 ? 4 : 0);
  }
  // row r of D delta over the corners that cross (the others' terms are zero)
  __device__ __forceinline__ double row(const double* __restrict__ D, int r, int w) const {
    double s = 0.0;
#pragma unroll
    for (int rb = 0; rb < 8; ++rb)
      if (kRefToCorner[rb] & w)
#pragma unroll
        for (int c = 0; c < 3; ++c) s += D[r * 24 + rb * 3 + c] * T[kRefToCorner[rb] & w][c];
    return s;
  }
  __device__ __forceinline__ double energy(const double* __restrict__ D, int w) const {  // delta . D delta / 2
    double e = 0.0;
#pragma unroll 1
    for (int ra = 0; ra < 8; ++ra)
      if (kRefToCorner[ra] & w)
#pragma unroll 1
        for (int c = 0; c < 3; ++c) e += T[kRefToCorner[ra] & w][c] * row(D, 3 * ra + c, w);
    return 0.5 * e;
  }
};

// Boundary nodes (x, y or z on a face of the box), each once: the two x faces
// whole, then the y faces at interior x, then the z faces at interior x and y.
// Consecutive indices are consecutive x where the set allows, so a warp's
// lanes share the boundary work instead of idling beside one boundary lane.
__host__ __device__ inline long long boundary_node_count(const GridDims& G) {
  const long long fx = G.nx > 1 ? 2 : 1, fy = G.ny > 1 ? 2 : 1, fz = G.nz > 1 ? 2 : 1;
  const long long ix = G.nx > 2 ? G.nx - 2 : 0, iy = G.ny > 2 ? G.ny - 2 : 0;
  return fx * G.ny * G.nz + ix * fy * G.nz + ix * iy * fz;
}

__device__ __forceinline__ void boundary_node(const GridDims& G, long long t, int& x, int& y, int& z) {
  const long long fx = G.nx > 1 ? 2 : 1, fy = G.ny > 1 ? 2 : 1;
  const long long ix = G.nx > 2 ? G.nx - 2 : 0, iy = G.ny > 2 ? G.ny - 2 : 0;
  const long long na = fx * G.ny * G.nz, nb = ix * fy * G.nz;
  if (t < na) {
    const long long r = t / fx;
    x = (t % fx) == 0 ? 0 : G.nx - 1;
    y = (int)(r % G.ny);
    z = (int)(r / G.ny);
  } else if (t < na + nb) {
    const long long s = t - na, r = s / ix;
    x = 1 + (int)(s % ix);
    y = (r % fy) == 0 ? 0 : G.ny - 1;
    z = (int)(r / fy);
  } else {
    const long long s = t - na - nb, r = s / ix;
    x = 1 + (int)(s % ix);
    y = 1 + (int)(r % iy);
    z = (r / iy) == 0 ? 0 : G.nz - 1;
  }
}

// b over the boundary nodes listed by boundary_node (b is zero elsewhere and
// cleared beforehand): one thread per boundary node.
// Few nodes, much FP64 work each: small blocks, which reach every SM on small grids,
// and no terms of corners that do not cross.  b 70 -> 32 us and C 47 -> 29 at 32^3,
// 672 -> 424 and 337 -> 166 at 300^3.
constexpr int kFematThreads = 64;
static __global__ void femat_b_kernel(GridDims G, JumpParams J, const int32_t* __restrict__ pix,
                               const double* __restrict__ dk, double* __restrict__ b) {
  __shared__ ElementJump jump;
  if (threadIdx.x < 8) jump.fill(G, J, threadIdx.x);
  __syncthreads();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= boundary_node_count(G)) return;
  int x, y, z;
  boundary_node(G, t, x, y, z);
  const long long m = E3D_IDX((long long)x + (long long)G.nx * y + (long long)G.nx * G.ny * z, G.ns);
  double acc[3] = {0.0, 0.0, 0.0};
  // elements containing m in reference order 27,7,6,5,25,15,14,13 (local node ra)
  for (int ra = 0; ra < 8; ++ra) {
    const int a = kRefToCorner[ra];
    const int ex = wrapi(x - (a & 1), G.nx), ey = wrapi(y - ((a >> 1) & 1), G.ny),
              ez = wrapi(z - ((a >> 2) & 1), G.nz);
    const int w = ElementJump::crossing(G, ex, ey, ez);
    if (!w) continue;
    const int ph = pix[E3D_IDX((long long)ex + (long long)G.nx * ey + (long long)G.nx * G.ny * ez, G.ns)];
    const double* D = dk + (long long)ph * 576;
    for (int i = 0; i < 3; ++i) acc[i] += jump.row(D, ra * 3 + i, w);
  }
  b[m] = acc[0];
  b[m + G.ns] = acc[1];
  b[m + 2 * G.ns] = acc[2];
}

// Constant C = 1/2 sum_e delta_e^T K_e delta_e over boundary elements.
static __global__ void __launch_bounds__(kFematThreads) femat_c_kernel(GridDims G, JumpParams J, const int32_t* __restrict__ pix,
                                                      const double* __restrict__ dk, double* partial) {
  __shared__ double red[kFematThreads / 32];
  double acc = 0.0;
  __shared__ ElementJump jump;
  if (threadIdx.x < 8) jump.fill(G, J, threadIdx.x);
  __syncthreads();
  // boundary elements: enumerate the three high faces without double counting
  const long long nfx = (long long)G.ny * G.nz;                        // i = nx-1
  const long long nfy = (long long)(G.nx - 1) * G.nz;                  // j = ny-1, i < nx-1
  const long long nfz = (long long)(G.nx - 1) * (G.ny - 1);            // k = nz-1, i < nx-1, j < ny-1
  const long long total = nfx + nfy + nfz;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    if (t < nfx) {
      i = G.nx - 1;
      j = (int)(t % G.ny);
      k = (int)(t / G.ny);
    } else if (t < nfx + nfy) {
      const long long s = t - nfx;
      j = G.ny - 1;
      i = (int)(s % (G.nx - 1));
      k = (int)(s / (G.nx - 1));
    } else {
      const long long s = t - nfx - nfy;
      k = G.nz - 1;
      i = (int)(s % (G.nx - 1));
      j = (int)(s / (G.nx - 1));
    }
    const int ph = pix[E3D_IDX((long long)i + (long long)G.nx * j + (long long)G.nx * G.ny * k, G.ns)];
    const double* D = dk + (long long)ph * 576;
    acc += jump.energy(D, ElementJump::crossing(G, i, j, k));
  }
  const double s = block_sum<kFematThreads>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Affine initial guess (src/elas3dxtal_pcg.f90:423-438).
// FP64-issue-bound: a thread takes `chunk` nodes of a z column, whose x and y terms
// are one sum, 4 FP64 instructions a node instead of 12 (300^3: 609 -> 234 us).
static __global__ void __launch_bounds__(256) affine_kernel(GridDims G, JumpParams J, int chunk, double* __restrict__ u) {
  const unsigned nxy = (unsigned)G.nx * (unsigned)G.ny, cols = (nxy + 255u) / 256u;
  const unsigned col = blockIdx.x % cols * 256u + threadIdx.x;
  if (col >= nxy) return;
  const double x = (int)(col % (unsigned)G.nx), y = (int)(col / (unsigned)G.nx);
  const double exx = J.E[0][0], eyy = J.E[1][1], ezz = J.E[2][2];
  const double exy = J.E[0][1], exz = J.E[0][2], eyz = J.E[1][2];
  const double c0 = x * exx + y * exy, c1 = x * exy + y * eyy, c2 = x * exz + y * eyz;
  const int z0 = (int)(blockIdx.x / cols) * chunk, z1 = min(G.nz, z0 + chunk);
  for (int zi = z0; zi < z1; ++zi) {
    const double z = zi;
    const long long m = (long long)col + (long long)nxy * zi;
    u[m] = c0 + z * exz;
    u[m + G.ns] = c1 + z * eyz;
    u[m + 2 * G.ns] = c2 + z * ezz;
  }
}
// Block-Jacobi (src/elas3dxtal_pcg.f90:1498-1520): sum of the node's diagonal
// 3x3 blocks over its 8 elements (reference order), inverted.  Stores the
// symmetric inverse as 6 SoA planes (00 11 22 01 02 12) in FP64 and FP32.
constexpr int kBjacobiPer = 4;
static __global__ void __launch_bounds__(256) bjacobi_kernel(GridDims G, int per, const int32_t* __restrict__ pix,
                                                             const double* __restrict__ dkd, double* __restrict__ minv,
                                                             float* __restrict__ minv32, int identity = 0) {
  // FP64-issue-bound (73 instructions a node), so a block of 256 * per nodes first
  // serves those inside a grain, whose eight elements are of one phase and whose
  // inverse is in the phase's table, and then inverts for the others side by side.
  // 300^3 polycrystal: 3.45 -> 0.81 ms.
  __shared__ unsigned short todo[256 * kBjacobiPer];
  __shared__ int n;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * (256 * per);
  auto store = [&](long long m, const double* s) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      if (minv) minv[m + q * G.ns] = s[q];
      if (minv32) minv32[m + q * G.ns] = (float)s[q];
    }
  };
  auto phases = [&](long long m, int (&ph)[8]) {  // of the elements around the node, by local node
    int x, y, z;
    node_xyz(G, m, x, y, z);
#pragma unroll
    for (int ra = 0; ra < 8; ++ra) {
      const int a = kRefToCorner[ra];
      const int ex = wrapi(x - (a & 1), G.nx), ey = wrapi(y - ((a >> 1) & 1), G.ny),
                ez = wrapi(z - ((a >> 2) & 1), G.nz);
      ph[ra] = pix[E3D_IDX((long long)ex + (long long)G.nx * ey + (long long)G.nx * G.ny * ez, G.ns)];
    }
  };
  for (int j = 0; j < per; ++j) {
    const int i = j * 256 + threadIdx.x;
    const long long m = base + i;
    if (m >= G.ns) break;
    if (identity) {  // plain CG: z = g
      const double one[6] = {1.0, 1.0, 1.0, 0.0, 0.0, 0.0};
      store(m, one);
      continue;
    }
    int ph[8];
    phases(m, ph);
    bool same = true;
#pragma unroll
    for (int ra = 1; ra < 8; ++ra) same = same && ph[ra] == ph[0];
    if (same) {
      double s[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) s[q] = __ldg(dkd + (long long)ph[0] * kDkdStride + 72 + q);
      store(m, s);
    } else {
      todo[atomicAdd(&n, 1)] = (unsigned short)i;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n; t += 256) {
    const long long m = base + todo[t];
    int ph[8];
    phases(m, ph);
    double M[6], s[6];  // the six distinct entries of the block, and of its inverse
#pragma unroll
    for (int ra = 0; ra < 8; ++ra) {
      const double* D = dkd + (long long)ph[ra] * kDkdStride + ra * 9;
      const double d[6] = {__ldg(D), __ldg(D + 4), __ldg(D + 8), __ldg(D + 1), __ldg(D + 2), __ldg(D + 5)};
#pragma unroll
      for (int i = 0; i < 6; ++i) M[i] = ra == 0 ? d[i] : M[i] + d[i];
    }
    invert3x3(M, s);
    store(m, s);
  }
}

// `per` above: four once that leaves every SM eight blocks (more nodes to share the
// few inversions among), else one.
inline int bjacobi_per(long long ns, int sms) { return ns >= (long long)sms * 8 * 256 * kBjacobiPer ? kBjacobiPer : 1; }
inline unsigned bjacobi_grid(long long ns, int per) { return (unsigned)((ns + 256 * per - 1) / (256 * per)); }

template <typename T>
__device__ __forceinline__ void precond3(const T* __restrict__ mi, long long m, long long ns, const T (&g)[3],
                                         T (&z)[3]) {
  const T a00 = mi[m], a11 = mi[m + ns], a22 = mi[m + 2 * ns];
  const T a01 = mi[m + 3 * ns], a02 = mi[m + 4 * ns], a12 = mi[m + 5 * ns];
  // z(i) = Minv(i,1) g1 + Minv(i,2) g2 + Minv(i,3) g3 (src/elas3dxtal_pcg.f90:1930-1932)
  z[0] = a00 * g[0] + a01 * g[1] + a02 * g[2];
  z[1] = a01 * g[0] + a11 * g[1] + a12 * g[2];
  z[2] = a02 * g[0] + a12 * g[1] + a22 * g[2];
}

// ---------------------------------------------------------------------------
// Stress (stress_OpenMP :2149-2408, stress_fullfield_OpenMP :2723-2833).
__device__ __forceinline__ void voxel_strain(const GridDims& G, const JumpParams& J, const double* __restrict__ u,
                                             int x, int y, int z, double (&eps)[6]) {
  double v[3][8];
  for (int a = 0; a < 8; ++a) {
    const int ox = a & 1, oy = (a >> 1) & 1, oz = (a >> 2) & 1;
    const int xx = x + ox >= G.nx ? 0 : x + ox, yy = y + oy >= G.ny ? 0 : y + oy,
              zz = z + oz >= G.nz ? 0 : z + oz;
    const long long mm = E3D_IDX((long long)xx + (long long)G.nx * yy + (long long)G.nx * G.ny * zz, G.ns);
    for (int c = 0; c < 3; ++c) v[c][a] = u[mm + c * G.ns];
  }
  // periodic jump, x then y then z as at :2282-2323
  if (x == G.nx - 1)
    for (int a = 0; a < 8; ++a)
      if (a & 1)
        for (int c = 0; c < 3; ++c) v[c][a] += J.E[c][0] * (double)G.nx;
  if (y == G.ny - 1)
    for (int a = 0; a < 8; ++a)
      if (a & 2)
        for (int c = 0; c < 3; ++c) v[c][a] += J.E[c][1] * (double)G.ny;
  if (z == G.nz - 1)
    for (int a = 0; a < 8; ++a)
      if (a & 4)
        for (int c = 0; c < 3; ++c) v[c][a] += J.E[c][2] * (double)G.nz;
  // centre strain = (1/4) x first-order Hadamard differences (engineering shear),
  // differences before sums: neighbours differ little, so they are nearly exact
  double dX[3], dY[3], dZ[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    dX[c] = ((v[c][1] - v[c][0]) + (v[c][3] - v[c][2])) + ((v[c][5] - v[c][4]) + (v[c][7] - v[c][6]));
    dY[c] = ((v[c][2] - v[c][0]) + (v[c][3] - v[c][1])) + ((v[c][6] - v[c][4]) + (v[c][7] - v[c][5]));
    dZ[c] = ((v[c][4] - v[c][0]) + (v[c][5] - v[c][1])) + ((v[c][6] - v[c][2]) + (v[c][7] - v[c][3]));
  }
  eps[0] = 0.25 * dX[0];
  eps[1] = 0.25 * dY[1];
  eps[2] = 0.25 * dZ[2];
  eps[3] = 0.25 * (dZ[0] + dX[2]);
  eps[4] = 0.25 * (dZ[1] + dY[2]);
  eps[5] = 0.25 * (dY[0] + dX[1]);
}

// Volume sums of stress and strain (src/elas3dxtal_pcg.f90:2149-2408).  The stress
// of a voxel is C(phase) . strain, so only the gradients are summed over the voxels,
// phase by phase: 81 additions a voxel instead of 130 FP64 operations.  They are
// 64-bit integers as in the fixed-point stencil, with one exponent for each component
// of u (its largest value over the grid) and the periodic jumps of it, and their sums,
// in two words of 64 bits, are exact and so do not depend on the order in which
// threads add a run of voxels of one phase to its sums.  300^3: 6.55 ms voxel by
// voxel in FP64, 1.03 with the maxima and the final sums.
// Of phase p, from word kPhaseSums * p: low and high halves of the nine sums (component
// c, direction d: 2 * (3 c + d); first-order Hadamard sums, four times the gradient),
// then the runs added, zero for a phase that has no voxel.  info: the exponents.
// Values that are not finite or out of the exponents' range: FP64, voxel by voxel,
// to the partials of pgrid blocks.
constexpr int kPhaseSums = 19;
struct StressInfo {
  int kx[3];           // kx[0] == kFxGeneral: the FP64 sums
  unsigned largest[3];  // size_word of each component's largest value
};

static __global__ void __launch_bounds__(256) component_max_kernel(long long ns, const double* __restrict__ u,
                                                                   StressInfo* __restrict__ info) {
  unsigned w[3] = {0, 0, 0};
  for (long long m = (long long)blockIdx.x * 256 + threadIdx.x; m < ns; m += (long long)gridDim.x * 256)
#pragma unroll
    for (int c = 0; c < 3; ++c) w[c] = max(w[c], size_word(__ldcg(u + m + c * ns)));
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const unsigned v = __reduce_max_sync(0xffffffffu, w[c]);
    if ((threadIdx.x & 31) == 0 && v) atomicMax(&info->largest[c], v);
  }
}

static __device__ __noinline__ void stress_general(const GridDims& G, const JumpParams& J, const int32_t* __restrict__ pix,
                                                   const double* __restrict__ cmod, int nphase,
                                                   const double* __restrict__ u, double* partial, int pgrid, double* red) {
  if ((int)blockIdx.x >= pgrid) return;
  double acc[12];
  for (int t = 0; t < 12; ++t) acc[t] = 0.0;
  for (long long m = (long long)blockIdx.x * kFxThreads + threadIdx.x; m < G.ns; m += (long long)pgrid * kFxThreads) {
    int x, y, z;
    node_xyz(G, m, x, y, z);
    double eps[6];
    voxel_strain(G, J, u, x, y, z, eps);
    const int ph = pix[m];
    for (int r = 0; r < 6; ++r) {
      double s = 0.0;
      for (int c = 0; c < 6; ++c) s += cmod[E3D_IDX(ph, nphase) + (long long)nphase * (r + 6 * c)] * eps[c];
      acc[r] += s;
      acc[6 + r] += eps[r];
    }
  }
  for (int t = 0; t < 12; ++t) {
    const double s = block_sum<kFxThreads>(acc[t], red);
    if (threadIdx.x == 0) partial[12 * (long long)blockIdx.x + t] = s;
  }
}

static __global__ void __launch_bounds__(kFxThreads) stress_sums_kernel(
    GridDims G, JumpParams J, const int32_t* __restrict__ pix, const double* __restrict__ cmod, int nphase,
    const double* __restrict__ u, unsigned long long* __restrict__ sums, StressInfo* __restrict__ info,
    double* partial, int pgrid) {
  constexpr int kHalo = TILE_X + kFxRows + 1, kRow = TILE_X + 1, cst = kRow * (kFxRows + 1);
  __shared__ long long node[2][3][cst];
  __shared__ double raw[3][kFxThreads + kHalo];
  __shared__ double red[kFxThreads / 32];
  const int tid = threadIdx.x;
  const double n3[3] = {(double)G.nx, (double)G.ny, (double)G.nz};
  int kx[3];
  bool general = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const unsigned w = info->largest[c];
    double big = w ? __hiloint2double((int)w + 1, 0) : 0.0;
    for (int d = 0; d < 3; ++d) big = fx_max(big, fabs(J.E[c][d] * n3[d]));
    kx[c] = w >= 0x7ff00000u ? kFxGeneral : fx_exponent_below(big);
    general = general || kx[c] == kFxGeneral;
  }
  if (blockIdx.x == 0 && tid < 3) info->kx[tid] = general ? kFxGeneral : tid == 0 ? kx[0] : tid == 1 ? kx[1] : kx[2];
  if (general) {
    stress_general(G, J, pix, cmod, nphase, u, partial, pgrid, red);
    return;
  }
  const int tx = tid % TILE_X, ty = tid / TILE_X;
  const long long tile = blockIdx.x;
  const int tix = (int)(tile % G.ntx), tiy = (int)((tile / G.ntx) % G.nty),
            tiz = (int)(tile / ((long long)G.ntx * G.nty));
  const int x0 = tix * TILE_X, y0 = tiy * kFxRows, z0 = tiz * G.tz;
  const int wx = min(TILE_X, G.nx - x0), wy = min(kFxRows, G.ny - y0), zend = min(G.nz, z0 + G.tz);
  const bool active = tx < wx && ty < wy;
  const int nhalo = wx + wy + 1;
  int hlx = wx, hly = wy;  // halo node of loader thread tid < nhalo
  if (tid < wy)
    hly = tid;
  else if (tid < wy + wx)
    hlx = tid - wy;
  const long long ns = G.ns, nxy = (long long)G.nx * G.ny;
  const long long own = (long long)(x0 + tx) + (long long)G.nx * (y0 + ty);
  const long long halo = (long long)wrapi(x0 + hlx, G.nx) + (long long)G.nx * wrapi(y0 + hly, G.ny);
  auto load = [&](int zl) {
    const long long zo = nxy * wrapi(zl, G.nz);
    if (active) {
      const long long m = E3D_IDX(own + zo, ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async_8(&raw[c][tid], u + m + c * ns);
    }
    if (tid < nhalo) {
      const long long m = E3D_IDX(halo + zo, ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async_8(&raw[c][kFxThreads + tid], u + m + c * ns);
    }
    cp_async_commit();
  };
  auto convert = [&](int buf) {
    cp_async_wait<0>();
    if (active) {
#pragma unroll
      for (int c = 0; c < 3; ++c) node[buf][c][ty * kRow + tx] = fx_from_double(raw[c][tid], kx[c]);
    }
    if (tid < nhalo) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        node[buf][c][E3D_IDX(hly * kRow + hlx, cst)] = fx_from_double(raw[c][kFxThreads + tid], kx[c]);
    }
  };
  // sum, x and y difference of the voxel's four nodes of a plane
  auto plane = [&](int buf, long long (&P)[3][3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long* v = node[buf][c] + ty * kRow + tx;
      const long long v0 = v[0], v1 = v[1], v2 = v[kRow], v3 = v[kRow + 1];
      const long long s0 = v0 + v1, s1 = v2 + v3;
      P[c][0] = s0 + s1;
      P[c][1] = (v1 - v0) + (v3 - v2);
      P[c][2] = s1 - s0;
    }
  };
  // what the periodic jumps add at the last voxel of x, y and z
  const bool jx = active && x0 + tx == G.nx - 1, jy = active && y0 + ty == G.ny - 1;
  auto jump = [&](int c, int d) { return 4 * fx_from_double(J.E[c][d] * n3[d], kx[c]); };
  unsigned long long lo[9] = {};
  long long hi[9] = {};
  int cur = -1;
  // Adds the runs of the lanes with `ends` to their phases' sums and clears them.  The
  // lanes of one phase are added up first (in pieces of 26 bits, whose sums fit 32),
  // and nineteen lanes then add a word each: every thread by itself, all to the words
  // of a few phases, took 158 us on a grid of 32^3, where this takes 9.5.
  auto flush = [&](bool ends) {
    const int lane = tid & 31;
    unsigned left = __ballot_sync(0xffffffffu, ends);
    while (left) {
      const int p = __shfl_sync(0xffffffffu, cur, __ffs(left) - 1);
      const bool in = ends && cur == p;
      unsigned long long word = 0;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const unsigned l0 = __reduce_add_sync(0xffffffffu, in ? (unsigned)lo[i] & 0x3ffffffu : 0u),
                       l1 = __reduce_add_sync(0xffffffffu, in ? (unsigned)(lo[i] >> 26) : 0u),
                       h0 = __reduce_add_sync(0xffffffffu, in ? (unsigned)hi[i] & 0x3ffffffu : 0u);
        const int h1 = __reduce_add_sync(0xffffffffu, in ? (int)(hi[i] >> 26) : 0);
        if (lane == 2 * i) word = l0 + ((unsigned long long)l1 << 26);
        if (lane == 2 * i + 1) word = h0 + (unsigned long long)((long long)h1 * (1 << 26));
      }
      if (lane == 18) word = 1;
      if (lane < kPhaseSums) atomicAdd(sums + kPhaseSums * (long long)E3D_IDX(p, nphase) + lane, word);
      left &= ~__ballot_sync(0xffffffffu, in);
    }
    if (ends) {
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        lo[i] = 0;
        hi[i] = 0;
      }
    }
  };
  load(z0);
  convert(0);
  load(z0 + 1);
  __syncthreads();
  long long Po[3][3] = {};
  if (active) plane(0, Po);
  for (int k = z0; k < zend; ++k) {
    const int ph = active ? __ldcs(pix + E3D_IDX(own + nxy * k, ns)) : -1;
    const int buf = (k + 1 - z0) & 1;
    convert(buf);
    if (k + 2 <= zend) load(k + 2);
    __syncthreads();
    if (__any_sync(0xffffffffu, ph != cur && cur >= 0)) flush(ph != cur && cur >= 0);
    cur = ph;
    if (!active) continue;
    long long Pn[3][3];
    plane(buf, Pn);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      long long e[3] = {Pn[c][1] + Po[c][1], Pn[c][2] + Po[c][2], Pn[c][0] - Po[c][0]};
      if (jx) e[0] += jump(c, 0);
      if (jy) e[1] += jump(c, 1);
      if (k == G.nz - 1) e[2] += jump(c, 2);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        Po[c][d] = Pn[c][d];
        lo[3 * c + d] += (unsigned)e[d];
        hi[3 * c + d] += e[d] >> 32;
      }
    }
  }
  flush(cur >= 0);
}

// The six sums of stress and of strain, from the sums over the phases.
static __global__ void __launch_bounds__(256) stress_total_kernel(int nphase, const unsigned long long* __restrict__ sums,
                                                                  const StressInfo* __restrict__ info,
                                                                  const double* __restrict__ cmod,
                                                                  const double* __restrict__ partial, int pgrid,
                                                                  double* __restrict__ out) {
  __shared__ double red[8];
  double acc[12];
  for (int t = 0; t < 12; ++t) acc[t] = 0.0;
  if (info->kx[0] == kFxGeneral) {
    for (int i = threadIdx.x; i < pgrid; i += 256)
      for (int t = 0; t < 12; ++t) acc[t] += partial[12 * (long long)i + t];
  } else {
    for (int p = threadIdx.x; p < nphase; p += 256) {
      const unsigned long long* sum = sums + kPhaseSums * (long long)p;
      if (sum[18] == 0) continue;  // no voxel: its stiffness, whatever it is, counts for nothing
      double g[3][3];
      for (int q = 0; q < 9; ++q) {
        const __int128 t = ((__int128)(long long)sum[2 * q + 1] << 32) + sum[2 * q];
        g[q / 3][q % 3] = ldexp(ldexp((double)(long long)(t >> 32), 32) + (double)(unsigned)t, -info->kx[q / 3] - 2);
      }
      const double eps[6] = {g[0][0], g[1][1], g[2][2], g[0][2] + g[2][0], g[1][2] + g[2][1], g[0][1] + g[1][0]};
      for (int c = 0; c < 6; ++c) acc[6 + c] += eps[c];
      for (int r = 0; r < 6; ++r) {
        double s = 0.0;
        for (int c = 0; c < 6; ++c) s += cmod[p + (long long)nphase * (r + 6 * c)] * eps[c];
        acc[r] += s;
      }
    }
  }
  for (int t = 0; t < 12; ++t) {
    const double s = block_sum<256>(acc[t], red);
    if (threadIdx.x == 0) out[t] = s;
  }
}

static __global__ void stress_field_kernel(GridDims G, JumpParams J, const int32_t* __restrict__ pix,
                                    const double* __restrict__ cmod, int nphase, const double* __restrict__ u,
                                    double* __restrict__ sigma, double* __restrict__ vm) {
  const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= G.ns) return;
  int x, y, z;
  node_xyz(G, m, x, y, z);
  double eps[6];
  voxel_strain(G, J, u, x, y, z, eps);
  const int ph = pix[m];
  double s6[6];
  for (int r = 0; r < 6; ++r) {
    double s = 0.0;
    for (int c = 0; c < 6; ++c) s += cmod[E3D_IDX(ph, nphase) + (long long)nphase * (r + 6 * c)] * eps[c];
    s6[r] = s;
    if (sigma) sigma[m + r * G.ns] = s;
  }
  if (vm) {
    const double a = s6[0] - s6[1], bq = s6[1] - s6[2], c = s6[2] - s6[0];
    vm[m] = sqrt(0.5 * (a * a + bq * bq + c * c + 6.0 * (s6[3] * s6[3] + s6[4] * s6[4] + s6[5] * s6[5])));
  }
}

// Phase B of the ring-fed kernel, whose shared memory the ring fills: as
// pcg_update_tiles_v below, with U nodes of a column per thread in registers
// (src/elas3dxtal_pcg.f90:1913-1932, symmetric Minv).
template <typename T, int U>
__device__ __forceinline__ double pcg_update_tiles(const GridDims& G, long long first, long long stride, T lam,
                                                   const T* __restrict__ hc, const T* __restrict__ Ah,
                                                   const T* __restrict__ hx, const T* __restrict__ hy,
                                                   const T* __restrict__ hd, const T* __restrict__ minv,
                                                   T* __restrict__ u, T* __restrict__ g, T* __restrict__ z) {
  const long long ns = G.ns;
  double zg_t = 0.0;
  const int tx = threadIdx.x % TILE_X, ty = threadIdx.x / TILE_X;
  const long long nxy = (long long)G.nx * G.ny;
  for (long long t = first; t < G.ntiles; t += stride) {
    const int tix = (int)(t % G.ntx);
    const int tiy = (int)((t / G.ntx) % G.nty);
    const int tiz = (int)(t / ((long long)G.ntx * G.nty));
    const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
    const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(G.tz, G.nz - z0);
    if (tx >= wx || ty >= wy) continue;
    const long long col = (long long)(x0 + tx) + (long long)G.nx * (y0 + ty);
    float zg32 = 0.f;  // FP32: this column's z.g, added to the FP64 sum once per tile
    for (int lz0 = 0; lz0 < wz; lz0 += U) {
      T ah[U][3], hv[U][3], uv[U][3], gv[U][3], mi[U][6];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (lz0 + j < wz) {
          const long long m = E3D_IDX(col + nxy * (z0 + lz0 + j), ns);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            ah[j][c] = __ldcg(Ah + m + c * ns);
            hv[j][c] = __ldcg(hc + m + c * ns);
            uv[j][c] = u[m + c * ns];
            gv[j][c] = g[m + c * ns];
          }
#pragma unroll
          for (int q = 0; q < 6; ++q) mi[j][q] = __ldg(minv + m + q * ns);
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (lz0 + j < wz) {
          const long long m = E3D_IDX(col + nxy * (z0 + lz0 + j), ns);
          halo_add_tile<T>(G, hx, hy, hd, tix, tiy, tiz, tx, ty, lz0 + j, ah[j]);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            u[m + c * ns] = uv[j][c] - lam * hv[j][c];
            gv[j][c] = gv[j][c] - lam * ah[j][c];
            g[m + c * ns] = gv[j][c];
          }
          const T z0v = mi[j][0] * gv[j][0] + mi[j][3] * gv[j][1] + mi[j][4] * gv[j][2];
          const T z1v = mi[j][3] * gv[j][0] + mi[j][1] * gv[j][1] + mi[j][5] * gv[j][2];
          const T z2v = mi[j][4] * gv[j][0] + mi[j][5] * gv[j][1] + mi[j][2] * gv[j][2];
          z[m] = z0v;
          z[m + ns] = z1v;
          z[m + 2 * ns] = z2v;
          if constexpr (sizeof(T) == 4)
            zg32 += z0v * gv[j][0] + z1v * gv[j][1] + z2v * gv[j][2];
          else
            zg_t += (double)(z0v * gv[j][0] + z1v * gv[j][1] + z2v * gv[j][2]);
        }
      }
    }
    if constexpr (sizeof(T) == 4) zg_t += (double)zg32;
  }
  return zg_t;
}

// ---------------------------------------------------------------------------
// Phase B of a PCG iteration over tiles first, first + stride, ...: g -= lam Ah
// (+ tile-edge halos), z = Minv g, u -= lam h too with UPD_U (else the next phase A
// does it); returns this thread's share of z.g (FP32: summed per thread and tile in
// FP32, then in FP64).  Bound by HBM in FP32, by the FP64 pipe as much in FP64.
// NTH threads share a tile, V consecutive nodes of a row each, NTH * V / 32 rows a
// step.  V = 4, 2 or 1 by the rows' alignment: a quarter or half of the load,
// store and address instructions of the one-node form.  Loads are in flight
// through S cp.async stages that the loading thread alone reads back, so that no
// barrier is needed and they hold no registers.  Iteration with two nodes a thread
// instead of one (four stages): FP32 500^3 6.00 -> 5.72 ms, 200^3 .414 -> .389, 100^3
// .0757 -> .0716; FP64 300^3 4.63 -> 4.52.  Four nodes a thread: 500^3 6.29.  The
// grid's warps side by side along memory instead of tile by tile: 8.0.
// ZMAX: the row maxima of the new z go to mz (FxRowMaxFused, for the next pass).
template <int BYTES>
__device__ __forceinline__ void cp_async_n(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  else if constexpr (BYTES == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
template <typename T, int V>
struct alignas(sizeof(T) * V) VecOf {
  T v[V];
};

// Values of one stage: per thread Ah 3, g 3, Minv 6 (and h 3, u 3 with UPD_U), V
// each, then the halo slots of the step's rows and planes: hy[3][planes][32],
// hx[3][rows], hd[3][planes].
template <int NTH, int V>
__host__ __device__ constexpr int pv_rows() {
  return NTH * V / TILE_X;
}
template <int NTH, int TY, int V>
__host__ __device__ constexpr int pv_planes() {
  return pv_rows<NTH, V>() > TY ? pv_rows<NTH, V>() / TY : 1;
}
template <typename T, int NTH, int TY, int V, bool UPD_U>
__host__ __device__ constexpr int pv_stage() {  // a multiple of 16 bytes
  const int halo = 3 * (pv_planes<NTH, TY, V>() * (TILE_X + 1) + pv_rows<NTH, V>()), a = 16 / (int)sizeof(T);
  return (UPD_U ? 18 : 12) * NTH * V + (halo + a - 1) / a * a;
}
// Bytes of S * VMAX / V stages, for every V up to VMAX.
template <typename T, int NTH, int TY, int VMAX, int S, bool UPD_U>
__host__ __device__ constexpr int pv_bytes() {
  int b = 0;
  for (int c : {VMAX * S * pv_stage<T, NTH, TY, 1, UPD_U>(), VMAX / 2 * S * pv_stage<T, NTH, TY, 2, UPD_U>(),
                VMAX == 4 ? S * pv_stage<T, NTH, TY, 4, UPD_U>() : 0})
    b = b > c ? b : c;
  return b * (int)sizeof(T);
}

template <typename T, int NTH, int TY, int V, int S, bool UPD_U, bool ZMAX>
__device__ __forceinline__ double pcg_update_tiles_v(const GridDims& G, long long first, long long stride, T lam,
                                                     const T* __restrict__ hc, const T* __restrict__ Ah,
                                                     const T* __restrict__ hx, const T* __restrict__ hy,
                                                     const T* __restrict__ hd, const T* __restrict__ minv,
                                                     T* __restrict__ u, T* __restrict__ g, T* __restrict__ z,
                                                     T* __restrict__ stages, int tid, unsigned* __restrict__ mz) {
  static_assert((S & (S - 1)) == 0, "stage count: a power of two");
  constexpr int F = UPD_U ? 18 : 12, SL = pv_stage<T, NTH, TY, V, UPD_U>(), R = pv_rows<NTH, V>(),
                PL = pv_planes<NTH, TY, V>();
  static_assert(R % TY == 0 || TY % R == 0, "whole planes a step, or whole steps a plane");
  constexpr int B = V * (int)sizeof(T);
  constexpr int kLanes = TILE_X / V;  // threads of a row
  using Vec = VecOf<T, V>;
  const long long ns = G.ns;  // in a register: G may lie in shared memory, read again after every copy issued
  const unsigned nx = (unsigned)G.nx, nxy = nx * (unsigned)G.ny;
  const int rs = tid / kLanes, tx = (tid % kLanes) * V;  // row slot of the step, first column
  const int pl = rs / TY;                                // plane of the step
  const long long per_c = G.ntiles * (long long)G.tz;
  double zg_t = 0.0;
  for (long long t = first; t < G.ntiles; t += stride) {
    const int tix = (int)(t % G.ntx);
    const int tiy = (int)((t / G.ntx) % G.nty);
    const int tiz = (int)(t / ((long long)G.ntx * G.nty));
    const int x0 = tix * TILE_X, y0 = tiy * TY, z0 = tiz * G.tz;
    const int wx = min(TILE_X, G.nx - x0), wy = min(TY, G.ny - y0), wz = min(G.tz, G.nz - z0);
    const int steps = (wz * TY + R - 1) / R;
    const int txl = tix == 0 ? G.ntx - 1 : tix - 1;
    const int tyd = tiy == 0 ? G.nty - 1 : tiy - 1;
    const long long plane = (long long)tiz * G.nty;
    const long long tX = (long long)txl + (long long)G.ntx * (tiy + plane);
    const long long tY = (long long)tix + (long long)G.ntx * (tyd + plane);
    const long long tD = (long long)txl + (long long)G.ntx * (tyd + plane);
    // of step j: plane and row of this thread, and whether it has nodes
    auto place = [&](int j, int& lz, int& row) {
      lz = (j * R + rs) / TY;
      row = R % TY == 0 ? rs % TY : (j * R + rs) % TY;
      return tx < wx && row < wy && lz < wz;
    };
    const unsigned base = (unsigned)(x0 + tx) + nx * (unsigned)y0 + nxy * (unsigned)z0;
    auto issue = [&](int j) {
      int lz, row;
      if (place(j, lz, row)) {
        T* d = stages + (j & (S - 1)) * SL;
        const unsigned m = base + nx * (unsigned)row + nxy * (unsigned)lz;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const unsigned long long i = E3D_IDX(value_of(m, c, ns), 3 * ns);
          cp_async_n<B>(d + (c * NTH + tid) * V, Ah + i);
          cp_async_n<B>(d + ((3 + c) * NTH + tid) * V, g + i);
          if constexpr (UPD_U) {
            cp_async_n<B>(d + ((12 + c) * NTH + tid) * V, hc + i);
            cp_async_n<B>(d + ((15 + c) * NTH + tid) * V, u + i);
          }
        }
#pragma unroll
        for (int q = 0; q < 6; ++q)
          cp_async_n<B>(d + ((6 + q) * NTH + tid) * V, minv + E3D_IDX(value_of(m, q, ns), 6 * ns));
        T* hs = d + F * NTH * V;
        if (row == 0) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
            cp_async_n<B>(hs + (c * PL + pl) * TILE_X + tx,
                          hy + E3D_IDX((c * per_c + tY * G.tz + lz) * TILE_X + tx, 3 * per_c * TILE_X));
        }
        if (tx == 0) {
          T* hxs = hs + 3 * PL * TILE_X;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            cp_async_n<sizeof(T)>(hxs + c * R + rs,
                                  hx + E3D_IDX((c * per_c + tX * G.tz + lz) * TY + row, 3 * per_c * TY));
          if (row == 0) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
              cp_async_n<sizeof(T)>(hxs + 3 * R + c * PL + pl, hd + E3D_IDX(c * per_c + tD * G.tz + lz, 3 * per_c));
          }
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int j = 0; j < S - 1; ++j) issue(j);
    float zg32 = 0.f;  // FP32: this thread's z.g, added to the FP64 sum once per tile
    unsigned zmax = 0;
    for (int j = 0; j < steps; ++j) {
      issue(j + S - 1);
      cp_async_wait<S - 1>();  // step j has landed
      int lz, row;
      if (!place(j, lz, row)) continue;
      const T* d = stages + (j & (S - 1)) * SL;
      const T* hs = d + F * NTH * V;
      auto field = [&](int q) { return *reinterpret_cast<const Vec*>(d + (q * NTH + tid) * V); };
      Vec ah[3], gv[3], zv[3], uv[3], hv[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        ah[c] = field(c);
        gv[c] = field(3 + c);
        if constexpr (UPD_U) {
          hv[c] = field(12 + c);
          uv[c] = field(15 + c);
        }
      }
      const Vec m00 = field(6), m11 = field(7), m22 = field(8), m01 = field(9), m02 = field(10), m12 = field(11);
      if (tx == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) ah[c].v[0] += hs[3 * PL * TILE_X + c * R + rs];
      }
      if (row == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const Vec a = *reinterpret_cast<const Vec*>(hs + (c * PL + pl) * TILE_X + tx);
#pragma unroll
          for (int i = 0; i < V; ++i) ah[c].v[i] += a.v[i];
        }
        if (tx == 0) {
#pragma unroll
          for (int c = 0; c < 3; ++c) ah[c].v[0] += hs[3 * PL * TILE_X + 3 * R + c * PL + pl];
        }
      }
      const unsigned m = base + nx * (unsigned)row + nxy * (unsigned)lz;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int i = 0; i < V; ++i) gv[c].v[i] -= lam * ah[c].v[i];
        const unsigned long long o = E3D_IDX(value_of(m, c, ns), 3 * ns);
        *reinterpret_cast<Vec*>(g + o) = gv[c];
        if constexpr (UPD_U) {
#pragma unroll
          for (int i = 0; i < V; ++i) uv[c].v[i] -= lam * hv[c].v[i];
          *reinterpret_cast<Vec*>(u + o) = uv[c];
        }
      }
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const T a = gv[0].v[i], b = gv[1].v[i], c = gv[2].v[i];
        zv[0].v[i] = m00.v[i] * a + m01.v[i] * b + m02.v[i] * c;
        zv[1].v[i] = m01.v[i] * a + m11.v[i] * b + m12.v[i] * c;
        zv[2].v[i] = m02.v[i] * a + m12.v[i] * b + m22.v[i] * c;
        const T zg = zv[0].v[i] * a + zv[1].v[i] * b + zv[2].v[i] * c;
        if constexpr (sizeof(T) == 4)
          zg32 += zg;
        else
          zg_t += zg;
        if constexpr (ZMAX)
          zmax = max(zmax, max(abs_hi(zv[0].v[i]), max(abs_hi(zv[1].v[i]), abs_hi(zv[2].v[i]))));
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) *reinterpret_cast<Vec*>(z + E3D_IDX(value_of(m, c, ns), 3 * ns)) = zv[c];
    }
    if constexpr (ZMAX) {  // a thread's nodes lie in one row; slots rs and rs + TY are of the same
      static_assert(R == TY || R == 2 * TY, "one slot a row, or two");
      const int half = V == 2 ? (tid & 31) / kLanes : 0;
      const unsigned a = __reduce_max_sync(0xffffffffu, half ? 0u : zmax),
                     b = V == 2 ? __reduce_max_sync(0xffffffffu, half ? zmax : 0u) : 0u;
      if (tid % kLanes == 0) mz[E3D_IDX(t * 2 * TY + rs, G.ntiles * 2 * TY)] = half ? b : a;
    }
    if constexpr (sizeof(T) == 4) zg_t += (double)zg32;
    cp_async_wait<0>();
  }
  return zg_t;
}

// du -= lam h over the nodes that a thread owns in apply_tile_f2.
static __device__ void flush_u_tiles_f2(const GridDims& G, long long first, long long stride, float lam,
                                        const float* __restrict__ h, float* __restrict__ u, int tid) {
  const unsigned nx = (unsigned)G.nx, nxy = nx * (unsigned)G.ny;
  const int tx = tid % TILE_X, ya = 2 * (tid / TILE_X);
  for (long long t = first; t < G.ntiles; t += stride) {
    const int tix = (int)(t % G.ntx);
    const int tiy = (int)((t / G.ntx) % G.nty);
    const int tiz = (int)(t / ((long long)G.ntx * G.nty));
    const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
    const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(G.tz, G.nz - z0);
    if (tx >= wx) continue;
    for (int row = ya; row < min(wy, ya + 2); ++row)
      for (int lz = 0; lz < wz; ++lz) {
        const unsigned m = (unsigned)(x0 + tx) + nx * (unsigned)(y0 + row) + nxy * (unsigned)(z0 + lz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const unsigned long long i = E3D_IDX(value_of(m, c, G.ns), 3 * G.ns);
          u[i] = u[i] - lam * __ldcg(h + i);
        }
      }
  }
}

// u -= lam h over the owned nodes of tiles first, first + stride, ... (the same
// tile and column ownership as apply_tile and pcg_update_tiles).
template <typename T>
__device__ void flush_u_tiles(const GridDims& G, long long first, long long stride, T lam, const T* __restrict__ h,
                              T* __restrict__ u) {
  const long long ns = G.ns;
  const int tx = threadIdx.x % TILE_X, ty = threadIdx.x / TILE_X;
  const long long nxy = (long long)G.nx * G.ny;
  for (long long t = first; t < G.ntiles; t += stride) {
    const int tix = (int)(t % G.ntx);
    const int tiy = (int)((t / G.ntx) % G.nty);
    const int tiz = (int)(t / ((long long)G.ntx * G.nty));
    const int x0 = tix * TILE_X, y0 = tiy * TILE_Y, z0 = tiz * G.tz;
    const int wx = min(TILE_X, G.nx - x0), wy = min(TILE_Y, G.ny - y0), wz = min(G.tz, G.nz - z0);
    if (tx >= wx || ty >= wy) continue;
    const long long col = (long long)(x0 + tx) + (long long)G.nx * (y0 + ty);
    for (int lz = 0; lz < wz; ++lz) {
      const long long m = E3D_IDX(col + nxy * (z0 + lz), ns);
#pragma unroll
      for (int c = 0; c < 3; ++c) u[m + c * ns] = u[m + c * ns] - lam * __ldcg(h + m + c * ns);
    }
  }
}

// ---------------------------------------------------------------------------
// Persistent PCG (dembx_OpenMP main loop, src/elas3dxtal_pcg.f90:1574-2012).
// One cooperative launch runs up to it_limit iterations; every block keeps an
// identical copy of the scalars (each reduces the same partials in the same
// order), so only two grid barriers per iteration are needed:
//   A: h_new = z + gamma*h_old (or z), Ah = K h_new, partial h.Ah   | barrier
//      lambda = gg/hAh (guards :1899-1907)
//   B: u -= lambda h ; g -= lambda Ah ; z = Minv g ; partial z.g     | barrier
//      (FP32 per-thread-load form: u -= lambda h moves into the next A)
//      rel_res, divergence reset (:1961-1981), gamma (:1988), stop test (:2007)
struct PcgState {
  double gg, gg0, rel_res_prev, gamma, rel_res, tol, hAh, gglast;
  double rel_at_replace;  // mixed form: rel_res of the last FP64 residual (set-up or replacement)
  double refine_drop;     // mixed form: replace once rel_res < refine_drop * rel_at_replace (0: never)
  int it, status, reset, resets, cur, max_iter, divergence_reset, refinements;
  // FP32 forms: iterations since the last replacement; fixed-point FP64: 1 where phase A
  // lacks its uneven tiles (pcg_uneven_kernel)
  int since_replace;
  int final_ready;  // the job engine ended on a converged FP64 replacement
};

struct GridBarrier {
  unsigned int count;  // arrivals in the low bits; the top bit flips when all are there
  unsigned int pad;
};

// Barrier among n blocks that run at the same time; `first` is true in exactly one
// of them.  The counting is that of cooperative groups' grid barrier, with a time limit
// and an error exit.  One atomic a block: the first adds 2^31 - (n - 1), the others 1, so that
// the n-th arrival flips the top bit and clears the rest.  Its latency is most of
// an iteration's overhead on small grids: with a generation that the last block
// raises after it has reset the count, and a pause of 128 ns between looks, an
// iteration at 32^3 takes 20.8 us in FP32 and 23.6 in FP64, with this 19.5 and 22.3;
// 64^3 29.0 and 27.0, 121 x 93 x 70 52.2 and 50.6.
// Waits are bounded by a wall-clock limit (globaltimer) and an iteration cap; on
// expiry, or when another block has flagged an error, it returns false and the
// caller exits.
static __device__ bool barrier_among(GridBarrier* gb, unsigned int n, bool first, int* err,
                                     unsigned long long timeout_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    const unsigned int old = atomicAdd(&gb->count, first ? 0x80000000u - (n - 1) : 1u);
    volatile unsigned int* count = &gb->count;
    unsigned long long t0 = 0, spins = 0;
    while (((*count ^ old) & 0x80000000u) == 0u) {
      ++spins;
      if (spins > 64) __nanosleep(64);
      if ((spins & 63ull) == 0ull) {
        if (*(volatile int*)err != DEV_OK) {
          ok = 0;
          break;
        }
        const unsigned long long now = global_timer_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > timeout_ns || spins > (1ull << 34)) {
          atomicExch(err, DEV_TIMEOUT);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
// The same over the whole grid of a cooperative launch.
static __device__ bool grid_barrier(GridBarrier* gb, int* err, unsigned long long timeout_ns) {
  return barrier_among(gb, gridDim.x, blockIdx.x == 0, err, timeout_ns);
}

// Sum of n per-block partials in a fixed order, returned to every thread.
template <int NT = e3d::NT>
static __device__ double reduce_broadcast(const double* partial, int n, double* red) {
  __shared__ double s_val;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += __ldcg(partial + i);
  const double t = block_sum<NT>(s, red);
  if (threadIdx.x == 0) s_val = t;
  __syncthreads();
  return s_val;
}

// Phase B's stages in the per-thread-load persistent kernels.  More take L1 from
// phase A's loads: 500^3 FP32 iteration 5.72 ms with two, 8.0 with four at V = 4.  Odd
// rows (V = 1) gain nothing from four either: 301 x 300 x 300 1.49 ms both, 499 x 500 x
// 500 7.65 with two and 7.69 with four.
constexpr int kPbStages = 2;

// Dynamic shared memory of those kernels: phase B's stages, and in the same bytes
// the fixed-point FP64 tile of phase A.
template <typename T, bool FX, int V>
constexpr int pcg_dyn_smem_bytes() {
  constexpr int b = kPbStages * (int)sizeof(T) *
                    pv_stage<T, FX ? kFxThreads : NT, FX ? kFxRows : TILE_Y, V, sizeof(T) == 8>();
  return FX && b < (int)sizeof(FxSmem<true>) ? (int)sizeof(FxSmem<true>) : b;
}

// T = double: the plain FP64 solve (u is the solution).  T = float: the inner
// loop of the mixed-precision solve (u is the FP32 correction since the last
// FP64 residual replacement; stencil, preconditioner and vectors in FP32, dot
// products and scalar recurrences in FP64).
template <typename T>
struct PcgArgs {
  ApplyArgs<T> A;  // x / hnew / zv / gamma / reset set per iteration
  T* h0;
  T* h1;
  T* u;
  T* g;
  T* z;
  T* Ah;
  const T* minv;
  double* partA;  // [gridDim.x]
  double* partB;  // [gridDim.x]
  PcgState* st;
  double* history;
  GridBarrier* bar;
  int* err;
  int it_limit;
  unsigned long long timeout_ns;
  const PlaneMaps* maps;  // TMA form only
  // fixed-point form only: tables, and the row maxima of z, h0 and h1
  const int4* fxtab;
  int fxkc;
  unsigned* mz;
  unsigned* mh0;
  unsigned* mh1;
  int* fxleave;  // set where a tile needs the FP64 form
  double* partG;  // partial h . A h of those tiles, kUnevenBlocks of them
  int it_end;     // the iteration to stop at
};
constexpr int kUnevenBlocks = 1216;  // eight an SM

// TMA (FP32 only): phase A reads its node planes through the block's plane
// ring (dynamic shared memory of kRingSmemBytes).  FX (FP64 only): phase A in
// fixed point, each tile scaled by its own values.  V: nodes of a row a thread
// takes at a time in phase B, what the rows' alignment allows.
// Where tiles need the FP64 form, phase A ends the launch without them, before anything
// but h_new and A h is written; pcg_uneven_kernel forms them, and the next launch goes
// on with phase B.  In this kernel the FP64 form, in line or called, would leave the
// fixed-point sweep too few registers (300^3: 6.6 ms an iteration instead of 4.5).
template <typename T, bool TMA, bool FX, int V>
__global__ void __launch_bounds__(FX ? kFxThreads : NT,
                                  FX               ? kFxBlocks
                                  : sizeof(T) == 4 ? (TMA && E3D_RING_ZS == 2 ? 1 : E3D_F32_BLOCKS_PER_SM)
                                                   : 1)
    pcg_persistent_kernel(PcgArgs<T> P) {
  constexpr int TY = FX ? kFxRows : TILE_Y, NT = TILE_X * TY;
  static_assert(!TMA || sizeof(T) == 4, "the plane ring feeds the FP32 stencil");
  static_assert(!FX || sizeof(T) == 8, "the fixed-point stencil is the FP64 one");
  using Smem = std::conditional_t<TMA, RingApplySmem<E3D_RING_ZS>, std::conditional_t<FX, char, ApplySmem<T>>>;
  __shared__ Smem sm;
  __shared__ double red[NT / 32];
  __shared__ PcgState S0;
  __shared__ uint64_t ring_bars[E3D_TMA_STAGES];
  __shared__ RingCursor ring_cur;
  PlaneRing ring;
  extern __shared__ __align__(128) unsigned char e3d_pcg_smem[];  // the plane ring, or what pcg_dyn_smem_bytes says
  if constexpr (TMA) ring_setup(ring, e3d_pcg_smem, ring_bars, &ring_cur, P.maps, P.err, P.timeout_ns);
  // The PCG scalars live in shared memory: every thread reads them after a
  // barrier, thread 0 alone updates them (all blocks compute the same values
  // from the same partials), so they hold no registers during the sweeps.
  PcgState& s = S0;
  if (threadIdx.x == 0) s = *P.st;
  __syncthreads();
  if (s.status != PCG_RUNNING) return;
  const bool lead = threadIdx.x == 0;
  const GridDims& G = P.A.g;
  const int it_end = FX ? min(P.it_end, s.max_iter) : min(s.it + P.it_limit, s.max_iter);
  if (FX && s.it >= P.it_end) return;  // launched ahead, and not needed
  bool resume = FX && s.since_replace != 0;  // phase A is done
  constexpr bool kDeferU = sizeof(T) == 4 && !TMA;
  T lam_pending = T(0);  // kDeferU: du -= lam_pending * h_pending not yet applied
  const T* h_pending = nullptr;
  if constexpr (FX) {
    if (!resume) {  // row maxima of the vectors that this launch starts from
      for (long long t = blockIdx.x; t < G.ntiles; t += gridDim.x) {
        const unsigned z = tile_row_max(G, t, P.z);
        const unsigned h = s.reset ? 0u : tile_row_max(G, t, s.cur ? P.h1 : P.h0);
        if (threadIdx.x % TILE_X == 0) {
          const int row = threadIdx.x / TILE_X;
          P.mz[E3D_IDX(t * 2 * TY + row, G.ntiles * 2 * TY)] = z;
          P.mz[E3D_IDX(t * 2 * TY + TY + row, G.ntiles * 2 * TY)] = 0u;
          (s.cur ? P.mh1 : P.mh0)[E3D_IDX(t * TY + row, G.ntiles * TY)] = h;
        }
      }
      if (!grid_barrier(P.bar, P.err, P.timeout_ns)) {
        if (blockIdx.x == 0 && lead) {
          s.status = PCG_TIMEOUT;
          *P.st = s;
        }
        return;
      }
    }
  }
  while (s.it < it_end) {
    const int cur = s.cur;
    if (!resume) {
      // ---- phase A: fused direction update + stencil + h.Ah
      ApplyArgs<T> A = P.A;
      A.x = cur ? P.h1 : P.h0;
      A.hnew = cur ? P.h0 : P.h1;
      A.zv = P.z;
      A.y = P.Ah;
      A.gamma = (T)s.gamma;
      A.reset = s.reset;
      if constexpr (kDeferU) {
        A.du = P.u;
        A.lam_prev = lam_pending;
      }
      double hAh_t = 0.0;
      if constexpr (TMA) ring_begin(ring, G, cur ? P.maps->h1 : P.maps->h0, blockIdx.x, gridDim.x, G.ntiles);
      for (long long t = blockIdx.x; t < G.ntiles; t += gridDim.x) {
        if constexpr (TMA) {
          apply_tile_ring<E3D_RING_ZS>(A, t, sm, hAh_t, ring);
        } else if constexpr (FX) {
          const FxArgs F{P.fxtab, P.fxkc, cur ? P.mh0 : P.mh1};
          const int kx = fx_tile_exponent(G, t, FxRowMaxFused{A.reset ? nullptr : cur ? P.mh1 : P.mh0, P.mz, A.gamma});
          if (kx != kFxGeneral)
            apply_tile_fx<true>(A, F, kx, t, *reinterpret_cast<FxSmem<true>*>(e3d_pcg_smem), hAh_t);
          else if (threadIdx.x < TY) {
            if (lead) *P.fxleave = 1;
            F.mx[E3D_IDX(t * TY + threadIdx.x, G.ntiles * TY)] = 0u;  // raised by pcg_uneven_kernel
          }
        } else {
          apply_tile<T, true, (sizeof(T) == 4 && E3D_F32_POLD_SMEM != 0), kDeferU>(A, t, sm, hAh_t);
        }
        __syncthreads();
      }
      {
        const double bs = block_sum<NT>(hAh_t, red);
        if (threadIdx.x == 0) P.partA[blockIdx.x] = bs;
      }
      if constexpr (TMA) fence_proxy_async_all();  // h_new stores before the next pass's TMA reads
      if (!grid_barrier(P.bar, P.err, P.timeout_ns)) {
        if (lead) s.status = PCG_TIMEOUT;
        break;
      }
      if constexpr (FX) {
        if (__ldcg(P.fxleave)) {
          if (lead) s.since_replace = 1;
          break;
        }
      }
    }
    lam_pending = T(0);  // applied by this phase A
    double hAh = reduce_broadcast<NT>(P.partA, gridDim.x, red);
    if constexpr (FX)
      if (resume) hAh += reduce_broadcast<NT>(P.partG, kUnevenBlocks, red);
    resume = false;
    if (lead) {
      if (FX) s.since_replace = 0;
      s.it += 1;
      s.cur ^= 1;
      s.hAh = hAh;
      if (!isfinite(hAh))
        s.status = PCG_BREAKDOWN;
      else if (fabs(hAh) < 1e-14)  // src/elas3dxtal_pcg.f90:1899-1902
        s.status = PCG_HAH;
    }
    __syncthreads();
    if (s.status != PCG_RUNNING) break;
    const double lambda = s.gg / hAh;
    const T lam = (T)lambda;
    // ---- phase B: u, g update, preconditioner, z.g -- node loop in tile order
    // (no index division); with kDeferU the u update waits for the next phase A.
    const T* hc = cur ? P.h0 : P.h1;  // the h_new of phase A
    double zg_t;
    if constexpr (TMA) {
      zg_t = pcg_update_tiles<T, E3D_PB_UNROLL_RING>(G, blockIdx.x, gridDim.x, lam, hc, P.Ah, P.A.hx, P.A.hy, P.A.hd,
                                                     P.minv, P.u, P.g, P.z);
    } else {
      zg_t = pcg_update_tiles_v<T, NT, TY, V, kPbStages, !kDeferU, FX>(
          G, blockIdx.x, gridDim.x, lam, hc, P.Ah, P.A.hx, P.A.hy, P.A.hd, P.minv, P.u, P.g, P.z,
          reinterpret_cast<T*>(e3d_pcg_smem), threadIdx.x, P.mz);
    }
    if constexpr (kDeferU) {
      lam_pending = lam;
      h_pending = hc;
    }
    {
      const double bs = block_sum<NT>(zg_t, red);
      if (threadIdx.x == 0) P.partB[blockIdx.x] = bs;
    }
    if constexpr (TMA) fence_proxy_async_all();  // z stores before the next pass's TMA reads
    if (!grid_barrier(P.bar, P.err, P.timeout_ns)) {
      if (lead) s.status = PCG_TIMEOUT;
      break;
    }
    const double gg_new = reduce_broadcast<NT>(P.partB, gridDim.x, red);
    if (lead) {
      const double gglast = s.gg;
      s.gg = gg_new;
      s.gglast = gglast;
      if (!isfinite(gg_new)) {
        s.status = PCG_BREAKDOWN;
      } else {
        const double rel_res = sqrt(gg_new / s.gg0);
        s.rel_res = rel_res;
        if (blockIdx.x == 0 && P.history) P.history[E3D_IDX(s.it - 1, s.max_iter)] = rel_res;
        if (s.divergence_reset && rel_res > 10.0 * s.rel_res_prev && s.it > 1) {  // :1961-1981
          s.reset = 1;
          s.resets += 1;
        } else {
          s.gamma = gg_new / gglast;
          s.reset = 0;
        }
        s.rel_res_prev = rel_res;
        if (rel_res < s.tol)
          s.status = PCG_CONVERGED;
        else if (sizeof(T) == 4 && s.refine_drop > 0.0 && rel_res < s.refine_drop * s.rel_at_replace)
          s.status = PCG_REPLACE;  // the host replaces the residual in FP64 and relaunches
      }
    }
    __syncthreads();
    if (s.status != PCG_RUNNING) break;
  }
  __syncthreads();
  if (lead && s.status == PCG_RUNNING && s.it >= s.max_iter) s.status = PCG_MAXITER;
  // The last update is applied by the threads whose phase A wrote those du and
  // h values (same tile and column ownership), so no barrier is needed.
  if constexpr (kDeferU)
    if (lam_pending != T(0)) flush_u_tiles<T>(G, blockIdx.x, gridDim.x, lam_pending, h_pending, P.u);
  if constexpr (TMA) ring_drain(ring);
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.st = s;
}

// The tiles that phase A left out, in the FP64 form, where it did (else nothing): h_new,
// A h, halos, row maxima of h_new and their share of h . A h.  Such tiles are few, so
// each is cut into eight or fewer parts along z, of two planes at least, or the march
// of one tile would be the time of all: a solve of 71 x 58 x 90, uneven for 12 of 140
// iterations, 19.2 ms with whole tiles, 17.9 with these; 16.4 without any such tile.
static __global__ void __launch_bounds__(kFxThreads, kFxBlocks) pcg_uneven_kernel(PcgArgs<double> P) {
  __shared__ ApplySmem<double, kFxRows> sm;
  __shared__ ApplyArgs<double> sA;
  __shared__ double red[kFxThreads / 32];
  const PcgState& s = *P.st;
  if (s.status != PCG_RUNNING || s.since_replace == 0) return;
  const int cur = s.cur;
  if (threadIdx.x == 0) {
    sA = P.A;
    sA.x = cur ? P.h1 : P.h0;
    sA.hnew = cur ? P.h0 : P.h1;
    sA.zv = P.z;
    sA.y = P.Ah;
    sA.gamma = s.gamma;
    sA.reset = s.reset;
  }
  __syncthreads();
  const FxRowMaxFused R{sA.reset ? nullptr : cur ? P.mh1 : P.mh0, P.mz, sA.gamma};
  unsigned* const mx = cur ? P.mh0 : P.mh1;
  const int planes = max(2, (sA.g.tz + 7) / 8), parts = (sA.g.tz + planes - 1) / planes;
  double dot = 0.0;
  for (long long i = blockIdx.x; i < sA.g.ntiles * parts; i += gridDim.x) {
    const long long t = i / parts;
    const int from = (int)(i % parts) * planes;
    if (from >= sA.g.nz - t / ((long long)sA.g.ntx * sA.g.nty) * sA.g.tz) continue;  // the last chunk is shorter
    if (fx_tile_exponent(sA.g, t, R) != kFxGeneral) continue;
    apply_tile<double, true, false, false, kFxRows>(sA, t, sm, dot, from, planes);
    const unsigned v = tile_row_max(sA.g, t, sA.hnew, from, planes);  // the thread's own stores
    if (threadIdx.x % TILE_X == 0)
      atomicMax(mx + E3D_IDX(t * kFxRows + threadIdx.x / TILE_X, sA.g.ntiles * kFxRows), v);
    __syncthreads();
  }
  dot = block_sum<kFxThreads>(dot, red);
  if (threadIdx.x == 0) P.partG[blockIdx.x] = dot;
}

// PCG set-up (src/elas3dxtal_pcg.f90:1527-1567): z = Minv g, partial z.g.
template <typename T>
__global__ void __launch_bounds__(256) pcg_init_kernel(GridDims G, const T* __restrict__ minv,
                                                       const T* __restrict__ g, T* __restrict__ z,
                                                       double* partial) {
  __shared__ double red[8];
  double acc = 0.0;
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < G.ns;
       m += (long long)gridDim.x * blockDim.x) {
    const T gv[3] = {g[m], g[m + G.ns], g[m + 2 * G.ns]};
    T zv[3];
    precond3<T>(minv, m, G.ns, gv, zv);
    for (int c = 0; c < 3; ++c) {
      z[m + c * G.ns] = zv[c];
      acc += (double)zv[c] * (double)gv[c];
    }
  }
  const double s = block_sum<256>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

static __global__ void pcg_init_scalars_kernel(const double* __restrict__ partial, int n, double gg0_ref,
                                        int criterion, float tol, int max_iter, int divergence_reset,
                                        double refine_drop, PcgState* st) {
  __shared__ double red[8];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  const double gg = block_sum<256>(s, red);
  if (threadIdx.x == 0) {
    PcgState S;
    S.gg = gg;
    S.gg0 = (criterion == 1) ? gg : gg0_ref;
    S.rel_res_prev = sqrt(gg / S.gg0);
    S.rel_res = S.rel_res_prev;
    S.gamma = 0.0;
    S.tol = (double)tol;
    S.hAh = 0.0;
    S.gglast = gg;
    S.it = 0;
    S.status = PCG_RUNNING;
    S.reset = 1;  // h = z on the first step (:1554-1562)
    S.resets = 0;
    S.cur = 0;
    S.max_iter = max_iter;
    S.divergence_reset = divergence_reset;
    S.refinements = 0;
    S.since_replace = 0;
    S.final_ready = 0;
    S.rel_at_replace = S.rel_res_prev;
    S.refine_drop = refine_drop;
    *st = S;
  }
}

// ---------------------------------------------------------------------------
// Mixed precision: FP64 residual replacement between FP32 inner chunks.
// u64 += du32 ; du32 = 0 (the inner loop restarts its correction at zero).
static __global__ void fold_correction_kernel(long long n3, const float* __restrict__ du, double* __restrict__ u,
                                       float* __restrict__ du_zero) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  u[i] += (double)du[i];
  du_zero[i] = 0.0f;
}

// g = K u + b from the FP64 stencil (in-tile part + halos), stored in FP64 and
// FP32; then z32 = Minv32 g32 and partial z.g for the replaced residual.
template <int TY>
static __global__ void __launch_bounds__(256) true_residual_kernel(GridDims G, const double* __restrict__ ku,
                                                            const double* __restrict__ hx,
                                                            const double* __restrict__ hy,
                                                            const double* __restrict__ hd,
                                                            const double* __restrict__ b, const float* __restrict__ minv32,
                                                            double* __restrict__ g64, float* __restrict__ g32,
                                                            float* __restrict__ z32, double* partial) {
  __shared__ double red[8];
  double acc = 0.0;
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < G.ns;
       m += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    node_xyz(G, m, x, y, z);
    double v[3] = {ku[m], ku[m + G.ns], ku[m + 2 * G.ns]};
    halo_add<double, TY>(G, hx, hy, hd, x, y, z, v);
    float gv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long i = m + c * G.ns;
      const double gd = v[c] + b[i];
      g64[i] = gd;
      gv[c] = (float)gd;
      g32[i] = gv[c];
    }
    float zv[3];
    precond3<float>(minv32, m, G.ns, gv, zv);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      z32[m + c * G.ns] = zv[c];
      acc += (double)zv[c] * (double)gv[c];
    }
  }
  const double s = block_sum<256>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Scalars after a residual replacement: gg from the true residual, gamma
// re-derived from it (the direction h is kept), and a convergence flag that
// only stands if the true residual also meets the tolerance.
static __global__ void replace_scalars_kernel(const double* __restrict__ partial, int n, PcgState* st,
                                       double* history) {
  __shared__ double red[8];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  const double gg = block_sum<256>(s, red);
  if (threadIdx.x == 0) {
    PcgState S = *st;
    S.gg = gg;
    S.refinements += 1;
    if (S.status == PCG_REPLACE) S.status = PCG_RUNNING;
    if (!isfinite(gg)) {
      S.status = PCG_BREAKDOWN;
    } else {
      const double rel = sqrt(gg / S.gg0);
      S.rel_res = rel;
      S.rel_res_prev = rel;
      S.rel_at_replace = rel;
      if (!S.reset) S.gamma = gg / S.gglast;
      if (history && S.it > 0) history[E3D_IDX(S.it - 1, S.max_iter)] = rel;
      if (S.status == PCG_CONVERGED && !(rel < S.tol)) S.status = PCG_RUNNING;
      if (S.status == PCG_RUNNING && rel < S.tol) S.status = PCG_CONVERGED;
    }
    *st = S;
  }
}

// g32 = (float) g64 at the start of a mixed solve.
static __global__ void to_float_kernel(long long n, const double* __restrict__ a, float* __restrict__ b) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

}  // namespace e3d
