// Kernels of the Navier-Stokes step's passes and their launchers, one
// instantiation per precision (sns_ns_c64.cu, sns_ns_c128.cu); the plan and the
// step's sequence are in sns_ns.cu.
#pragma once

#include <math.h>
#include <stdlib.h>

#include <algorithm>

#include "sns_fft.cuh"
#include "sns_fft_core.cuh"
#include "sns_ns.cuh"
#include "sns_tiles.cuh"
#include "sns_tma.cuh"

namespace sns {

// ---- limits of the passes' tile forms, as the plan asks them -------------------

// Shared memory of the TMA-staged K3: the stage (6 G rows), 128 bytes of
// alignment slack, the 6 G padded rows of the exchanges and two mbarriers.
inline size_t xcross_tma_smem(int L, int G, size_t esz) {
  return ((size_t)6 * G * L + (size_t)6 * G * xrow_stride(L, (int)esz)) * esz + 128 + 16;
}

// Whether the TMA-staged K3 can run G rows per tile on the (complex) box.
inline bool x_tma_ok(const NSPlan& p, int G) {
  const int TPL = p.nx >= 16 ? p.nx / 16 : 1;
  const size_t esz = p.prec == PREC_C128 ? 16 : 8;
  return !p.real && ((int64_t)p.ny * p.nz) % G == 0 && 6 * G * TPL <= max_threads(p.prec) &&
         xcross_tma_smem(p.nx, G, esz) <= 220 * 1024 && ((size_t)G * p.nx * esz) % 16 == 0;
}

// Shared memory of the TMA-staged K1: S stages of the three components'
// W x G x L tiles, then the 3 W G padded rows of the line FFTs' exchanges,
// 128 bytes of alignment slack and the S + 1 mbarriers.
inline size_t zcurl_tma_smem(int L, int W, int G, int S, size_t esz) {
  return ((size_t)S * 3 * W * G * L + (size_t)3 * W * G * tile_stride(L, W, (int)esz)) * esz +
         128 + 8 * (size_t)(S + 1);
}

// Whether the TMA-staged K1 can run W x G tiles with S stages on the box.
inline bool k1_tma_ok(const NSPlan& p, int W, int G, int S) {
  if (p.nz < 16 || p.nz > 1024) return false;
  const int TPL = p.nz / 16;
  const int esz = p.prec == PREC_C128 ? 16 : 8;
  const int zb = p.nz < 256 ? p.nz : 256;
  return p.nx % W == 0 && p.ny % G == 0 && 3 * W * G * TPL <= max_threads(p.prec) &&
         zcurl_tma_smem(p.nz, W, G, S, esz) <= 220 * 1024 &&
         field_box_ok(p.nx, p.ny, p.nz, esz, W, G, zb);
}

// Shared memory of K5 with K1 carried: 3 W update rows, and 3 W exchange
// rows unless the new velocity is read back from V (reload).
inline size_t update_carry_smem(int L, int W, size_t esz, bool reload, int E = 16) {
  return (size_t)(reload ? 3 : 6) * W * tile_stride(L, W, (int)esz, E) * esz;
}
// Elements per thread of the carrying update pass beside the plane pass: short
// lines of small boxes in shorter chains of more threads (complex64 steps on
// B200: 16^3 10.7 us with 16, 9.6 with 8, 8.3 with 4; 32^3 13.7, 12.4, 12.0).
inline int carry_elems(const NSPlan& p) {
  return !p.plane || p.nz < 16 || p.nz > 64 ? 16 : p.nz <= 32 ? 4 : 8;
}

// Whether K5 with K1 carried can run W-line tiles on the box.
inline bool carry_ok(const NSPlan& p, int W, bool reload) {
  if (W > p.nx || p.nx % W) return false;
  const int E = carry_elems(p);
  const int TPL = p.nz >= E ? p.nz / E : 1;
  const size_t esz = p.prec == PREC_C128 ? 16 : 8;
  return 3 * W * TPL <= max_threads(p.prec) &&
         update_carry_smem(p.nz, W, esz, reload, E) <= 220 * 1024;
}

// Shared memory of the TMA-staged K5: the stage (3 W x L boxes), 128 bytes of
// alignment slack, the 3 W padded rows and two mbarriers.
inline size_t update_tma_smem(int L, int W, size_t esz) {
  return ((size_t)3 * W * L + (size_t)3 * W * tile_stride(L, W, (int)esz)) * esz + 128 + 16;
}

// Whether the TMA-staged K5 can run W-line tiles on the box.
inline bool z_tma_ok(const NSPlan& p, int W) {
  if (p.nz < 16 || p.nz > 1024 || W > p.nx || p.nx % W) return false;
  const int TPL = p.nz / 16;
  const int esz = p.prec == PREC_C128 ? 16 : 8;
  return 3 * W * TPL <= max_threads(p.prec) && update_tma_smem(p.nz, W, esz) <= 220 * 1024 &&
         field_box_ok(p.nx, p.ny, p.nz, esz, W, 1, p.nz < 256 ? p.nz : 256);
}

// ---- the passes at a precision ---------------------------------------------------
template <typename T>
int ns_xcross(const NSPlan& pl, const FieldPtrs& f, int64_t rows, int* err, cudaStream_t s);
template <typename T>
int ns_xcross_real(const NSPlan& pl, const FieldPtrs& f, int64_t rows, cudaStream_t s);
template <typename T>
int ns_zcurl(const NSPlan& pl, const FieldPtrs& f, int* err, cudaStream_t s);
template <typename T, bool SGS>
int ns_update_as(const NSPlan& pl, const UpdateArgs& a, int* err, cudaStream_t s);
template <typename T>
int ns_update_carry(const NSPlan& pl, const UpdateArgs& a, cudaStream_t s);

#ifdef SNS_NS_PASSES

// Largest CTA of the z passes.  Their thread counts are 3 or 9 times a power of
// two, so complex128 ones of up to 512 threads have at most 384, and compiled for
// that they have 168 registers instead of 128: a 384-thread CTA has the SM to
// itself either way, and K1's 100 bytes of spills a thread go (B200, 256^3:
// TMA-staged K1 0.542 -> 0.501 ms, K5 0.706 -> 0.685; 128^3 74.4 -> 68.5 and 95.5
// -> 93.3 us).
template <typename T>
constexpr int kZThreads = sizeof(T) == 8 ? 384 : MaxThreads<T>::value;

// ---------------------------------------------------------------------------
// K3: x lines -- inverse 6 fields, cross product, forward 3 fields.
template <typename T, int L>
__global__ void __launch_bounds__(MaxThreads<T>::value)
    k_xcross(FieldPtrs f, const cx_t<T>* __restrict__ tw, int G, T scale2, int64_t pf, int rev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  pdl_wait();
  xcross_tile<T, L>(ParamFields{f}, tw, G, scale2,
                    tile_order((int64_t)blockIdx.x, (int64_t)gridDim.x, rev), (int)blockDim.x,
                    reinterpret_cast<cx_t<T>*>(smem_raw), pf, (int64_t)gridDim.x);
}

// K3 for CTAs of at most 192 threads, compiled for five resident CTAs per SM
// (64 registers per thread instead of 80): more warps to hide the row loads'
// latency, at the price of a few spilled registers.
template <typename T, int L>
__global__ void __launch_bounds__(192, 5)
    k_xcross_occ(FieldPtrs f, const cx_t<T>* __restrict__ tw, int G, T scale2, int64_t pf, int rev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  pdl_wait();
  xcross_tile<T, L>(ParamFields{f}, tw, G, scale2,
                    tile_order((int64_t)blockIdx.x, (int64_t)gridDim.x, rev), (int)blockDim.x,
                    reinterpret_cast<cx_t<T>*>(smem_raw), pf, (int64_t)gridDim.x);
}

// K3 with TMA-staged tiles: a persistent CTA walks the tiles blockIdx.x,
// + gridDim.x, ...; the G rows of each of the six fields of its next tile (G L
// contiguous elements per field) come into a shared-memory stage as six bulk
// copies on an mbarrier, issued as soon as the current tile's threads have
// read the stage into registers, so the loads overlap the transforms and the
// cross product.  Bounded waits and the stall test as in k_zcurl_tma.
template <typename T, int L>
__global__ void __launch_bounds__(MaxThreads<T>::value)
    k_xcross_tma(FieldPtrs f, const cx_t<T>* __restrict__ tw, int G, T scale2, int64_t ntiles,
                 int rev, int* err, long long stall_cycles) {
  using C = cx_t<T>;
  constexpr int E = LinePlan<L>::E, TPL = LinePlan<L>::TPL;
  constexpr int RS = xrow_stride(L, (int)sizeof(C));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int per = G * L;  // elements of one field's rows of a tile
  const uint32_t raw = tc::smem_u32(smem_raw);
  C* stage = reinterpret_cast<C*>(smem_raw + (((raw + 127u) & ~127u) - raw));
  C* rows = stage + 6 * per;
  uint64_t* full = reinterpret_cast<uint64_t*>(rows + 6 * G * RS);  // stage, stall test
  const int64_t stride = gridDim.x;
  pdl_trigger();
  if (threadIdx.x == 0) {
    tc::mbar_init(&full[0], 1);
    tc::mbar_init(&full[1], 1);
  }
  __syncthreads();
  pdl_wait();  // the rows are written by the y pass before
  auto issue = [&](int64_t blk) {  // thread 0
    const int64_t e0 = tile_order(blk, ntiles, rev) * per;
    if ((tc::smem_u32(stage) & 127u) || ((e0 * (int64_t)sizeof(C)) & 15)) {
      atomicExch(err, 2);
      tma::arrive(&full[0]);
      return;
    }
    tma::expect_tx(&full[0], (uint32_t)(6 * per * sizeof(C)));
#pragma unroll 1
    for (int fl = 0; fl < 6; fl++)
      tma::load_bulk(stage + fl * per, reinterpret_cast<const C*>(select_ptr(f.in, fl)) + e0,
                     (uint32_t)(per * sizeof(C)), &full[0]);
  };
  if (threadIdx.x == 0 && (int64_t)blockIdx.x < ntiles) issue(blockIdx.x);
  int it = 0;
#pragma unroll 1
  for (int64_t blk = blockIdx.x; blk < ntiles; blk += stride, it++) {
    const bool more = blk + stride < ntiles;
    bool ok = tc::mbar_wait(&full[0], (uint32_t)(it & 1), tc::kWaitCycles);
    if (stall_cycles > 0 && it == 0) ok = ok && tc::mbar_wait(&full[1], 0, stall_cycles);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        atomicExch(err, 1);
        tc::mbar_wait(&full[0], (uint32_t)(it & 1), tc::kWaitCycles);
      }
      __syncthreads();
      return;
    }
    xcross_tile_from<T, L>(ParamFields{f}, tw, G, scale2, tile_order(blk, ntiles, rev),
                           (int)blockDim.x, rows,
                           [&](int fld, int gl, int j, C (&v)[E]) {
                             const C* src = stage + fld * per + gl * L + j;
#pragma unroll
                             for (int e = 0; e < E; e++) v[e] = src[TPL * e];
                             // every thread has read the stage: refill it
                             __syncthreads();
                             if (threadIdx.x == 0 && more) {
                               tma::fence_proxy_async();
                               issue(blk + stride);
                             }
                           });
    // the rows are free for the next tile
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// K3 of a real-field run: G pairs of rows of L / 2 half-spectrum values.
template <typename T, int L>
__global__ void __launch_bounds__(384, sizeof(T) == 4 ? 2 : 1)
    k_xcross_real(FieldPtrs f, const cx_t<T>* __restrict__ tw, int G, T scale2, int rev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  pdl_wait();
  xcross_real_tile<T, L>(ParamFields{f}, tw, G, scale2,
                         tile_order((int64_t)blockIdx.x, (int64_t)gridDim.x, rev),
                         (int)blockDim.x, reinterpret_cast<cx_t<T>*>(smem_raw));
}

// ---------------------------------------------------------------------------
// K1: z lines -- inverse of V and of omega = i k x V from one load of V.
template <typename T, int L, bool RELOAD>
__global__ void __launch_bounds__(MaxThreads<T>::value)
    k_zcurl(const LineGeo geo, const FieldPtrs f, const cx_t<T>* __restrict__ tw, int wshift) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  pdl_wait();
  const int64_t blk = tile_order((int64_t)blockIdx.x, (int64_t)gridDim.x, geo.rev);
  if constexpr (RELOAD)
    curl_zpass_tile_reload<T, L>(geo, ParamFields{f}, tw, wshift, blk,
                                 reinterpret_cast<cx_t<T>*>(smem_raw));
  else
    curl_zpass_tile<T, L>(geo, ParamFields{f}, tw, wshift, blk,
                          reinterpret_cast<cx_t<T>*>(smem_raw));
}

// K1 with TMA-staged tiles.  A persistent CTA walks the tiles blockIdx.x,
// blockIdx.x + gridDim.x, ...; the three components of V of a tile come into
// shared memory as TMA boxes (W x G x L elements each, one box per component
// and 256 z planes) while the CTA transforms the tile before it, so the
// HBM reads overlap the line FFTs instead of preceding them.  S = 2: two
// stages, the next tile's load is issued as the current tile starts; S = 1:
// one stage, refilled as soon as the current tile's last read of it is done
// (before its omega transforms).  Every wait on a stage is bounded: a wait
// that runs out sets *err, waits (with the full budget again) for the CTA's
// copies still in flight and ends the CTA.  stall_cycles > 0 is the test of
// that path: the first tile's wait also waits that long on a barrier that
// nothing arrives at.
template <typename T, int L, int S>
__global__ void __launch_bounds__(kZThreads<T>)
    k_zcurl_tma(const __grid_constant__ CUtensorMap m0, const __grid_constant__ CUtensorMap m1,
                const __grid_constant__ CUtensorMap m2, const LineGeo geo, const FieldPtrs f,
                const cx_t<T>* __restrict__ tw, int wshift, int* err, long long stall_cycles) {
  using C = cx_t<T>;
  constexpr int ZB = L < 256 ? L : 256;  // z planes per box
  // the TMA writes to 128-byte aligned shared memory: the stages start at the
  // first 128-byte boundary of the dynamic block (the launch adds the slack),
  // then the rows, then the mbarriers (the stages', then the stall test's)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lines = geo.W * geo.G;
  const int comp = lines * L;  // elements of one component's tile
  const uint32_t raw = tc::smem_u32(smem_raw);
  C* stage0 = reinterpret_cast<C*>(smem_raw + (((raw + 127u) & ~127u) - raw));
  C* rows = stage0 + S * 3 * comp;
  uint64_t* full = reinterpret_cast<uint64_t*>(rows + 3 * lines * tile_stride(L, geo.W, (int)sizeof(C)));
  const int64_t ntiles = geo.TA * geo.TB;
  const int64_t stride = gridDim.x;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int k = 0; k <= S; k++) tc::mbar_init(&full[k], 1);
    tma::prefetch_map(&m0);
    tma::prefetch_map(&m1);
    tma::prefetch_map(&m2);
  }
  __syncthreads();
  // V is written by the step before (its update pass)
  pdl_wait();
  auto issue = [&](int64_t b, int k) {  // thread 0
    const int64_t blk = tile_order(b, ntiles, geo.rev);
    const int u = (int)(sizeof(C) / 8);
    const int x0 = (int)((blk % geo.TA) * geo.W) * u, y0 = (int)((blk / geo.TA) * geo.G);
    C* st = stage0 + k * 3 * comp;
    // self-check of the box (16-byte aligned x, inside the field, 128-byte
    // aligned destination): a bad one is recorded and not loaded, and the
    // stage's barrier is released without it
    if ((x0 & 1) || x0 + geo.W * u > geo.nx * u || y0 + geo.G > geo.ny ||
        (tc::smem_u32(st) & 127u)) {
      atomicExch(err, 2);
      tma::arrive(&full[k]);
      return;
    }
    tma::expect_tx(&full[k], (uint32_t)(3 * comp * sizeof(C)));
#pragma unroll 1
    for (int z0 = 0; z0 < L; z0 += ZB) {
      tma::load_3d(st + z0 * lines, &m0, x0, y0, z0, &full[k]);
      tma::load_3d(st + comp + z0 * lines, &m1, x0, y0, z0, &full[k]);
      tma::load_3d(st + 2 * comp + z0 * lines, &m2, x0, y0, z0, &full[k]);
    }
  };
  const int64_t first = blockIdx.x;
  if (threadIdx.x == 0 && first < ntiles) issue(first, 0);
  int it = 0;
#pragma unroll 1
  for (int64_t blk = first; blk < ntiles; blk += stride, it++) {
    const int k = S == 1 ? 0 : (it & 1);
    const uint32_t par = S == 1 ? (uint32_t)(it & 1) : (uint32_t)((it >> 1) & 1);
    const bool more = blk + stride < ntiles;
    if (S == 2 && threadIdx.x == 0 && more) {
      // stage k ^ 1 was last read by the previous tile, before the barrier
      // that closed it
      tma::fence_proxy_async();
      issue(blk + stride, k ^ 1);
    }
    bool ok = tc::mbar_wait(&full[k], par, tc::kWaitCycles);
    if (stall_cycles > 0 && it == 0) ok = ok && tc::mbar_wait(&full[S], 0, stall_cycles);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        atomicExch(err, 1);
        tc::mbar_wait(&full[k], par, tc::kWaitCycles);
        if (S == 2 && more) tc::mbar_wait(&full[k ^ 1], (uint32_t)(((it + 1) >> 1) & 1), tc::kWaitCycles);
      }
      __syncthreads();
      return;
    }
    curl_zpass_tile_staged<T, L>(geo, ParamFields{f}, tw, wshift,
                                 tile_order(blk, ntiles, geo.rev), stage0 + k * 3 * comp, rows,
                                 [&] {
                                   if (S == 1) {
                                     __syncthreads();
                                     if (threadIdx.x == 0 && more) {
                                       tma::fence_proxy_async();
                                       issue(blk + stride, 0);
                                     }
                                   }
                                 });
    // the stage and the rows are free for the next tile
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// K5: z lines -- forward 3 fields + Nyquist zeroing, then the AB2 /
// projection / CN update per mode.
template <typename T, int L, bool SGS>
__global__ void __launch_bounds__(kZThreads<T>)
    k_zfwd_update(const UpdateArgs a, const cx_t<T>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[4][32];
  pdl_trigger();
  pdl_wait();
  zfwd_update_tile<T, L, SGS>(a, tw, (int64_t)blockIdx.x, (int)blockDim.x,
                              reinterpret_cast<cx_t<T>*>(smem_raw), red);
}

// K5 with the next step's K1 carried in it (zfwd_update_curl_tile): the
// update, then the z-inverse of the new V and of i k x V into a.Uo.
template <typename T, int L, bool RELOAD, int EM = 16>
__global__ void __launch_bounds__(kZThreads<T>)
    k_zfwd_update_curl(const UpdateArgs a, const cx_t<T>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[4][32];
  pdl_trigger();
  pdl_wait();
  zfwd_update_curl_tile<T, L, RELOAD, EM>(a, tw, (int64_t)blockIdx.x, (int)blockDim.x,
                                      reinterpret_cast<cx_t<T>*>(smem_raw), red);
}

// K5 with TMA-staged tiles (plain step, no closure).  A persistent CTA walks
// the tiles blockIdx.x, + gridDim.x, ...; the three components of the cross
// product for a tile (W x L boxes) come into a shared-memory stage by TMA, and
// the next tile's boxes are issued as soon as the current tile's threads have
// read the stage into registers, so they load under the current tile's
// transforms and update.  V and the history are read as before.  The
// diagnostics of each tile go to its own slot of a.stats, as in k_zfwd_update.
// Bounded waits and the stall test as in k_zcurl_tma.
template <typename T, int L>
__global__ void __launch_bounds__(MaxThreads<T>::value)
    k_zfwd_update_tma(const __grid_constant__ CUtensorMap m0, const __grid_constant__ CUtensorMap m1,
                      const __grid_constant__ CUtensorMap m2, const UpdateArgs a,
                      const cx_t<T>* __restrict__ tw, int64_t ntiles, int* err,
                      long long stall_cycles) {
  using C = cx_t<T>;
  constexpr int E = LinePlan<L>::E, TPL = LinePlan<L>::TPL;
  constexpr int ZB = L < 256 ? L : 256;  // z planes per box
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[4][32];
  const int W = a.W;
  const int comp = W * L;  // elements of one component's tile
  const uint32_t raw = tc::smem_u32(smem_raw);
  C* stage = reinterpret_cast<C*>(smem_raw + (((raw + 127u) & ~127u) - raw));
  C* rows = stage + 3 * comp;
  uint64_t* full =
      reinterpret_cast<uint64_t*>(rows + 3 * W * tile_stride(L, W, (int)sizeof(C)));
  const int64_t stride = gridDim.x;
  pdl_trigger();
  if (threadIdx.x == 0) {
    tc::mbar_init(&full[0], 1);
    tc::mbar_init(&full[1], 1);
    tma::prefetch_map(&m0);
    tma::prefetch_map(&m1);
    tma::prefetch_map(&m2);
  }
  __syncthreads();
  pdl_wait();  // the cross product comes from the y pass before
  auto issue = [&](int64_t blk) {  // thread 0
    const int u = (int)(sizeof(C) / 8);
    const int64_t base = blk * W;
    const int x0 = (int)(base & (a.nx - 1)) * u, y0 = (int)(base >> a.lx);
    if ((x0 & 1) || x0 + W * u > a.nx * u || y0 >= a.ny || (tc::smem_u32(stage) & 127u)) {
      atomicExch(err, 2);
      tma::arrive(&full[0]);
      return;
    }
    tma::expect_tx(&full[0], (uint32_t)(3 * comp * sizeof(C)));
#pragma unroll 1
    for (int z0 = 0; z0 < L; z0 += ZB) {
      tma::load_3d(stage + z0 * W, &m0, x0, y0, z0, &full[0]);
      tma::load_3d(stage + comp + z0 * W, &m1, x0, y0, z0, &full[0]);
      tma::load_3d(stage + 2 * comp + z0 * W, &m2, x0, y0, z0, &full[0]);
    }
  };
  if (threadIdx.x == 0 && (int64_t)blockIdx.x < ntiles) issue(blockIdx.x);
  int it = 0;
#pragma unroll 1
  for (int64_t blk = blockIdx.x; blk < ntiles; blk += stride, it++) {
    const bool more = blk + stride < ntiles;
    bool ok = tc::mbar_wait(&full[0], (uint32_t)(it & 1), tc::kWaitCycles);
    if (stall_cycles > 0 && it == 0) ok = ok && tc::mbar_wait(&full[1], 0, stall_cycles);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        atomicExch(err, 1);
        tc::mbar_wait(&full[0], (uint32_t)(it & 1), tc::kWaitCycles);
      }
      __syncthreads();
      return;
    }
    zfwd_update_tile_from<T, L, false>(a, tw, blk, (int)blockDim.x, rows, red,
                                       [&](int fld, int w, int j, C (&v)[E]) {
                                         const C* src = stage + fld * comp + j * W + w;
#pragma unroll
                                         for (int e = 0; e < E; e++) v[e] = src[TPL * e * W];
                                         if (!a.fourier) {
                                           const int64_t nxy = (int64_t)a.nx * a.ny;
                                           ab2_rows<E>(a, fld, blk * W + w + nxy * j, nxy * TPL, v);
                                         }
                                         // every thread has read the stage: refill it
                                         __syncthreads();
                                         if (threadIdx.x == 0 && more) {
                                           tma::fence_proxy_async();
                                           issue(blk + stride);
                                         }
                                       });
    // the rows and the reduction slots are free for the next tile
    __syncthreads();
  }
}

// ---- launchers --------------------------------------------------------------------
namespace {

template <typename T, int L>
int launch_xcross(const NSPlan& pl, const FieldPtrs& f, int64_t rows, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  const int G = pl.xG;
  const int threads = 6 * G * TPL;
  const size_t smem = (size_t)6 * G * xrow_stride(L, (int)sizeof(C)) * sizeof(C);
  if (pl.x_occ && threads <= 192) {
    static bool attr_o[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_o[dev & 63]) {
      cudaError_t e = allow_max_dynamic_smem(k_xcross_occ<T, L>);
      if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_xcross_occ)");
      attr_o[dev & 63] = true;
    }
    const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
      const int64_t pf = tiles_in_waves(k_xcross_occ<T, L>, threads, smem, pl.pf_waves);
    cudaError_t e = launch_pdl(k_xcross_occ<T, L>, dim3((unsigned)(rows / G)), dim3(threads), smem,
                               s, f, tw, G, (T)pl.scale2, pl.rev ? -pf : pf, (int)pl.rev);
    if (e != cudaSuccess) return cuda_status(e, "k_xcross_occ");
    return OK;
  }
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_xcross<T, L>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_xcross)");
    attr[dev & 63] = true;
  }
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  const int blocks = (int)(rows / G);
  const int64_t pf = tiles_in_waves(k_xcross<T, L>, threads, smem, pl.pf_waves);
  cudaError_t e = launch_pdl(k_xcross<T, L>, dim3(blocks), dim3(threads), smem, s, f, tw, G,
                             (T)pl.scale2, pl.rev ? -pf : pf, (int)pl.rev);
  if (e != cudaSuccess) return cuda_status(e, "k_xcross");
  return OK;
}

// Stall test of the TMA-staged passes (SNS_TMA_STALL_TEST=<cycles>; 0: none).
inline long long tma_stall_cycles() {
  const char* e = getenv("SNS_TMA_STALL_TEST");
  const long long v = e ? atoll(e) : 0;
  return v > 0 ? v : 0;
}

template <typename T, int L>
int launch_xcross_tma(const NSPlan& pl, const FieldPtrs& f, int64_t rows, int* err,
                      cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  const int G = pl.xG;
  const int threads = 6 * G * TPL;
  const size_t smem = xcross_tma_smem(L, G, sizeof(C));
  for (int i = 0; i < 6; i++)
    if (reinterpret_cast<uintptr_t>(f.in[i]) & 15) {
      set_error("K3 TMA tile: a field is not 16-byte aligned");
      return ERR_UNSUPPORTED;
    }
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_xcross_tma<T, L>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_xcross_tma)");
    attr[dev & 63] = true;
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_xcross_tma<T, L>,
                                                                threads, smem);
  if (e != cudaSuccess) return cuda_status(e, "occupancy(k_xcross_tma)");
  if (per_sm < 1) {
    set_error("K3 TMA tile: does not fit on an SM");
    return ERR_UNSUPPORTED;
  }
  const int64_t ntiles = rows / G;
  const int blocks = (int)std::min<int64_t>(ntiles, (int64_t)per_sm * sm_count());
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  if (!tw) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  e = launch_pdl(k_xcross_tma<T, L>, dim3((unsigned)blocks), dim3(threads), smem, s, f, tw, G,
                 (T)pl.scale2, ntiles, (int)pl.rev, err, tma_stall_cycles());
  if (e != cudaSuccess) return cuda_status(e, "k_xcross_tma");
  return OK;
}

template <typename T, int L, bool RELOAD>
int launch_zcurl_as(const NSPlan& pl, const FieldPtrs& f, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  LineGeo g{};
  g.L = L;
  g.W = pl.k1W;
  g.G = pl.k1G;
  g.axis = 2;
  g.nx = pl.nx;
  g.ny = pl.ny;
  g.nz = pl.nz;
  g.kx_half = pl.real;
  g.rev = pl.rev;
  g.ps = (int64_t)pl.nx * pl.ny;
  g.gs = pl.nx;
  g.TA = pl.nx / g.W;
  g.TB = pl.ny / g.G;
  g.sa = g.W;
  g.sb = (int64_t)g.G * pl.nx;
  const int threads = 3 * g.W * g.G * TPL;
  const size_t smem =
      (size_t)(RELOAD ? 3 : 6) * g.W * g.G * tile_stride(L, g.W, (int)sizeof(C)) * sizeof(C);
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_zcurl<T, L, RELOAD>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_zcurl)");
    attr[dev & 63] = true;
  }
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  if (!tw) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  int wshift = 0;
  while ((1 << wshift) < g.W) wshift++;
  g.pf = tiles_in_waves(k_zcurl<T, L, RELOAD>, threads, smem, pl.pf_waves);
  if (g.rev) g.pf = -g.pf;
  cudaError_t e = launch_pdl(k_zcurl<T, L, RELOAD>, dim3((unsigned)(g.TA * g.TB)), dim3(threads),
                             smem, s, g, f, tw, wshift);
  if (e != cudaSuccess) return cuda_status(e, "k_zcurl");
  return OK;
}

template <typename T, int L, int S>
int launch_zcurl_tma(const NSPlan& pl, const FieldPtrs& f, int* err, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  constexpr int ZB = L < 256 ? L : 256;
  LineGeo g{};
  g.L = L;
  g.W = pl.k1W;
  g.G = pl.k1G;
  g.axis = 2;
  g.nx = pl.nx;
  g.ny = pl.ny;
  g.nz = pl.nz;
  g.kx_half = pl.real;
  g.rev = pl.rev;
  g.ps = (int64_t)pl.nx * pl.ny;
  g.gs = pl.nx;
  g.TA = pl.nx / g.W;
  g.TB = pl.ny / g.G;
  g.sa = g.W;
  g.sb = (int64_t)g.G * pl.nx;
  const int threads = 3 * g.W * g.G * TPL;
  const size_t smem = zcurl_tma_smem(L, g.W, g.G, S, sizeof(C));
  CUtensorMap m[3];
  for (int d = 0; d < 3; d++) {
    const int rc = field_tensor_map(&m[d], f.in[d], pl.nx, pl.ny, pl.nz, (int)sizeof(C), g.W,
                                    g.G, ZB);
    if (rc) return rc;
  }
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_zcurl_tma<T, L, S>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_zcurl_tma)");
    attr[dev & 63] = true;
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_zcurl_tma<T, L, S>,
                                                                threads, smem);
  if (e != cudaSuccess) return cuda_status(e, "occupancy(k_zcurl_tma)");
  if (per_sm < 1) {
    set_error("K1 TMA tile: does not fit on an SM");
    return ERR_UNSUPPORTED;
  }
  const int64_t ntiles = g.TA * g.TB;
  const int blocks = (int)std::min<int64_t>(ntiles, (int64_t)per_sm * sm_count());
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  if (!tw) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  int wshift = 0;
  while ((1 << wshift) < g.W) wshift++;
  e = launch_pdl(k_zcurl_tma<T, L, S>, dim3((unsigned)blocks), dim3(threads), smem, s, m[0], m[1],
                 m[2], g, f, tw, wshift, err, tma_stall_cycles());
  if (e != cudaSuccess) return cuda_status(e, "k_zcurl_tma");
  return OK;
}

template <typename T, int L>
int launch_zcurl(const NSPlan& pl, const FieldPtrs& f, int* err, cudaStream_t s) {
  if (pl.k1_tma && err)
    return pl.k1_stages == 1 ? launch_zcurl_tma<T, L, 1>(pl, f, err, s)
                             : launch_zcurl_tma<T, L, 2>(pl, f, err, s);
  return pl.k1_reload ? launch_zcurl_as<T, L, true>(pl, f, s)
                      : launch_zcurl_as<T, L, false>(pl, f, s);
}

template <typename T, int L>
int launch_xcross_real(const NSPlan& pl, const FieldPtrs& f, int64_t rows, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  const int G = pl.xG;
  const int threads = 6 * G * TPL;
  const size_t smem = (size_t)6 * G * xrow_stride(L, (int)sizeof(C)) * sizeof(C);
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_xcross_real<T, L>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_xcross_real)");
    attr[dev & 63] = true;
  }
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  if (!tw) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  cudaError_t e = launch_pdl(k_xcross_real<T, L>, dim3((unsigned)(rows / (2 * G))), dim3(threads),
                             smem, s, f, tw, G, (T)pl.scale2, (int)pl.rev);
  if (e != cudaSuccess) return cuda_status(e, "k_xcross_real");
  return OK;
}

template <typename T, int L, bool SGS>
int launch_update(const NSPlan& pl, const UpdateArgs& a, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  constexpr int NF = SGS ? 9 : 3;
  // a tile wider than the thread limit is z-transformed in two halves
  int threads = NF * a.W * TPL;
  if (threads > MaxThreads<T>::value && a.W % 2 == 0) threads /= 2;
  if (threads > MaxThreads<T>::value) {
    set_error("update pass: the tile width does not fit the thread limit");
    return ERR_ARG;
  }
  const size_t smem = (size_t)NF * a.W * tile_stride(L, a.W, (int)sizeof(C)) * sizeof(C);
  const int blocks = (int)(((int64_t)pl.nx * pl.ny) / a.W);
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_zfwd_update<T, L, SGS>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_zfwd_update)");
    attr[dev & 63] = true;
  }
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  UpdateArgs ap = a;
  ap.pf = SGS ? 0 : tiles_in_waves(k_zfwd_update<T, L, SGS>, threads, smem, pl.pf_waves);
  ap.pf_self = SGS ? 0 : pl.z_pfself;
  cudaError_t e = launch_pdl(k_zfwd_update<T, L, SGS>, dim3(blocks), dim3(threads), smem, s, ap,
                             tw);
  if (e != cudaSuccess) return cuda_status(e, "k_zfwd_update");
  return OK;
}

template <typename T, int L, bool RELOAD, int EM = 16>
int launch_update_carry(const NSPlan& pl, const UpdateArgs& a, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L, RADIX16_FIRST, EM>::TPL;
  const int threads = 3 * a.W * TPL;
  const size_t smem = update_carry_smem(L, a.W, sizeof(C), RELOAD, EM);
  const int blocks = (int)(((int64_t)pl.nx * pl.ny) / a.W);
  if (a.W > pl.nx || pl.nx % a.W || threads > MaxThreads<T>::value) {
    set_error("K5 with K1 carried: the tile width does not fit the box");
    return ERR_ARG;
  }
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_zfwd_update_curl<T, L, RELOAD, EM>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_zfwd_update_curl)");
    attr[dev & 63] = true;
  }
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  UpdateArgs ap = a;
  ap.pf = tiles_in_waves(k_zfwd_update_curl<T, L, RELOAD, EM>, threads, smem, pl.pf_waves);
  ap.pf_self = pl.z_pfself;
  cudaError_t e =
      launch_pdl(k_zfwd_update_curl<T, L, RELOAD, EM>, dim3(blocks), dim3(threads), smem, s, ap, tw);
  if (e != cudaSuccess) return cuda_status(e, "k_zfwd_update_curl");
  return OK;
}

template <typename T, int L>
int launch_update_tma(const NSPlan& pl, const UpdateArgs& a, int* err, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int TPL = LinePlan<L>::TPL;
  constexpr int ZB = L < 256 ? L : 256;
  const int threads = 3 * a.W * TPL;
  const size_t smem = update_tma_smem(L, a.W, sizeof(C));
  CUtensorMap m[3];
  for (int d = 0; d < 3; d++) {
    const int rc = field_tensor_map(&m[d], a.U[d], pl.nx, pl.ny, pl.nz, (int)sizeof(C), a.W, 1, ZB);
    if (rc) return rc;
  }
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_zfwd_update_tma<T, L>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_zfwd_update_tma)");
    attr[dev & 63] = true;
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_zfwd_update_tma<T, L>,
                                                                threads, smem);
  if (e != cudaSuccess) return cuda_status(e, "occupancy(k_zfwd_update_tma)");
  if (per_sm < 1) {
    set_error("K5 TMA tile: does not fit on an SM");
    return ERR_UNSUPPORTED;
  }
  const int64_t ntiles = ((int64_t)pl.nx * pl.ny) / a.W;
  const int blocks = (int)std::min<int64_t>(ntiles, (int64_t)per_sm * sm_count());
  const C* tw = reinterpret_cast<const C*>(twiddles(L, sizeof(T) == 8 ? PREC_C128 : PREC_C64));
  if (!tw) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  e = launch_pdl(k_zfwd_update_tma<T, L>, dim3((unsigned)blocks), dim3(threads), smem, s, m[0],
                 m[1], m[2], a, tw, ntiles, err, tma_stall_cycles());
  if (e != cudaSuccess) return cuda_status(e, "k_zfwd_update_tma");
  return OK;
}

}  // namespace

template <typename T>
int ns_xcross_real(const NSPlan& pl, const FieldPtrs& f, int64_t rows, cudaStream_t s) {
  switch (pl.nx_phys) {
    case 32: return launch_xcross_real<T, 32>(pl, f, rows, s);
    case 64: return launch_xcross_real<T, 64>(pl, f, rows, s);
    case 128: return launch_xcross_real<T, 128>(pl, f, rows, s);
    case 256: return launch_xcross_real<T, 256>(pl, f, rows, s);
    case 512: return launch_xcross_real<T, 512>(pl, f, rows, s);
    case 1024: return launch_xcross_real<T, 1024>(pl, f, rows, s);
    default: set_error("real-field NS step: nx must be a power of two in [32, 1024]"); return ERR_UNSUPPORTED;
  }
}

template <typename T>
int ns_zcurl(const NSPlan& pl, const FieldPtrs& f, int* err, cudaStream_t s) {
  switch (pl.nz) {
    case 4: return launch_zcurl<T, 4>(pl, f, err, s);
    case 8: return launch_zcurl<T, 8>(pl, f, err, s);
    case 16: return launch_zcurl<T, 16>(pl, f, err, s);
    case 32: return launch_zcurl<T, 32>(pl, f, err, s);
    case 64: return launch_zcurl<T, 64>(pl, f, err, s);
    case 128: return launch_zcurl<T, 128>(pl, f, err, s);
    case 256: return launch_zcurl<T, 256>(pl, f, err, s);
    case 512: return launch_zcurl<T, 512>(pl, f, err, s);
    case 1024: return launch_zcurl<T, 1024>(pl, f, err, s);
    default: set_error("fused NS step: nz must be a power of two in [4, 1024]"); return ERR_UNSUPPORTED;
  }
}

template <typename T>
int ns_xcross(const NSPlan& pl, const FieldPtrs& f, int64_t rows, int* err, cudaStream_t s) {
  const bool tma = pl.x_tma && err;
  switch (pl.nx) {
#define SNS_XCROSS_CASE(L)                                                                   \
  case L:                                                                                    \
    return tma ? launch_xcross_tma<T, L>(pl, f, rows, err, s) : launch_xcross<T, L>(pl, f, rows, s);
    SNS_XCROSS_CASE(4)
    SNS_XCROSS_CASE(8)
    SNS_XCROSS_CASE(16)
    SNS_XCROSS_CASE(32)
    SNS_XCROSS_CASE(64)
    SNS_XCROSS_CASE(128)
    SNS_XCROSS_CASE(256)
    SNS_XCROSS_CASE(512)
    SNS_XCROSS_CASE(1024)
#undef SNS_XCROSS_CASE
    default: set_error("fused NS step: nx must be a power of two in [4, 1024]"); return ERR_UNSUPPORTED;
  }
}

template <typename T, bool SGS>
int ns_update_as(const NSPlan& pl, const UpdateArgs& a, int* err, cudaStream_t s) {
  const bool tma = !SGS && pl.z_tma && err;
  switch (pl.nz) {
#define SNS_UPDATE_CASE(L)                                                                   \
  case L:                                                                                    \
    if constexpr (L >= 16) {                                                                 \
      if (tma) return launch_update_tma<T, L>(pl, a, err, s);                                \
    }                                                                                        \
    return launch_update<T, L, SGS>(pl, a, s);
    SNS_UPDATE_CASE(4)
    SNS_UPDATE_CASE(8)
    SNS_UPDATE_CASE(16)
    SNS_UPDATE_CASE(32)
    SNS_UPDATE_CASE(64)
    SNS_UPDATE_CASE(128)
    SNS_UPDATE_CASE(256)
    SNS_UPDATE_CASE(512)
    SNS_UPDATE_CASE(1024)
#undef SNS_UPDATE_CASE
    default: set_error("fused NS step: nz must be a power of two in [4, 1024]"); return ERR_UNSUPPORTED;
  }
}

template <typename T>
int ns_update_carry(const NSPlan& pl, const UpdateArgs& a, cudaStream_t s) {
  const bool r = pl.carry_reload;
  switch (pl.nz) {
#define SNS_CARRY_CASE(L)                                                                    \
  case L:                                                                                    \
    if constexpr (L >= 16 && L <= 64) {                                                      \
      constexpr int EM = L <= 32 ? 4 : 8;                                                    \
      if (!r && carry_elems(pl) == EM) return launch_update_carry<T, L, false, EM>(pl, a, s); \
    }                                                                                        \
    return r ? launch_update_carry<T, L, true>(pl, a, s) : launch_update_carry<T, L, false>(pl, a, s);
    SNS_CARRY_CASE(4)
    SNS_CARRY_CASE(8)
    SNS_CARRY_CASE(16)
    SNS_CARRY_CASE(32)
    SNS_CARRY_CASE(64)
    SNS_CARRY_CASE(128)
    SNS_CARRY_CASE(256)
    SNS_CARRY_CASE(512)
    SNS_CARRY_CASE(1024)
#undef SNS_CARRY_CASE
    default: set_error("fused NS step: nz must be a power of two in [4, 1024]"); return ERR_UNSUPPORTED;
  }
}

// Every pass at precision T (once per source file that defines SNS_NS_PASSES).
#define SNS_NS_PASSES_OF(T)                                                                   \
  template int ns_xcross<T>(const NSPlan&, const FieldPtrs&, int64_t, int*, cudaStream_t);    \
  template int ns_xcross_real<T>(const NSPlan&, const FieldPtrs&, int64_t, cudaStream_t);      \
  template int ns_zcurl<T>(const NSPlan&, const FieldPtrs&, int*, cudaStream_t);              \
  template int ns_update_as<T, true>(const NSPlan&, const UpdateArgs&, int*, cudaStream_t);   \
  template int ns_update_as<T, false>(const NSPlan&, const UpdateArgs&, int*, cudaStream_t);  \
  template int ns_update_carry<T>(const NSPlan&, const UpdateArgs&, cudaStream_t);
#endif

}  // namespace sns
