// Tracer particles on the GPU: the move of src/Particle.cpp:12-46 for a whole
// population at once, one thread per particle (exec/ns.cpp:157-203 moves its
// 10000 particles one by one in an OpenMP loop).
//
// A particle at x in [0, 2 pi]^3 takes the cell index ind_d = trunc(x_d / h_d)
// (the reference's INT is uint64_t), h_d = 2 pi / n_d, clamped to n_d - 2 (so
// the upper neighbour is always a grid point, without periodic wrap), the
// fractions rd_d = (x_d - ind_d h_d) / h_d, the trilinear interpolation of the real parts of the three velocity
// components, then x += v K and the wrap x >= 2 pi -> x - 2 pi, x <= 0 ->
// x + 2 pi.  The eight corner terms are summed in the reference's order with
// the reference's left-to-right products, in FP64 without fused multiply-adds,
// so a complex128 velocity gives the reference's positions to the last bit.
//
// The 24 reads of a particle are scattered over the fields.  Where the fields
// exceed L2 each costs a DRAM access that brings 64 bytes or more for the 16 it
// serves: 10^6 particles in a 256^3 complex64 velocity read 1.31 GB from DRAM
// for 0.56 GB asked for, at 73 % of its rate (222 us a move on B200).  Large
// populations are therefore moved in the order of kParticleBins bands of grid
// rows, so that the particles in flight share a part of the fields that stays
// in L2: a counting pass, a pass that lists the particles by band and the move,
// together 157 us (DRAM reads 0.50 GB).  Results do not depend on the order.
#include <math.h>

#include <mutex>

#include "../../include/spectral_b200.h"
#include "sns_common.cuh"
#include "sns_ops.cuh"

namespace sns {
namespace {

// u[{i,j,k}] * w0 * w1 * w2, evaluated as ((u * w0) * w1) * w2
__device__ __forceinline__ double term(double u, double w0, double w1, double w2) {
  return __dmul_rn(__dmul_rn(__dmul_rn(u, w0), w1), w2);
}

constexpr int kParticleBins = 64;
constexpr int kBinThreads = 256, kBinPer = 8;  // particles per thread of the binning passes

// Band of grid rows (y fastest, then z) that a particle reads, for the order of
// the moves only.
__device__ __forceinline__ int particle_bin(const double* __restrict__ loc, int64_t p, float sy,
                                            float sz, int ny, int nz) {
  const int j = min(max((int)((float)loc[3 * p + 1] * sy), 0), ny - 1);
  const int k = min(max((int)((float)loc[3 * p + 2] * sz), 0), nz - 1);
  return (int)((((int64_t)k * ny + j) * kParticleBins) / ((int64_t)ny * nz));
}

// LIST = false: adds each band's count to counts[band].  LIST = true: counts
// holds them; `cursor` (zero) hands out each band's places, and order receives
// the particles band by band.
template <bool LIST>
__global__ void __launch_bounds__(kBinThreads)
    k_particles_bin(const double* __restrict__ loc, int64_t np, float sy, float sz, int ny, int nz,
                    int* __restrict__ counts, int* __restrict__ cursor, int* __restrict__ order) {
  __shared__ int local[kParticleBins], place[kParticleBins];
  const int t = threadIdx.x;
  if (t < kParticleBins) local[t] = 0;
  __syncthreads();
  const int64_t p0 = (int64_t)blockIdx.x * (kBinThreads * kBinPer) + t;
  int bin[kBinPer], rank[kBinPer];
#pragma unroll
  for (int i = 0; i < kBinPer; i++) {
    const int64_t p = p0 + i * kBinThreads;
    bin[i] = p < np ? particle_bin(loc, p, sy, sz, ny, nz) : -1;
    if (bin[i] >= 0) rank[i] = atomicAdd(&local[bin[i]], 1);
  }
  __syncthreads();
  if constexpr (!LIST) {
    if (t < kParticleBins && local[t]) atomicAdd(&counts[t], local[t]);
  } else {
    if (t < kParticleBins) {
      int base = 0;
      for (int b = 0; b < t; b++) base += counts[b];
      place[t] = base + (local[t] ? atomicAdd(&cursor[t], local[t]) : 0);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kBinPer; i++)
      if (bin[i] >= 0) order[place[bin[i]] + rank[i]] = (int)(p0 + i * kBinThreads);
  }
}

// order: the particles in the order of the moves (null: as they are).
// Three blocks of 256 per SM: room for a particle's reads in flight (85
// registers).  B200, ordered: 138 us a move against 151 with four blocks, 179
// with five (spills), 140 with two.
template <typename T>
__global__ void __launch_bounds__(256, 3) k_particles_move(double* __restrict__ loc, double* __restrict__ vel, int64_t np,
                                 const int* __restrict__ order,
                                 const cx_t<T>* __restrict__ u0, const cx_t<T>* __restrict__ u1,
                                 const cx_t<T>* __restrict__ u2, int64_t nx, int64_t ny,
                                 int64_t nz, double K) {
  const double two_pi = 2 * M_PI;
  const int64_t nxy = nx * ny;
  const int64_t dims[3] = {nx, ny, nz};
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < np;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = order ? order[q] : q;
    double x[3], rd[3], om[3];
    int64_t ind[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      x[d] = loc[3 * p + d];
      const double h = __ddiv_rn(two_pi, (double)dims[d]);
      ind[d] = (int64_t)__ddiv_rn(x[d], h);
      if (ind[d] >= dims[d] - 1) ind[d] = dims[d] - 2;
      // a position outside [0, 2 pi] (never produced by the wrap from inside)
      // is clamped to the first cell instead of indexing out of the field
      if (ind[d] < 0) ind[d] = 0;
      rd[d] = __ddiv_rn(__dsub_rn(x[d], __dmul_rn((double)ind[d], h)), h);
      om[d] = __dsub_rn(1.0, rd[d]);
    }
    // all 24 reads in flight before the first is used; corners in the order of
    // src/Particle.cpp:27-34
    const int64_t at = ind[0] + nx * ind[1] + nxy * ind[2];
    const int64_t c[8] = {0, 1, 1 + nx, nx, nxy, 1 + nxy, 1 + nx + nxy, nx + nxy};
    T w[3][8];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const cx_t<T>* __restrict__ u = (d == 0 ? u0 : d == 1 ? u1 : u2) + at;
#pragma unroll
      for (int q = 0; q < 8; q++) w[d][q] = u[c[q]].x;
    }
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double s = term((double)w[d][0], om[0], om[1], om[2]);
      s = __dadd_rn(s, term((double)w[d][1], rd[0], om[1], om[2]));
      s = __dadd_rn(s, term((double)w[d][2], rd[0], rd[1], om[2]));
      s = __dadd_rn(s, term((double)w[d][3], om[0], rd[1], om[2]));
      s = __dadd_rn(s, term((double)w[d][4], om[0], om[1], rd[2]));
      s = __dadd_rn(s, term((double)w[d][5], rd[0], om[1], rd[2]));
      s = __dadd_rn(s, term((double)w[d][6], rd[0], rd[1], rd[2]));
      s = __dadd_rn(s, term((double)w[d][7], om[0], rd[1], rd[2]));
      v[d] = s;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double y = __dadd_rn(x[d], __dmul_rn(v[d], K));
      if (y >= two_pi)
        y = __dsub_rn(y, two_pi);
      else if (y <= 0)
        y = __dadd_rn(two_pi, y);
      loc[3 * p + d] = y;
      if (vel) vel[3 * p + d] = v[d];
    }
  }
}

// Workspace of one call, ordered on its stream: from a memory pool of this file's
// own per device, which keeps at most 64 MB between calls (sns_pool_trim gives
// them back).
std::mutex mu;
cudaMemPool_t pools[64] = {};

void* workspace(size_t bytes, cudaStream_t s) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  cudaMemPool_t pool;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) {
        cudaGetLastError();
        pools[dev] = nullptr;
        return nullptr;
      }
      uint64_t keep = 64ull << 20;
      cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
    pool = pools[dev];
  }
  void* p = nullptr;
  if (cudaMallocFromPoolAsync(&p, bytes, pool, s) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

// Populations worth ordering: fields well beyond L2, and particles enough that
// several share what a DRAM access brings and the two passes over them pay.
// B200, a move in us as they are / ordered, by MB of the fields: 131 (176^3
// complex64) 1M 127 / 133, 2.5M 314 / 330; 170 (192^3) 550k 88 / 90, 700k 109 / 105,
// 1M 152 / 137; 262 (176^3 complex128) 400k 86 / 90, 550k 115 / 106; 403 (256^3) 300k
// 74 / 83, 550k 127 / 116, 1M 226 / 167; 805 (256^3 complex128) 300k 92 / 102, 550k
// 153 / 152, 1M 272 / 226; 1359 (384^3) 1M 277 / 249.  Not under stream capture (a
// graph would own the workspace).
bool ordered(int64_t np, int64_t n, size_t esz, cudaStream_t s) {
  const double bytes = 3.0 * esz * n;
  if (bytes < 165e6 || np < (bytes < 250e6 ? 700000 : 550000) || np > 0x7fffffff || np * 64 < n)
    return false;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return st == cudaStreamCaptureStatusNone;
}

}  // namespace

void particles_trim() {
  std::lock_guard<std::mutex> lock(mu);
  for (cudaMemPool_t p : pools)
    if (p) cudaMemPoolTrimTo(p, 0);
}

}  // namespace sns

using namespace sns;

extern "C" int sns_particles_move(double* loc, double* vel, int64_t np, const void* const u[3],
                                  int64_t nx, int64_t ny, int64_t nz, int prec, double K,
                                  void* stream) {
  if (np < 0 || (np > 0 && (!loc || !u || !u[0] || !u[1] || !u[2]))) {
    set_error("sns_particles_move: null pointer or negative count");
    return ERR_ARG;
  }
  if (nx < 2 || ny < 2 || nz < 2) {
    set_error("sns_particles_move: every dimension must be at least 2");
    return ERR_ARG;
  }
  if (prec != PREC_C64 && prec != PREC_C128) {
    set_error("sns_particles_move: unknown precision");
    return ERR_ARG;
  }
  if (np == 0) return OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  int* work = nullptr;
  const int* order = nullptr;
  if (ordered(np, nx * ny * nz, esz, s))
    work = static_cast<int*>(workspace(sizeof(int) * (2 * kParticleBins + (size_t)np), s));
  if (work) {
    int* counts = work;
    int* cursor = work + kParticleBins;
    int* list = work + 2 * kParticleBins;
    int rc = cuda_status(cudaMemsetAsync(work, 0, sizeof(int) * 2 * kParticleBins, s),
                         "sns_particles_move");
    const float sy = (float)((double)ny / (2 * M_PI)), sz = (float)((double)nz / (2 * M_PI));
    const unsigned blocks = (unsigned)((np + kBinThreads * kBinPer - 1) / (kBinThreads * kBinPer));
    if (!rc) {
      k_particles_bin<false><<<blocks, kBinThreads, 0, s>>>(loc, np, sy, sz, (int)ny, (int)nz,
                                                            counts, cursor, list);
      k_particles_bin<true><<<blocks, kBinThreads, 0, s>>>(loc, np, sy, sz, (int)ny, (int)nz,
                                                           counts, cursor, list);
      rc = cuda_status(cudaGetLastError(), "k_particles_bin");
    }
    if (rc) {
      cudaFreeAsync(work, s);
      return rc;
    }
    order = list;
  }
  const int threads = 256;
  const int64_t want = (np + threads - 1) / threads;
  const unsigned blocks = (unsigned)(want < 0x7fffffff ? want : 0x7fffffff);
  if (prec == PREC_C128)
    k_particles_move<double><<<blocks, threads, 0, s>>>(
        loc, vel, np, order, reinterpret_cast<const double2*>(u[0]),
        reinterpret_cast<const double2*>(u[1]), reinterpret_cast<const double2*>(u[2]), nx, ny, nz,
        K);
  else
    k_particles_move<float><<<blocks, threads, 0, s>>>(
        loc, vel, np, order, reinterpret_cast<const float2*>(u[0]),
        reinterpret_cast<const float2*>(u[1]), reinterpret_cast<const float2*>(u[2]), nx, ny, nz,
        K);
  const cudaError_t e = cudaGetLastError();
  if (work) cudaFreeAsync(work, s);
  if (e != cudaSuccess) return cuda_status(e, "k_particles_move");
  return OK;
}
