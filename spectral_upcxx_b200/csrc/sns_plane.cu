// K2 + K3 + K4 of the NS step for planes that fit a CTA's shared memory.
//
// On small boxes a step is bound by the latency of its launches: at 32^3 the
// three passes of the xy phase took 4 us each for 0.8 MB of L2-resident data.
// Here one CTA per xy plane keeps the six fields' plane (up to 4096 complex64
// or 2048 complex128 points each) in shared memory from the y-inverse to the
// y-forward: one launch, a read of six fields and a write of three instead of
// 27 field passes.  Steps with it and the carrying update pass against the five
// passes on B200 (complex64): 32 x 32 x 64 12.6 against 22.6 us, 64^3 28.4 against
// 31.0 us, 64 x 64 x 256 82 against 94 us; complex128 32 x 32 x 64 17.7 against 30.2
// us; few large planes leave SMs idle (the line is at plane_least, sns_ns.cu).  At
// 64 x 64 it is bound by issue on the SMs that hold a plane (45 % of
// the slots, one CTA of 24 warps per SM), below by the chain of its five line
// FFTs.
#include "../../include/spectral_b200.h"
#include "sns_common.cuh"
#include "sns_fft.cuh"
#include "sns_fft_core.cuh"
#include "sns_plane.cuh"
#include "sns_tiles.cuh"

namespace sns {
namespace {

// Elements of a line per thread: the fewest with which all six fields of the
// plane are transformed at once by up to the thread limit, else 16 with three
// fields at a time.
template <typename T, int NX, int NY>
struct PlaneShape {
  static constexpr int most = MaxThreads<T>::value;
  static constexpr int E = 6 * NX * NY / 4 <= most ? 4 : 6 * NX * NY / 8 <= most ? 8 : 16;
  static constexpr int P = NX * NY / E;              // threads per field
  static constexpr int FI = 6 * P <= most ? 6 : 3;   // fields at a time
  static constexpr int RS = xrow_stride(NX, (int)sizeof(cx_t<T>), E);
  static constexpr int FS = NY * RS;                 // slots per field
  static constexpr size_t smem = (size_t)6 * FS * sizeof(cx_t<T>);
  using Y = LinePlan<NY, RADIX16_FIRST, E>;
};

// REAL: rows of NX half-spectrum values of real lines of 2 NX points; the x
// lines are pairs of rows (real_pair_load), in the pair's slots.  twx: the table
// of the x lines' length.
template <typename T, int NX, int NY, bool REAL>
__global__ void __launch_bounds__(PlaneShape<T, NX, NY>::FI * PlaneShape<T, NX, NY>::P)
    k_plane_cross(const FieldPtrs f, const cx_t<T>* __restrict__ twx,
                  const cx_t<T>* __restrict__ twy, T scale2) {
  using C = cx_t<T>;
  using SH = PlaneShape<T, NX, NY>;
  constexpr int E = SH::E, P = SH::P, FI = SH::FI, RS = SH::RS, FS = SH::FS;
  constexpr int LX = REAL ? 2 * NX : NX;       // points of an x line
  constexpr int RX = REAL ? 2 * RS : RS;       // slots of an x line
  constexpr int TX = LX / E, TY = SH::Y::TPL;
  static_assert(LinePlan<LX, RADIX16_FIRST, E>::E == E && SH::Y::E == E && TX <= 32, "plane tile");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int fi = threadIdx.x / P, t = threadIdx.x % P;
  const int cx = t % NX, cj = t / NX;  // y lines: adjacent x in adjacent threads
  const int rj = t % TX, ry = t / TX;  // x lines: a line's threads in one warp
  const int64_t col0 = (int64_t)blockIdx.x * NX * NY + cx + (int64_t)cj * NX;
  pdl_trigger();
  pdl_wait();
  C v[E];
  auto column = [&](C* fld) { return fld + pad_pos(cx); };
  auto y_fft = [&](C* fld, T sg) {
    line_fft_at<NY, RADIX16_FIRST, E>(
        v, column(fld), [](int p) { return p * RS; }, cj, twy, sg, [] { __syncthreads(); });
  };
  // y-inverse into the plane
#pragma unroll 1
  for (int f0 = 0; f0 < 6; f0 += FI) {
    const C* __restrict__ src = reinterpret_cast<const C*>(select_ptr(f.in, f0 + fi)) + col0;
    C* fld = sm + (f0 + fi) * FS;
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = src[e * TY * NX];
    y_fft(fld, (T)1);
#pragma unroll
    for (int e = 0; e < E; e++) column(fld)[(cj + TY * e) * RS] = v[e];
  }
  __syncthreads();
  // x-inverse in place
#pragma unroll 1
  for (int f0 = 0; f0 < 6; f0 += FI) {
    C* row = sm + (f0 + fi) * FS + ry * RX;
    if constexpr (REAL)
      real_pair_load<LX>(
          v, rj, [&](int k) { return row[pad_pos(k)]; }, [&](int k) { return row[RS + pad_pos(k)]; });
    else
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = row[pad_pos(rj + TX * e)];
    line_sync<TX>();
    line_fft<LX, false, RADIX16_FIRST, E>(v, row, rj, twx, (T)1);
#pragma unroll
    for (int e = 0; e < E; e++) row[pad_pos(rj + TX * e)] = v[e];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < NX * NY; q += FI * P) {
    C* at = sm + (q / LX) * RX + pad_pos(q % LX);
    C u[3], w[3], c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      u[d] = at[d * FS];
      w[d] = at[(3 + d) * FS];
    }
    cross_point<REAL>(u, w, scale2, c);
#pragma unroll
    for (int d = 0; d < 3; d++) at[d * FS] = c[d];
  }
  __syncthreads();
  // x-forward, then y-forward, of the three products
  C* fld = sm + fi * FS;
  // whole warps of the fields 3..5 skip the x lines
  if (fi < 3 || P % 32 != 0) {
    C* row = fld + ry * RX;
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = row[pad_pos(rj + TX * e)];
    line_sync<TX>();
    line_fft<LX, false, RADIX16_FIRST, E>(v, row, rj, twx, (T)-1);
    if constexpr (REAL) {
      C zn[E / 2];
      real_pair_mirror<LX>(v, zn, row, rj, [] { line_sync<TX>(); });
      line_sync<TX>();
#pragma unroll
      for (int e = 0; e < E / 2; e++)
        real_pair_split(v[e], zn[e], &row[pad_pos(rj + TX * e)], &row[RS + pad_pos(rj + TX * e)]);
    } else {
#pragma unroll
      for (int e = 0; e < E; e++) row[pad_pos(rj + TX * e)] = v[e];
    }
  }
  __syncthreads();
  // every thread takes part in the block barriers of the y lines; those of the
  // fields 3..5 drop their result
#pragma unroll
  for (int e = 0; e < E; e++) v[e] = column(fld)[(cj + TY * e) * RS];
  __syncthreads();
  y_fft(fld, (T)-1);
  if (fi < 3) {
    C* __restrict__ dst = reinterpret_cast<C*>(select_ptr(f.out, fi)) + col0;
#pragma unroll
    for (int e = 0; e < E; e++) dst[e * TY * NX] = v[e];
  }
}

template <typename T, int NX, int NY, bool REAL>
int launch_plane(const FieldPtrs& f, int nz, double scale2, cudaStream_t s) {
  using C = cx_t<T>;
  constexpr int prec = sizeof(T) == 8 ? PREC_C128 : PREC_C64;
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr[dev & 63]) {
    cudaError_t e = allow_max_dynamic_smem(k_plane_cross<T, NX, NY, REAL>);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_plane_cross)");
    attr[dev & 63] = true;
  }
  const C* twx = reinterpret_cast<const C*>(twiddles(REAL ? 2 * NX : NX, prec));
  const C* twy = reinterpret_cast<const C*>(twiddles(NY, prec));
  if (!twx || !twy) {
    set_error("twiddle table allocation failed");
    return ERR_ALLOC;
  }
  cudaError_t e = launch_pdl(k_plane_cross<T, NX, NY, REAL>, dim3(nz),
                             dim3(PlaneShape<T, NX, NY>::FI * PlaneShape<T, NX, NY>::P),
                             PlaneShape<T, NX, NY>::smem, s, f, twx, twy, (T)scale2);
  if (e != cudaSuccess) return cuda_status(e, "k_plane_cross");
  return OK;
}

template <typename T, int NX, int NY>
int plane_as(const FieldPtrs& f, int nz, bool real, double scale2, cudaStream_t s) {
  if constexpr (NX * NY * sizeof(cx_t<T>) <= 4096 * 8) {
    return real ? launch_plane<T, NX, NY, true>(f, nz, scale2, s) : launch_plane<T, NX, NY, false>(f, nz, scale2, s);
  } else {
    set_error("plane pass: the plane does not fit a CTA");
    return ERR_UNSUPPORTED;
  }
}

template <typename T, int NX>
int plane_y(const FieldPtrs& f, int ny, int nz, bool real, double scale2, cudaStream_t s) {
  switch (ny) {
    case 16: return plane_as<T, NX, 16>(f, nz, real, scale2, s);
    case 32: return plane_as<T, NX, 32>(f, nz, real, scale2, s);
    case 64: return plane_as<T, NX, 64>(f, nz, real, scale2, s);
    case 128: return plane_as<T, NX, 128>(f, nz, real, scale2, s);
    default: return plane_as<T, NX, 256>(f, nz, real, scale2, s);
  }
}

template <typename T>
int plane_x(const FieldPtrs& f, int nx, int ny, int nz, bool real, double scale2, cudaStream_t s) {
  switch (nx) {
    case 16: return plane_y<T, 16>(f, ny, nz, real, scale2, s);
    case 32: return plane_y<T, 32>(f, ny, nz, real, scale2, s);
    case 64: return plane_y<T, 64>(f, ny, nz, real, scale2, s);
    case 128: return plane_y<T, 128>(f, ny, nz, real, scale2, s);
    default: return plane_y<T, 256>(f, ny, nz, real, scale2, s);
  }
}

}  // namespace

bool plane_supported(int nx, int ny, int prec) {
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  return is_pow2(nx) && is_pow2(ny) && nx >= 16 && ny >= 16 && nx <= 256 && ny <= 256 &&
         (size_t)nx * ny * esz <= 4096 * 8;
}

int plane_run(void* const in[6], void* const out[3], int nx, int ny, int nz, int prec, bool real,
              double scale2, cudaStream_t s) {
  if (!plane_supported(nx, ny, prec)) {
    set_error("plane pass: the plane does not fit a CTA");
    return ERR_UNSUPPORTED;
  }
  FieldPtrs f{};
  f.n = 6;
  for (int i = 0; i < 6; i++) f.in[i] = in[i];
  for (int i = 0; i < 3; i++) f.out[i] = out[i];
  return prec == PREC_C128 ? plane_x<double>(f, nx, ny, nz, real, scale2, s)
                           : plane_x<float>(f, nx, ny, nz, real, scale2, s);
}

}  // namespace sns
