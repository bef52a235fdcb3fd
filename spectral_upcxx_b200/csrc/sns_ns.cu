// Fused pseudo-spectral Navier-Stokes step (exec/ns.cpp:167-217).
//
// State: V (Fourier velocity, 3 fields) and C0 (V x omega of the previous step,
// 3 fields); work: U (6 fields).  One step is five passes:
//
//   K1  z-inverse of (V, i k x V): the curl is formed while the tile loads
//       (ns.cpp:206 + Vector::cross's inverse copies, src/Vector.cpp:74-77)
//   K2  y-inverse of the 6 fields
//   K3  x-inverse, 1/N^2-scaled complex cross product u x omega, x-forward
//       (src/Vector.cpp:79-89), 6 fields in, 3 out
//   K4  y-forward of the 3 fields
//   K5  z-forward of 3 cross1 - cross0 + Nyquist zeroing, then per mode the AB2 /
//       projection / Crank-Nicolson update (ns.cpp:170-187) written over V, FP64
//       diagnostics (ns.cpp:206-210)
//
// The history cross0 is kept as K4 left it, before its z-forward (the transform
// is linear), so K5 reads nine fields and writes three: cross1 is neither
// transformed on its own nor written.  U[0..2] and C0 take turns as the place
// where a step builds its cross product and where its history is (HIST_Z_*);
// a state that was just set has its Fourier history in C0.
//
// The reference runs 9 separate 3D FFTs plus ~25 eager field sweeps and 15
// deep copies per step; here the history copies (ns.cpp:213-217) are
// in-place updates and every intermediate lives in U.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <set>
#include <tuple>
#include <vector>

#include "sns_fft.cuh"
#include "sns_ns.cuh"
#include "sns_ns_passes.cuh"
#include "sns_ops.cuh"
#include "sns_tiles.cuh"

namespace sns {

__global__ void k_stats_final(const double* part, int blocks, double* out) {
  __shared__ double sm[4][256];
  double a = 0, b = 0, c = 0, m = 0;
  for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
    a += part[4 * i];
    b += part[4 * i + 1];
    c += part[4 * i + 2];
    m = fmax(m, part[4 * i + 3]);
  }
  sm[0][threadIdx.x] = a;
  sm[1][threadIdx.x] = b;
  sm[2][threadIdx.x] = c;
  sm[3][threadIdx.x] = m;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sm[0][threadIdx.x] += sm[0][threadIdx.x + o];
      sm[1][threadIdx.x] += sm[1][threadIdx.x + o];
      sm[2][threadIdx.x] += sm[2][threadIdx.x + o];
      sm[3][threadIdx.x] = fmax(sm[3][threadIdx.x], sm[3][threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; k++) out[k] = sm[k][0];
}

// ---------------------------------------------------------------------------
// host side

namespace {

// K3 of the plan: complex rows, or half-spectrum rows of a real-field run
int xpass(const NSPlan& pl, const FieldPtrs& f, int64_t rows, int* err, cudaStream_t s) {
  if (pl.real)
    return pl.prec == PREC_C128 ? ns_xcross_real<double>(pl, f, rows, s)
                                : ns_xcross_real<float>(pl, f, rows, s);
  return pl.prec == PREC_C128 ? ns_xcross<double>(pl, f, rows, err, s)
                              : ns_xcross<float>(pl, f, rows, err, s);
}

int elems(int L) { return L >= 16 ? 16 : L; }

constexpr double kL2Bytes = 126e6;  // L2 of the B200

// K3 tile: G rows of all six fields, in CTAs of at most 192 threads
// (complex64) or 96 (complex128): small CTAs drift apart, so one CTA's loads
// run under another's transforms.  B200, 256^3: complex64 0.266 ms with 192
// threads, 0.283 with 96 and with 384; complex128 0.598 with 96, 0.614 with
// 192, 0.737 with 384.
int x_tile_rows(int nx, int64_t rows, int prec) {
  const int TPL = nx / elems(nx);
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  int G = 1;
  while (6 * (G * 2) * TPL <= (prec == PREC_C128 ? 96 : 192) && rows % (G * 2) == 0 &&
         (size_t)6 * G * 2 * xrow_stride(nx, (int)esz) * esz <= 110 * 1024)
    G *= 2;
  return G;
}

// Planes from which one CTA per plane is the faster xy phase.  Planes of up to
// 16 KB a field: always.  Larger ones take an SM each, for a time that depends on
// the plane alone, so few of them leave most SMs idle.  Whole steps on B200 in us,
// five passes / plane: complex64 64 x 64 by planes 16 19.5 / 22.8, 32 24.4 / 25.4,
// 64 31.0 / 28.4, 256 94 / 82, 1024 711 / 497; 16 x 256 by 4 18.5 / 19.2, 16 22.5 /
// 20.3; real rows of 256 by 32 64 30.7 / 32.6, 128 47.0 / 40.7; complex128 64 x 32 by
// 8 19.8 / 22.6, 16 22.9 / 22.3, 32 29.5 / 24.6 (real 16 23.1 / 24.6, 32 30.0 / 26.8).
// (Beyond, the plane form stays ahead or within 4 %.)
int plane_least(int nx, int ny, int prec, bool real) {
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  if ((size_t)nx * ny * esz <= 16 * 1024) return 0;
  if (prec == PREC_C128) return real ? 32 : 16;
  return real ? std::min(2 * nx, 128) : std::min(nx, 64);
}

// Whether the xy phase runs as one CTA per plane: where the plane fits and there
// are planes enough (SNS_PLANE=0: never, 1: wherever it fits), unless a form of the
// separate passes is asked for.
bool plane_wanted(int nx, int ny, int nz, int prec, bool real) {
  const char* e = getenv("SNS_PLANE");
  if (e && e[0] == '0') return false;
  if (!(e && e[0] == '1') && nz < plane_least(nx, ny, prec, real)) return false;
  for (const char* v : {"SNS_K1_TMA", "SNS_K1_RELOAD", "SNS_K1_SPLIT", "SNS_K1_LINES",
                        "SNS_K1_SMEM_KB", "SNS_X_TMA", "SNS_X_OCC", "SNS_Y_TMA", "SNS_LINE_W",
                        "SNS_RADIX_ORDER", "SNS_Z_TMA", "SNS_Z_W", "SNS_Z_PFSELF", "SNS_CARRY",
                        "SNS_PF", "SNS_XY_PASSES", "SNS_XY_CHUNK", "SNS_XYC"})
    if (getenv(v)) return false;
  return plane_supported(nx, ny, prec);
}

}  // namespace

int cross_xpass(void* const in[6], void* const out[3], int nx, int ny, int nz, int prec,
                double scale2, cudaStream_t s) {
  NSPlan pl{};
  pl.nx = pl.nx_phys = nx;
  pl.ny = ny;
  pl.nz = nz;
  pl.prec = prec;
  pl.scale2 = scale2;
  pl.xG = x_tile_rows(nx, (int64_t)ny * nz, prec);
  pl.rev = true;
  FieldPtrs f{};
  f.n = 6;
  for (int i = 0; i < 6; i++) f.in[i] = in[i];
  for (int i = 0; i < 3; i++) f.out[i] = out[i];
  return xpass(pl, f, (int64_t)ny * nz, nullptr, s);
}

bool ns_fits_l2(const NSPlan& p) {
  const double esz = p.prec == PREC_C128 ? 16 : 8;
  return 12.0 * esz * p.nx * p.ny * p.nz <= kL2Bytes;
}

int ns_plan(NSPlan& pl, int nx, int ny, int nz, int prec, int zW, int lineW, bool real,
            bool separate) {
  pl = NSPlan{};
  pl.real = real;
  pl.nx_phys = nx;
  if (real) {
    // half spectrum: kx = 0 .. nx/2-1 stored (the kx = nx/2 plane is zero)
    if (!is_pow2(nx) || nx < 32 || nx > 1024) {
      set_error("real-field NS step: nx must be a power of two in [32, 1024]");
      return ERR_UNSUPPORTED;
    }
    nx /= 2;
  }
  pl.nx = nx;
  pl.ny = ny;
  pl.nz = nz;
  pl.prec = prec;
  for (int n : {nx, ny, nz})
    if (!is_pow2(n) || n < 4 || n > 1024) {
      set_error("fused NS step: dimensions must be powers of two in [4, 1024]");
      return ERR_UNSUPPORTED;
    }
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  // fields beyond L2: the step streams from HBM
  const bool big = !ns_fits_l2(pl);
  {
    // (a real-field run: pairs of rows, as lines of the physical nx)
    const int TPL = pl.nx_phys / elems(pl.nx_phys);
    const int G = x_tile_rows(pl.nx_phys, (int64_t)ny * nz / (real ? 2 : 1), prec);
    pl.scale2 = 1.0 / (((double)pl.nx_phys * ny * nz) * ((double)pl.nx_phys * ny * nz));
    if (6 * G * TPL > max_threads(prec)) {
      set_error("fused NS step: nx too large for the x-pass tile");
      return ERR_UNSUPPORTED;
    }
    pl.xG = G;
    // the TMA-staged form on request (SNS_X_TMA=1), with the widest tile up
    // to G that fits its stage.  Measured on B200 at 256^3 it does not pay:
    // complex64 0.315 ms against 0.284 (G = 4) and 0.262 (G = 2, direct);
    // complex128 0.700 against 0.756 (G = 4) and 0.599 (G = 1, direct): the
    // rows are contiguous, so direct loads already stream, and the stage
    // halves the CTAs an SM holds.  The tuner still tries it.
    // the five-CTA form of the direct-load pass on request (SNS_X_OCC=1)
    const char* eo = getenv("SNS_X_OCC");
    pl.x_occ = eo && eo[0] == '1';
    const char* e = getenv("SNS_X_TMA");
    pl.x_tma = false;
    if (e && e[0] == '1')
      for (int g = G; g >= 1 && !pl.x_tma; g /= 2)
        if (x_tma_ok(pl, g)) {
          pl.x_tma = true;
          pl.xG = g;
        }
  }
  // K1 tile: W adjacent z lines x G groups of the three components, one
  // CTA for all six outputs (SNS_K1_SPLIT=1: one output field per CTA)
  {
    // 16 adjacent lines keep the half-warps of the exchanges on distinct banks;
    // the two row sets of a 16-line tile take 210 KB at 256 (opt-in limit 227 KB)
    // Two CTAs per SM (112 KB each), so that one CTA's loads overlap the
    // other's transforms; tile_stride keeps narrower runs free of bank
    // conflicts.  SNS_K1_SMEM_KB overrides the cap (220: one CTA per SM).
    const int TPL = nz / elems(nz);
    const int cap = max_threads(prec);
    size_t smem_cap = 112 * 1024;
    if (const char* e = getenv("SNS_K1_SMEM_KB")) {
      const int v = atoi(e);
      if (v >= 16 && v <= 220) smem_cap = (size_t)v * 1024;
    }
    int W = 1;
    const int Wmax = prec == PREC_C128 ? 8 : 16;
    while (W * 2 <= Wmax && nx % (W * 2) == 0 && 3 * (W * 2) * TPL <= cap &&
           (size_t)6 * (W * 2) * tile_stride(nz, W * 2, (int)esz) * esz <= smem_cap)
      W *= 2;
    int G = 1;
    while (ny % (G * 2) == 0 && 3 * W * (G * 2) * TPL <= 384 &&
           (size_t)6 * W * (G * 2) * tile_stride(nz, W, (int)esz) * esz <= smem_cap)
      G *= 2;
    pl.k1W = W;
    pl.k1G = G;
    const char* e = getenv("SNS_K1_SPLIT");
    pl.k1_fused = !(e && e[0] == '1') && 3 * W * G * TPL <= cap &&
                  (size_t)6 * W * G * tile_stride(nz, W, (int)esz) * esz <= smem_cap;
  }
  // K5 tile: W adjacent z lines of three fields
  {
    const int TPL = nz / elems(nz);
    int W = 1;
    int Wmax = prec == PREC_C128 ? 8 : 16;
    if (zW > 0) Wmax = zW;  // a tuned width
    // tile width override for tuning sweeps (SNS_Z_W, a power of two; a
    // width beyond the thread limit is transformed in two halves, with one
    // CTA per SM)
    bool wide = false;
    if (const char* e = zW > 0 ? nullptr : getenv("SNS_Z_W")) {
      const int v = atoi(e);
      if (v >= 1 && (v & (v - 1)) == 0) Wmax = v;
      wide = true;
    }
    while (W * 2 <= Wmax && nx % (W * 2) == 0 &&
           3 * (W * 2) * TPL <= (wide ? 2 : 1) * max_threads(prec) &&
           (size_t)3 * W * 2 * tile_stride(nz, W * 2, (int)esz) * esz <= (wide ? 220 : 110) * 1024)
      W *= 2;
    pl.zW = W;
    pl.update_blocks = (nx / W) * ny;
    // the TMA-staged form on request (SNS_Z_TMA=1), the widest tile up to W
    // that fits its stage.  Measured on B200 at 256^3 it does not pay: complex64
    // 0.500 ms (W = 16) and 0.657 (W = 8) against 0.435 direct; complex128
    // 1.159 (W = 8) against 1.016.  The cross product is only a third of the
    // pass's reads (the history joins as its lines load, V in the update), the stage
    // and the rows fill
    // the SM's shared memory at one CTA, and the persistent tiles add two
    // barriers each.  The tuner still tries it.
    const char* ez = getenv("SNS_Z_TMA");
    pl.z_tma = false;
    if (ez && ez[0] == '1')
      for (int w = W; w >= 1 && !pl.z_tma; w /= 2)
        if (z_tma_ok(pl, w)) {
          pl.z_tma = true;
          pl.zW = w;
          pl.update_blocks = (nx / w) * ny;
        }
    // K1 carried in the update pass on request (SNS_CARRY=1), at the widest
    // tile up to W whose update and exchange rows fit two CTAs per SM
    // (SNS_CARRY=2: the new velocity read back from V, K5's shared memory)
    const char* ecr = getenv("SNS_CARRY");
    pl.carry = false;
    pl.carry_reload = ecr && ecr[0] == '2';
    if (ecr && (ecr[0] == '1' || ecr[0] == '2'))
      for (int w = W; w >= 1 && !pl.carry; w /= 2)
        if (carry_ok(pl, w, pl.carry_reload) &&
            update_carry_smem(nz, w, esz, pl.carry_reload) <= 110 * 1024) {
          pl.carry = true;
          pl.z_tma = false;
          pl.zW = w;
          pl.update_blocks = (nx / w) * ny;
        }
    // L2 prefetch of each tile's V once its cross product and history have been
    // loaded (asked before those loads it delayed them), where it comes from HBM
    // (SNS_Z_PFSELF = 0, 1).  B200, 256^3: complex64 0.369 ms against 0.408
    // without, complex128 0.686 against 0.784.
    const char* epf = getenv("SNS_Z_PFSELF");
    pl.z_pfself = epf ? epf[0] == '1' : big;
    // closure update: nine fields in the tile
    const int cap = std::min(576, max_threads(prec));
    int Ws = 1;
    while (Ws * 2 <= Wmax && ((int64_t)nx * ny) % (Ws * 2) == 0 && 9 * (Ws * 2) * TPL <= cap &&
           (size_t)9 * Ws * 2 * tile_stride(nz, Ws * 2, (int)esz) * esz <= 110 * 1024)
      Ws *= 2;
    pl.sgs_W = Ws;
    pl.sgs_blocks = (int)(((int64_t)nx * ny) / Ws);
  }
  // xy phase: three separate full-domain passes by default.  Two fused forms
  // move a third of their HBM bytes but measured slower on B200, the passes
  // being bound by latency and issue rather than bytes: SNS_XYC=1 selects one
  // thread-block-cluster pass over each plane (sns_xyc.cu; nx = ny = 128, or
  // 256 in complex64; 1.28 vs 0.69 ms at 256^3), SNS_XY_PASSES=1 the
  // persistent dataflow launch through L2 (sns_xy.cu; 1.13 vs 0.69 ms).
  // K1 walks its tiles back from where K5 ended (both follow the xy plane),
  // K3 back from where K2 ended (both follow z).  B200, whole complex64 step:
  // 0.5 to 1 % at 256^3, 3.5 % at 128^3.
  pl.rev = true;
  const char* env = getenv("SNS_XY_PASSES");
  const bool dataflow = env && env[0] == '1';
  pl.use_xy = !real && dataflow && xy_supported(nx, ny, prec) &&
              xy_plan(pl.xy, nx, ny, nz, prec) == OK;
  pl.use_xyc = !real && !pl.use_xy && xyc_supported(nx, ny, prec);
  // separate passes run in slabs of xy_chunk planes (SNS_XY_CHUNK; 0 = one slab)
  pl.xy_chunk = 0;
  if (const char* e = getenv("SNS_XY_CHUNK")) pl.xy_chunk = atoi(e);
  if (pl.xy_chunk > 0 && pl.xy_chunk < nz) pl.use_xyc = false;
  pl.passes = (pl.use_xy || pl.use_xyc || (pl.xy_chunk > 0 && pl.xy_chunk < nz)) ? 3 : 5;
  pl.lineW = lineW > 0 ? lineW : 0;
  pl.lineT = 0;
  pl.lineOrd = 0;
  {
    // The y passes of fields beyond L2 over TMA-staged tiles in complex64
    // (SNS_Y_TMA = 0: direct loads, 1 or 2 stages).  B200, 256^3, both passes:
    // complex64 0.418 ms against 0.473 with direct loads; complex128 0.85
    // against 0.75.
    const char* e = getenv("SNS_Y_TMA");
    const int v = e ? atoi(e) : big && prec == PREC_C64 ? 1 : 0;
    pl.y_tma = 0;
    if ((v == 1 || v == 2) &&
        line_tma_ok(axis_geo(1, nx, ny, nz, prec, pl.lineW, pl.lineT), prec, v))
      pl.y_tma = v;
  }
  pl.tuned = false;
  pl.k1_lines = false;  // enabled by a caller that provides the work fields W
  {
    // L2 prefetch of the tile a wave or two ahead (SNS_PF = 0, 1, 2 waves)
    const char* e = getenv("SNS_PF");
    pl.pf_waves = e ? std::max(0, std::min(4, atoi(e))) : 0;
  }
  {
    const char* e = getenv("SNS_K1_RELOAD");
    pl.k1_reload = e && e[0] == '1';
  }
  {
    // K1 over TMA-staged tiles, one stage by default (SNS_K1_TMA = 0: off,
    // 2: two stages); an explicit SNS_K1_RELOAD=1 or SNS_K1_SPLIT=1 keeps
    // that form.  Measured on B200 at 256^3: complex64 0.27 ms against 0.37
    // (reload tile), complex128 0.50 against 0.92 (reload; 0.79 split, before).
    const char* e = getenv("SNS_K1_TMA");
    const char* es = getenv("SNS_K1_SPLIT");
    const int v = e ? atoi(e) : ((pl.k1_reload || (es && es[0] == '1')) ? 0 : 1);
    pl.k1_stages = v == 2 ? 2 : 1;
    pl.k1_tma = false;
    if (v == 1 || v == 2) {
      // the widest tile of at most 384 threads that fits the stages
      const int TPL = nz / elems(nz);
      for (int W = 16; W >= 1 && !pl.k1_tma; W /= 2)
        for (int G = 4; G >= 1 && !pl.k1_tma; G /= 2)
          if (3 * W * G * TPL <= 384 && k1_tma_ok(pl, W, G, pl.k1_stages)) {
            pl.k1_tma = true;
            pl.k1_fused = true;
            pl.k1W = W;
            pl.k1G = G;
          }
    }
  }
  pl.k1lW = 0;
  pl.k1lT = 0;
  pl.plane = !separate && plane_wanted(nx, ny, nz, prec, real);
  if (pl.plane) {
    // two launches per step: the plane pass, and the update pass with the next
    // step's K1 carried in it, in CTAs enough for the SMs
    const int Wmax = prec == PREC_C128 ? 8 : 16;
    int W = 1;
    pl.carry = false;
    while (W * 2 <= Wmax && nx % (W * 2) == 0 && (nx / (W * 2)) * ny >= 128) W *= 2;
    for (; W >= 1 && !pl.carry; W /= 2)
      if (carry_ok(pl, W, false)) {
        pl.carry = true;
        pl.carry_reload = false;
        pl.zW = W;
        pl.update_blocks = (nx / W) * ny;
      }
    pl.passes = 3;
  }
  pl.kc2 = 1e300;
  pl.sgs_klo = 0;
  pl.sgs_kinv = 1e30;
  return OK;
}

namespace {

// K1 as a z pass of V into U[0..5] (the fused tile or one field per CTA).
int run_k1(const NSPlan& pl, void* const V[3], void* const U[6], int* err_word, cudaStream_t s) {
  FieldPtrs f{};
  f.n = 6;
  for (int d = 0; d < 3; d++) f.in[d] = V[d];
  for (int i = 0; i < 6; i++) f.out[i] = U[i];
  if (pl.k1_fused)
    return pl.prec == PREC_C128 ? ns_zcurl<double>(pl, f, err_word, s)
                                : ns_zcurl<float>(pl, f, err_word, s);
  LineGeo g = axis_geo(2, pl.nx, pl.ny, pl.nz, pl.prec, pl.lineW);
  g.kx_half = pl.real;
  g.rev = pl.rev;
  return run_line_pass(g, f, +1, 0, 1.0, pl.prec, s, PRO_CURL6);
}

}  // namespace

namespace {

// The six fields a step works in: its cross product is built where its history
// is not.
struct StepFields {
  void* U[6];
  void* H[3];
};
StepFields step_fields(void* const C0[3], void* const U[6], int hist) {
  StepFields f;
  for (int i = 0; i < 3; i++) {
    f.U[i] = hist == HIST_Z_U ? C0[i] : U[i];
    f.H[i] = hist == HIST_Z_U ? U[i] : C0[i];
    f.U[3 + i] = U[3 + i];
  }
  return f;
}

}  // namespace

int ns_k1_once(const NSPlan& pl, void* const V[3], void* const C0[3], void* const U[6], int hist,
               int* sync_words, cudaStream_t s) {
  if (pl.k1_lines) {
    set_error("ns_k1_once: K1 as a line pass writes the work fields W, not U");
    return ERR_ARG;
  }
  return run_k1(pl, V, step_fields(C0, U, hist).U,
                sync_words ? sync_words + xy_sync_words(pl.nz) - 1 : nullptr, s);
}

int ns_hist_fourier(const NSPlan& pl, void* const* src, void* const* dst, int n, cudaStream_t s) {
  FieldPtrs f{};
  f.n = n;
  for (int i = 0; i < n; i++) {
    f.in[i] = src[i];
    f.out[i] = dst[i];
  }
  LineGeo g = axis_geo(2, pl.nx, pl.ny, pl.nz, pl.prec);
  g.kx_half = pl.real;
  int rc = run_line_pass(g, f, -1, PASS_ZERO_NYQUIST, 1.0, pl.prec, s);
  for (int i = 0; i < n && !rc && pl.kc2 < 1e300; i++)
    rc = op_cutoff(dst[i], pl.kc2, pl.real, Dims{pl.nx, pl.ny, pl.nz}, pl.prec, s);
  return rc;
}

int ns_step_once(const NSPlan& pl, void* const V[3], void* const C0[3], void* const U_[6],
                 double* stats, int* sync_words, double nu, double dt, cudaStream_t s,
                 cudaEvent_t* ev, void* const* W, bool* carried, int* hist) {
  const int h0 = hist ? *hist : HIST_FOURIER;
  const StepFields sf = step_fields(C0, U_, h0);
  void* const(&U)[6] = sf.U;
  const int nx = pl.nx, ny = pl.ny, nz = pl.nz, prec = pl.prec;
  // the error word of the step's bounded waits
  int* err_word = sync_words ? sync_words + xy_sync_words(nz) - 1 : nullptr;
  int rc;
  int pass = 0;
  auto mark = [&]() {
    if (ev) cudaEventRecord(ev[pass], s);
    pass++;
  };
  mark();
  const bool lines = pl.k1_lines && W && !pl.use_xy && !pl.use_xyc && !pl.plane;
  // K1 carried in the previous step's K5: U already holds its output
  const bool carry = pl.carry && carried && !lines;
  const bool have_k1 = carry && *carried;
  if (carried) *carried = false;
  // K1: z-inverse of (V, i k x V)
  if (have_k1) {
    mark();
  } else if (lines) {
    // V and the z derivatives i kz Vx, i kz Vy (taken on the way in), each
    // field z-inverse-transformed on its own; K2 forms omega from them
    FieldPtrs f{};
    f.n = kNSLineWork;
    for (int d = 0; d < 3; d++) f.in[d] = V[d];
    f.in[3] = V[0];
    f.in[4] = V[1];
    for (int i = 0; i < kNSLineWork; i++) f.out[i] = W[i];
    f.ikmask = 0x18u;
    LineGeo g = axis_geo(2, nx, ny, nz, prec, pl.k1lW, pl.k1lT);
    g.kx_half = pl.real;
    rc = run_line_pass(g, f, +1, 0, 1.0, prec, s, PRO_IKAXIS);
    if (rc) return rc;
    mark();
  } else {
    if ((rc = run_k1(pl, V, U, err_word, s))) return rc;
    mark();
  }
  if (pl.use_xy) {
    // K2 + K3 + K4 as one persistent dataflow launch (sns_xy.cu)
    if ((rc = xy_run(pl.xy, U, sync_words, s))) return rc;
    mark();
  } else if (pl.use_xyc) {
    // K2 + K3 + K4 as one cluster pass over each plane (sns_xyc.cu)
    if ((rc = xyc_run(U, nx, ny, nz, prec, s))) return rc;
    mark();
  } else if (pl.plane) {
    // K2 + K3 + K4 with one CTA per plane (sns_plane.cu)
    if ((rc = plane_run(U, U, nx, ny, nz, prec, pl.real, pl.scale2, s))) return rc;
    mark();
  }
  // K2, K3, K4 on the planes [z0, z0 + pz): the passes treat the slab as an
  // nx*ny*pz field at an offset pointer (the 1/N^2 scale keeps the full N)
  const size_t esz = prec == PREC_C128 ? 16 : 8;
  auto xy_range = [&](int z0, int pz, bool marks) -> int {
    const size_t off = esz * (size_t)z0 * nx * ny;
    void* Uc[6];
    for (int i = 0; i < 6; i++) Uc[i] = static_cast<char*>(U[i]) + off;
    if (lines) {  // K2: y-inverse of V and of omega formed from the five z-inverted fields
      FieldPtrs f{};
      f.n = 6;
      for (int i = 0; i < kNSLineWork; i++) f.in[i] = static_cast<char*>(W[i]) + off;
      f.in[5] = f.in[0];
      for (int i = 0; i < 6; i++) f.out[i] = Uc[i];
      LineGeo g = axis_geo(1, nx, ny, pz, prec, pl.lineW, pl.lineT, pl.lineOrd);
      g.kx_half = pl.real;
      g.pfw = pl.pf_waves;
      int r = run_line_pass(g, f, +1, 0, 1.0, prec, s, PRO_OMEGA);
      if (r) return r;
      if (marks) mark();
    } else {  // K2: y-inverse of the six fields
      FieldPtrs f{};
      f.n = 6;
      for (int i = 0; i < 6; i++) f.in[i] = f.out[i] = Uc[i];
      LineGeo g = axis_geo(1, nx, ny, pz, prec, pl.lineW, pl.lineT, pl.lineOrd);
      g.pfw = pl.pf_waves;
      int r = pl.y_tma && err_word && line_tma_ok(g, prec, pl.y_tma)
                  ? run_line_pass_tma(g, f, +1, 0, 1.0, prec, s, pl.y_tma, err_word)
                  : run_line_pass(g, f, +1, 0, 1.0, prec, s);
      if (r) return r;
      if (marks) mark();
    }
    {  // K3: x-inverse, cross product, x-forward
      FieldPtrs f{};
      f.n = 6;
      for (int i = 0; i < 6; i++) f.in[i] = Uc[i];
      for (int i = 0; i < 3; i++) f.out[i] = Uc[i];
      const int64_t rows = (int64_t)ny * pz;
      int r = xpass(pl, f, rows, err_word, s);
      if (r) return r;
      if (marks) mark();
    }
    {  // K4: y-forward of the cross product
      FieldPtrs f{};
      f.n = 3;
      for (int i = 0; i < 3; i++) f.in[i] = f.out[i] = Uc[i];
      LineGeo g = axis_geo(1, nx, ny, pz, prec, pl.lineW, pl.lineT, pl.lineOrd);
      g.pfw = pl.pf_waves;
      int r = pl.y_tma && err_word && line_tma_ok(g, prec, pl.y_tma)
                  ? run_line_pass_tma(g, f, -1, 0, 1.0, prec, s, pl.y_tma, err_word)
                  : run_line_pass(g, f, -1, 0, 1.0, prec, s);
      if (r) return r;
    }
    return OK;
  };
  if (!pl.use_xy && !pl.use_xyc && !pl.plane) {
    if (pl.xy_chunk > 0 && pl.xy_chunk < nz) {
      // slabs of xy_chunk planes, so each slab's intermediates stay in L2
      for (int z0 = 0; z0 < nz; z0 += pl.xy_chunk)
        if ((rc = xy_range(z0, std::min(pl.xy_chunk, nz - z0), false))) return rc;
    } else if ((rc = xy_range(0, nz, true))) {
      return rc;
    }
    mark();
  }
  // K5: z-forward + Nyquist zeroing + AB2/projection/CN update
  {
    UpdateArgs a{};
    for (int d = 0; d < 3; d++) {
      a.U[d] = U[d];
      a.V[d] = V[d];
      a.C0[d] = sf.H[d];
    }
    a.fourier = h0 == HIST_FOURIER;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.W = pl.zW;
    a.lx = 0;
    while ((1 << a.lx) < nx) a.lx++;
    a.hK = dt / 2;
    a.nuhK = nu * dt / 2;
    a.stats = stats;
    a.kc2 = pl.kc2;
    a.kx_half = pl.real;
    if (carry) {
      // K5 with the next step's K1 carried: the next step's fields receive the
      // z-inverse of the new V and of its curl (over this step's history, which
      // the tile has read)
      for (int i = 0; i < 3; i++) {
        a.Uo[i] = sf.H[i];
        a.Uo[3 + i] = U[3 + i];
      }
      rc = prec == PREC_C128 ? ns_update_carry<double>(pl, a, s) : ns_update_carry<float>(pl, a, s);
    } else {
      rc = ns_update(pl, a, false, s, err_word);
    }
    if (rc) return rc;
    if (carried) *carried = carry;
    if (hist) *hist = h0 == HIST_Z_U ? HIST_Z_C0 : HIST_Z_U;
    mark();
  }
  return OK;
}

namespace {

constexpr size_t kTuneSmemCap = 220 * 1024;

// Seeded values in [-1, 1) for the tuner's timing steps, so that every pass
// runs on data of the magnitude a run has (a counter hash, not a statistical
// generator).
template <typename T>
__global__ void k_fill_tune(cx_t<T>* p, int64_t n, uint32_t seed) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t h = (uint32_t)i * 2654435761u ^ seed;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    const uint32_t h2 = h * 3266489917u ^ (h >> 16);
    p[i] = mk((T)((int32_t)h) * (T)4.656612873077393e-10,
              (T)((int32_t)h2) * (T)4.656612873077393e-10);
  }
}

int fill_tune(void* p, int64_t n, int prec, uint32_t seed, cudaStream_t s) {
  const int grid = std::max(1, std::min(4 * sm_count(), (int)((n + 255) / 256)));
  if (prec == PREC_C128)
    k_fill_tune<double><<<grid, 256, 0, s>>>(reinterpret_cast<double2*>(p), n, seed);
  else
    k_fill_tune<float><<<grid, 256, 0, s>>>(reinterpret_cast<float2*>(p), n, seed);
  SNS_CHECK_LAUNCH("k_fill_tune");
  return OK;
}

bool k1_ok(const NSPlan& p, int W, int G, bool reload) {
  const int TPL = p.nz / elems(p.nz);
  const size_t esz = p.prec == PREC_C128 ? 16 : 8;
  return p.nx % W == 0 && p.ny % G == 0 && 3 * W * G * TPL <= max_threads(p.prec) &&
         (size_t)(reload ? 3 : 6) * W * G * tile_stride(p.nz, W, (int)esz) * esz <= kTuneSmemCap;
}
bool xg_ok(const NSPlan& p, int G) {
  const int TPL = p.nx_phys / elems(p.nx_phys);
  const size_t esz = p.prec == PREC_C128 ? 16 : 8;
  const int cap = p.real ? 384 : max_threads(p.prec);  // k_xcross_real launch bound
  return ((int64_t)p.ny * p.nz) % (p.real ? 2 * G : G) == 0 && 6 * G * TPL <= cap &&
         (size_t)6 * G * xrow_stride(p.nx_phys, (int)esz) * esz <= kTuneSmemCap;
}
bool zw_ok(const NSPlan& p, int W, int max_blocks, bool halves = false) {
  const int TPL = p.nz / elems(p.nz);
  const size_t esz = p.prec == PREC_C128 ? 16 : 8;
  // halves: the plain update pass may transform a tile in two halves of W/2
  const int thr = 3 * W * TPL / (halves && 3 * W * TPL > max_threads(p.prec) ? 2 : 1);
  return p.nx % W == 0 && thr <= max_threads(p.prec) &&
         (size_t)3 * W * tile_stride(p.nz, W, (int)esz) * esz <= kTuneSmemCap &&
         ((int64_t)p.nx * p.ny) / W <= max_blocks;
}

}  // namespace

int ns_tune_plan(NSPlan& pl, void* const V[3], void* const C0[3], void* const U[6],
                 double* stats, int max_blocks, int* sync_words, cudaStream_t s,
                 void* const* W) {
  if (pl.plane) pl.tuned = true;  // nothing to choose: the plane pass has one form
  if (pl.passes != kNSPasses) return OK;
  cudaEvent_t ev[kNSPasses + 1];
  int rc = OK;
  // the timing steps run on seeded data (with dt = 0 and nu = 0 a step only
  // projects V, so the values stay bounded); the caller clears them after
  const int64_t n = (int64_t)pl.nx * pl.ny * pl.nz;
  for (int d = 0; d < 3 && rc == OK; d++) {
    rc = fill_tune(V[d], n, pl.prec, 17u + d, s);
    if (rc == OK) rc = fill_tune(C0[d], n, pl.prec, 29u + d, s);
  }
  int made = 0;
  for (; made < kNSPasses + 1 && rc == OK; made++)
    rc = cuda_status(cudaEventCreate(&ev[made]), "ns_tune_plan(events)");
  // time of the passes in the bit mask `passes` of a candidate plan: one step
  // to set the kernels up, then the least of five timed steps
  auto measure = [&](const NSPlan& c, unsigned passes, float* out) -> int {
    float best = 3.4e38f;
    bool carried = false;
    int hist = HIST_FOURIER;
    for (int r = 0; r < 6; r++) {
      int e = ns_step_once(c, V, C0, U, stats, sync_words, 0.0, 0.0, s, r ? ev : nullptr, W,
                           &carried, &hist);
      if (e) return e;
      if (!r) continue;
      if ((e = cuda_status(cudaEventSynchronize(ev[kNSPasses]), "ns_tune_plan"))) return e;
      float sum = 0;
      for (int p = 0; p < kNSPasses; p++)
        if ((passes >> p) & 1u) {
          float t = 0;
          cudaEventElapsedTime(&t, ev[p], ev[p + 1]);
          sum += t;
        }
      best = std::min(best, sum);
    }
    *out = best;
    return OK;
  };
  // SNS_TUNE_LOG=1 prints every candidate's time to stderr
  const bool log = getenv("SNS_TUNE_LOG") && getenv("SNS_TUNE_LOG")[0] == '1';
  // margin > 0: cands[0] is the incumbent plan, and another candidate
  // replaces it only when faster by that fraction (whole-step timings of a few
  // steps vary by 1-2 % between runs)
  auto pick = [&](std::vector<NSPlan>& cands, unsigned passes, float margin = 0.f) -> int {
    float best = 3.4e38f, t0 = 3.4e38f;
    int bi = -1;
    for (size_t i = 0; i < cands.size(); i++) {
      float t = 0;
      int e = measure(cands[i], passes, &t);
      if (e) return e;
      if (log)
        fprintf(stderr,
                "ns_tune passes=0x%x cand=%zu ms=%.4f k1=%dx%d%s%s xG=%d%s zW=%d%s%s lineW=%d "
                "lineT=%d ord=%d ytma=%d pf=%d\n",
                passes, i, t, cands[i].k1W, cands[i].k1G, cands[i].k1_tma ? "(tma)" : "",
                cands[i].k1_reload ? "(reload)" : "", cands[i].xG,
                cands[i].x_tma ? "(tma)" : cands[i].x_occ ? "(occ)" : "",
                cands[i].zW, cands[i].z_tma ? "(tma)" : cands[i].z_pfself ? "(pfs)" : "",
                cands[i].carry ? (cands[i].carry_reload ? "(+K1r)" : "(+K1)") : "",
                cands[i].lineW, cands[i].lineT, cands[i].lineOrd, cands[i].y_tma,
                cands[i].pf_waves);
      if (i == 0) t0 = t;
      if (t < best) {
        best = t;
        bi = (int)i;
      }
    }
    if (margin > 0.f && bi > 0 && best > t0 * (1.f - margin)) bi = 0;
    if (bi >= 0) pl = cands[bi];
    return OK;
  };
  std::vector<NSPlan> c;
  const NSPlan given = pl;
  // K1: the z-inverse + curl pass as a fused tile (its shape), one output
  // field per CTA, or the five-field line pass with the curl formed in K2
  // (its run width and thread cap); timed with K2, whose input it sets
  if (rc == OK) {
    c.clear();
    c.push_back(pl);
    for (int reload = 0; reload < 2; reload++)
      for (int Wd : {2, 4, 8, 16})
        for (int G : {1, 2, 4})
          if (k1_ok(pl, Wd, G, reload)) {
            NSPlan q = pl;
            q.k1W = Wd;
            q.k1G = G;
            q.k1_fused = true;
            q.k1_reload = reload;
            q.k1_lines = false;
            q.k1_tma = false;
            c.push_back(q);
          }
    // the persistent pass over TMA-staged tiles (one or two stages)
    if (sync_words)
      for (int S = 1; S <= 2; S++)
        for (int Wd : {2, 4, 8, 16})
          for (int G : {1, 2, 4})
            if (k1_tma_ok(pl, Wd, G, S)) {
              NSPlan q = pl;
              q.k1W = Wd;
              q.k1G = G;
              q.k1_fused = true;
              q.k1_tma = true;
              q.k1_stages = S;
              q.k1_lines = false;
              c.push_back(q);
            }
    NSPlan split = pl;
    split.k1_fused = false;
    split.k1_lines = false;
    split.k1_tma = false;
    c.push_back(split);
    if (W)
      for (int Wd : {8, 16})
        for (int T : {256, 512}) {
          NSPlan q = pl;
          q.k1_lines = true;
          q.k1_tma = false;
          q.k1lW = Wd;
          q.k1lT = T;
          c.push_back(q);
        }
    rc = pick(c, 0x3u);
  }
  // K2 + K4: run width and thread cap, then radix order, of the y line passes
  if (rc == OK) {
    c.clear();
    c.push_back(pl);
    std::set<std::tuple<int, int, int>> seen;  // tiles listed (thread caps often share one)
    for (int W : {4, 8, 16, 32})
      for (int T : {64, 128, 256, 512})
        for (int S = 0; S <= (sync_words ? 2 : 0); S++) {
          const LineGeo g = axis_geo(1, pl.nx, pl.ny, pl.nz, pl.prec, W, T);
          if (!seen.insert({g.W, g.G, S}).second) continue;
          NSPlan q = pl;
          q.lineW = W;
          q.lineT = T;
          q.y_tma = S;
          if (S && !line_tma_ok(axis_geo(1, pl.nx, pl.ny, pl.nz, pl.prec, W, T, pl.lineOrd),
                                pl.prec, S))
            continue;
          c.push_back(q);
        }
    rc = pick(c, 0xAu);
  }
  if (rc == OK && pl.ny >= 64 && pl.ny <= 1024) {
    c.clear();
    for (int o = 0; o < kRadixOrders; o++) {
      NSPlan q = pl;
      q.lineOrd = o;
      if (q.y_tma && !line_tma_ok(axis_geo(1, pl.nx, pl.ny, pl.nz, pl.prec, pl.lineW, pl.lineT, o),
                                  pl.prec, q.y_tma))
        continue;
      c.push_back(q);
    }
    rc = pick(c, 0xAu);
  }
  // K3: rows per CTA of the x cross pass
  if (rc == OK) {
    c.clear();
    c.push_back(pl);
    for (int G : {1, 2, 4, 8, 16}) {
      if (xg_ok(pl, G)) {
        NSPlan q = pl;
        q.xG = G;
        q.x_tma = false;
        q.x_occ = false;
        c.push_back(q);
        // the five-CTA form, for CTAs of at most 192 threads (complex64)
        if (!pl.real && pl.prec == PREC_C64 && 6 * G * (pl.nx / elems(pl.nx)) <= 192) {
          q.x_occ = true;
          c.push_back(q);
        }
      }
      if (sync_words && x_tma_ok(pl, G)) {
        NSPlan q = pl;
        q.xG = G;
        q.x_occ = false;
        q.x_tma = true;
        c.push_back(q);
      }
    }
    rc = pick(c, 0x4u);
  }
  // K5: adjacent z lines per CTA of the update pass
  if (rc == OK) {
    c.clear();
    c.push_back(pl);
    for (int W : {2, 4, 8, 16, 32, 64}) {
      if (zw_ok(pl, W, max_blocks, true))
        for (int pfs = 0; pfs < 2; pfs++) {
          NSPlan q = pl;
          q.zW = W;
          q.z_tma = false;
          q.z_pfself = pfs == 1;
          q.update_blocks = (pl.nx / W) * pl.ny;
          c.push_back(q);
        }
      if (sync_words && zw_ok(pl, W, max_blocks) && z_tma_ok(pl, W)) {
        NSPlan q = pl;
        q.zW = W;
        q.z_tma = true;
        q.update_blocks = (pl.nx / W) * pl.ny;
        c.push_back(q);
      }
    }
    rc = pick(c, 0x10u);
  }
  // the passes so chosen against the plan as it was, over the whole step: a tile
  // that is faster in its own pass can cost the next one, and single passes of
  // small boxes are a few microseconds (a 32 x 64 x 256 complex64 step on B200:
  // 56.3 to 57.0 us tuned pass by pass, 55.4 by default, now 55.8)
  if (rc == OK) {
    c = {given, pl};
    rc = pick(c, 0x1Fu);
  }
  // K5 with the next step's K1 carried in it (tile widths), against the
  // plan so far, over the whole step: it trades K1's pass for a heavier K5.
  // Measured slower in steady state on B200 at 256^3 (whole step 1.37 to 1.44
  // against 1.30 ms; complex128 2.74 to 2.90 against 2.57), so it is only tried
  // on request (SNS_TUNE_CARRY=1)
  const char* etc = getenv("SNS_TUNE_CARRY");
  if (rc == OK && !pl.k1_lines && !getenv("SNS_CARRY") && etc && etc[0] == '1') {
    c.clear();
    c.push_back(pl);
    for (int reload = 0; reload < 2; reload++)
      for (int Wd : {2, 4, 8, 16, 32})
        if (zw_ok(pl, Wd, max_blocks) && carry_ok(pl, Wd, reload)) {
          NSPlan q = pl;
          q.carry = true;
          q.carry_reload = reload;
          q.z_tma = false;
          q.zW = Wd;
          q.update_blocks = (pl.nx / Wd) * pl.ny;
          c.push_back(q);
        }
    rc = pick(c, 0x1Fu, 0.02f);
  }
  // L2 prefetch distance of all five passes, timed over the whole step
  // (unless SNS_PF fixes it)
  if (rc == OK && !getenv("SNS_PF")) {
    c.clear();
    c.push_back(pl);
    for (int pw : {0, 1, 2}) {
      if (pw == pl.pf_waves) continue;
      NSPlan q = pl;
      q.pf_waves = pw;
      c.push_back(q);
    }
    rc = pick(c, 0x1Fu, 0.02f);
  }
  for (int i = 0; i < made; i++) cudaEventDestroy(ev[i]);
  if (rc == OK) pl.tuned = true;
  return rc;
}

int ns_update(const NSPlan& pl, const UpdateArgs& a, bool sgs, cudaStream_t s, int* err) {
  if (pl.prec == PREC_C128)
    return sgs ? ns_update_as<double, true>(pl, a, err, s) : ns_update_as<double, false>(pl, a, err, s);
  return sgs ? ns_update_as<float, true>(pl, a, err, s) : ns_update_as<float, false>(pl, a, err, s);
}

// The normalisation sns_ns_stats applies on the host (mean |div|, 1/2 <|u|^2>,
// 1/2 <|omega|^2> of the unnormalised Fourier fields), with the same divisions.
__global__ void k_stats_normalise(double* out4, double N) {
  if (threadIdx.x == 0) {
    out4[0] = out4[0] / N;
    out4[1] = 0.5 * out4[1] / (N * N);
    out4[2] = 0.5 * out4[2] / (N * N);
  }
}

int ns_stats_normalise(double* out4, double N, cudaStream_t s) {
  k_stats_normalise<<<1, 32, 0, s>>>(out4, N);
  SNS_CHECK_LAUNCH("k_stats_normalise");
  return OK;
}

int ns_stats_final(const double* partials, int blocks, double* out4, cudaStream_t s) {
  k_stats_final<<<1, 256, 0, s>>>(partials, blocks, out4);
  SNS_CHECK_LAUNCH("k_stats_final");
  return OK;
}

}  // namespace sns
