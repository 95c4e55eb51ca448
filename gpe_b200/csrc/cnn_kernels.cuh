// cnn_kernels.cuh -- the learned coarse-grid correction: a 4-layer 3x3x3
// conv3d network (2 -> 16 -> 16 -> 16 -> 2 channels, GELU between layers,
// BF16 weights and activations, FP32 accumulation) applied to psi after a
// coarse time step, and its training kernels.
//
// Activation layout (global and shared memory): bf16 [Zp][Yp][H][Xp][8] with
// Xp = nx + 2, Yp = ny + 2, Zp = nz + 2 (one periodic ghost site per side,
// written by the kernel that writes the interior) and the 16 channels split
// into H = 2 halves of 8.  One x-row half is therefore a run of 16-byte
// records, which is exactly the no-swizzle K-major core-matrix layout of a
// tcgen05 A operand (8 sites x 8 channels per 128-byte core matrix): the A
// operand of tap (dz, dy, dx) for 128 consecutive sites of a row is the row's
// address + 16 * dx, with LBO = the half stride.  No im2col copy exists.
//
// Forward / dgrad kernel: one CTA per (y-slab of 8 rows, z-chunk) item;
// warp 0 streams input planes (8 + 2 rows, both halves, the full padded x
// extent) into a 4-slot ring -- in this layout those rows are one contiguous
// range, fetched by a single 1-D bulk copy (a tensor-map tile with its
// 16-byte innermost extent moved the same bytes several times slower); warp 1
// issues, per input plane and per (input row, dx), ONE tcgen05.mma (M = 128
// sites, N = 144, K = 16) whose D block covers every output site that input row
// feeds: 3 output rows x 3 output planes x 16 channels.  The accumulators of
// three output planes rotate in TMEM; when an input plane's MMAs complete, one
// output plane is finished.  Its rows are handed over in two halves of four:
// the 8 epilogue warps of a half copy its rows to registers (tcgen05.ld
// 32x32b), zero their slots, release them to the MMA warp, and only then run
// the epilogue and the stores, which overlap the other half's MMAs and the next
// plane's.  Every MMA accumulates; slots are zero when a plane first receives
// data.
//
// What bounds it: instruction issue of the epilogue (GELU, packing, stores;
// about 75% of all issue slots) and then the bytes, 134 MB a layer forward, 201
// where the pre-activation is written or read too.  At 128^3, a layer forward
// 50.3 -> 33.8 us, with pre-activation 52 -> 42, dgrad 71 -> 46.8, the last
// layer 35.6 -> 27.9 (of these the elected lane, see tc::elect_one, took an MMA
// from 110 to 45 cycles of the issuing thread; stores whose ghost images are
// predicated rather than searched for, and the halves, the rest).  One CTA of 8
// rows per SM in place of two of 4 reads 1.25 instead of 1.5 times the input and
// keeps four planes in flight in the same shared memory.
//
// Weight-gradient kernel: D[(xrow, ci), (yrow, co)] += X[xrow, ci, x + dx] *
// dY[yrow, co, x] summed over x in 16-site K steps; A (X) and B (dY) are
// MN-major operands read in place: 8 consecutive X rows x 2 halves form the 16
// M-groups of an M = 128 operand, 6 dY rows x 2 halves the 12 N-groups of an
// N = 96 one, and the blocks with xrow - yrow = 0, 1, 2 are the dy taps of all
// six rows.  An MMA takes about 90 cycles whatever its N up to 96 (both
// operands come out of shared memory across the grain), so this does in one
// what took six with N = 16 (one dY row): 578 -> 66 us a layer at 128^3.  One
// accumulator of 96 TMEM columns per (dz, dx), so a CTA takes five of the nine
// (dz, dx) taps or the other four (5 x 96 = 480 of 512 columns), over an equal
// share of all (slab, plane) positions.  The epilogue warps sum dY's channels
// (the bias gradient) from the same tiles meanwhile.
// All waits are bounded; a timeout sets *status.
#pragma once

#include <cuda_bf16.h>

#include "device_utils.cuh"
#include "tcgen05.cuh"
#include "vec2.cuh"

namespace gpe {
namespace cnn {

constexpr int CH = 16;
constexpr int NTAP = 27;
constexpr int NLAYER = 4;

// forward / dgrad
constexpr int TYF = 8;          // output rows per item
constexpr int HROWS = TYF / 2;  // rows whose accumulators are handed over together
constexpr int FSLOTS = 4;       // input planes in the shared-memory ring
constexpr int F_EPI_WARPS = 4 * HROWS;  // one per lane quarter and row of a half
constexpr int F_THREADS = 32 * (2 + F_EPI_WARPS);
// Accumulators: three output planes in a rotating ring (plane z in slot
// z mod 3), each with the TYF output rows of the slab, column
// (row * 3 + slot) * 16 + co.  Input row y' (box row i) of input plane j
// feeds output rows y'-1, y', y'+1 of output planes j-1, j, j+1 (all three
// slots): for an interior input row one contiguous block of 144 columns,
// so a single MMA with N = 144 covers all nine (dz, dy) taps of one dx; the
// slab's first two and last two input rows feed only one or two of its
// rows and use N = 48 / 96 with the matching part of B.
constexpr int OSLOTS = 3;
constexpr int ACC_ROWS = TYF;
constexpr int NSTACK = 3 * OSLOTS * CH;          // 144
constexpr uint32_t F_TMEM_COLS = 512;
static_assert(ACC_ROWS * OSLOTS * CH <= (int)F_TMEM_COLS, "accumulator ring fits TMEM");
// B tile of one (rotation j mod 3, dx): rows n = (jrow * 3 + s) * 16 + co
// hold tap (dz index 2 - ((s - rot + 1) mod 3), dy index 2 - jrow, dx);
// K = 16 input channels in two halves: [2][144][8] bf16.
constexpr int WT_BYTES = 2 * NSTACK * 8 * 2;     // 4608
constexpr int W_TILES = 9;                       // 3 rotations x 3 dx
// Per output-channel count: accumulator columns per (row, slot) and the
// MMA's N.  The last layer has 2 output channels: 9 x 2 = 18 columns padded
// to N = 32 (the 14 extra B rows are zero; they add exact zeros to columns
// of the next rows, which accumulate in the same MMA stream).
template <int CO>
struct OutShape {
  static constexpr int CW = CO;
  static constexpr int NB = CO == 16 ? NSTACK : 32;  // rows of one B tile
  static constexpr int WTB = 2 * NB * 8 * 2;
  // N of an MMA feeding `cnt` (1..3) of the slab's rows, rounded up to 16
  __host__ __device__ static constexpr int n_of(int cnt) {
    return CO == 16 ? 48 * cnt : ((6 * cnt + 15) / 16) * 16;
  }
};
static_assert(OutShape<2>::NB >= 9 * 2, "padded N holds the 18 real columns");
// every MMA's D block (padded N included) stays inside the allocation
static_assert((TYF - 1) * OSLOTS * 2 + 32 <= (int)F_TMEM_COLS, "padded blocks fit");
// after the weights: 2*FSLOTS + 6 mbarriers, TMEM address, abort flag, and 16
// biases that are read four at a time
constexpr int F_TAIL_BYTES = 256, F_BIAS_OFF = 128;
static_assert((2 * FSLOTS + 6) * 8 + 8 <= F_BIAS_OFF && F_BIAS_OFF % 16 == 0 &&
                  F_BIAS_OFF + CH * 4 <= F_TAIL_BYTES, "tail fits");
static_assert(W_TILES * OutShape<16>::WTB % 16 == 0 && W_TILES * OutShape<2>::WTB % 16 == 0,
              "the tail starts on 16 bytes");

// weight gradient
constexpr int TYW = 6;            // dY rows of a slab
constexpr int XROWS = TYW + 2;    // X rows they need: M = 128 = 8 rows x 16 channels
constexpr int WSLOTS = 4;         // X planes in the ring (two in use)
constexpr int DSLOTS = 3;         // dY planes
constexpr int W_EPI_WARPS = 4;
constexpr int W_THREADS = 32 * (2 + W_EPI_WARPS);
constexpr uint32_t W_TMEM_COLS = 512;
constexpr int W_NCOL = TYW * CH;  // 96 columns per accumulator
constexpr int W_TAPS0 = 5;        // (dz, dx) taps 0-4 in one role, 5-8 in the other
constexpr int W_PART = W_TAPS0 * 3 * CH * CH;  // floats of one CTA's partial sums
static_assert(XROWS * CH == 128, "X rows fill M");
static_assert(W_TAPS0 * W_NCOL <= (int)W_TMEM_COLS, "accumulators fit TMEM");

enum Epi { EPI_GELU = 0, EPI_GELU_PRE = 1, EPI_DELTA = 2, EPI_RESID = 3, EPI_DGELU = 4 };

struct ConvParams {
  const __nv_bfloat16* in;          // input activations [Zp][Yp][Hin][Xp][8]
  const __nv_bfloat16* w;           // [27][2][16][8]
  const float* bias;                // [16] or null
  int nx, ny, nz, Xp, Yp, Zp, Hin;
  int nslab, nzc, zchunk, nitems;
  uint32_t slot_bytes;
  __nv_bfloat16* act_out;           // [Zp][Yp][2][Xp][8]
  __nv_bfloat16* pre_out;           // EPI_GELU_PRE
  const __nv_bfloat16* pre_in;      // EPI_DGELU
  float* delta;                     // EPI_DELTA: dense [nz][ny][nx][2]
  float* psi;                       // EPI_RESID: solver field (complex64)
  int psi_Nx, psi_Ny, psi_gh;       // its pitches and ghost layers
  float out_scale;
  int* status;
  unsigned long long wait_limit_ns;
};

struct WgradParams {
  const __nv_bfloat16* x;           // layer input [Zp][Yp][2][Xp][8]
  const __nv_bfloat16* dy;          // gradient of the layer output, same layout
  int nx, ny, nz, Xp, Yp, Zp;
  int nslab;                        // slabs of TYW rows
  int role0;                        // CTAs that take taps 0..W_TAPS0-1
  uint32_t xslot_bytes, dslot_bytes;
  float* partials;                  // [gridDim.x][W_TAPS0][3 dy][16 co][16 ci]
  float* bpartials;                 // [role0][16]
  int* status;
  unsigned long long wait_limit_ns;
};

// GELU in its tanh form (Hendrycks & Gimpel, 2016):
//   gelu(x) = 0.5 x (1 + t),  t = tanh(u),  u = sqrt(2/pi) (x + 0.044715 x^3),
//   gelu'(x) = 0.5 (1 + t) + 0.5 x (1 - t^2) u',  u' = sqrt(2/pi) (1 + 3 * 0.044715 x^2).
// tanh through the hardware tanh.approx.f32 instruction (one MUFU operation,
// relative error about 2^-11, below the bfloat16 rounding of the result).
constexpr float GELU_C = 0.7978845608028654f;  // sqrt(2/pi)
constexpr float GELU_A = 0.044715f;

__device__ __forceinline__ float tanh_approx(float u) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return t;
}
// Two values at once on the packed FP32x2 pipe: u = x (C + C A x^2),
// gelu = h + h t with h = x / 2, t = tanh(u) (two scalar MUFU operations).
__device__ __forceinline__ float2 gelu2(float2 x) {
  const float2 x2 = __fmul2_rn(x, x);
  const float2 k = __ffma2_rn(make_float2(GELU_C * GELU_A, GELU_C * GELU_A), x2,
                              make_float2(GELU_C, GELU_C));
  const float2 u = __fmul2_rn(x, k);
  const float2 t = make_float2(tanh_approx(u.x), tanh_approx(u.y));
  const float2 h = __fmul2_rn(x, make_float2(0.5f, 0.5f));
  return __ffma2_rn(h, t, h);
}
__device__ __forceinline__ float2 gelu_grad2(float2 x) {
  constexpr float A3 = 3.0f * GELU_A;
  const float2 c2 = make_float2(GELU_C, GELU_C), one = make_float2(1.0f, 1.0f),
               half = make_float2(0.5f, 0.5f);
  const float2 v = __fmul2_rn(
      c2, __ffma2_rn(__fmul2_rn(make_float2(GELU_A, GELU_A), x), __fmul2_rn(x, x), x));
  const float2 t = make_float2(tanh_approx(v.x), tanh_approx(v.y));
  const float2 du = __fmul2_rn(c2, __ffma2_rn(__fmul2_rn(make_float2(A3, A3), x), x, one));
  const float2 dt = __ffma2_rn(make_float2(-t.x, -t.y), t, one);
  return __ffma2_rn(__fmul2_rn(__fmul2_rn(half, x), dt), du, __fmul2_rn(half, __fadd2_rn(one, t)));
}

__device__ __forceinline__ size_t act_index(int Xp, int Yp, int x, int y, int z, int h) {
  return ((((size_t)z * Yp + y) * 2 + h) * Xp + x) * 8;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// 16 channels of the interior site (x, y, z), whose first half's record is at q,
// and of its periodic ghost images (halo 1; an axis of one site has both) in a
// [.][.][2][Xp][8] buffer.  An image lies a whole period away along its axes.
// Those along x are predicated stores, those along y and z branches that a warp
// on one row takes as a whole.
__device__ __forceinline__ void store_act16(__nv_bfloat16* q, int Xp, int Yp, int nx, int ny,
                                            int nz, int x, int y, int z, const float (&a)[16],
                                            bool ghosts) {
  uint4 lo, hi;
  lo.x = pack_bf16x2(a[0], a[1]);   lo.y = pack_bf16x2(a[2], a[3]);
  lo.z = pack_bf16x2(a[4], a[5]);   lo.w = pack_bf16x2(a[6], a[7]);
  hi.x = pack_bf16x2(a[8], a[9]);   hi.y = pack_bf16x2(a[10], a[11]);
  hi.z = pack_bf16x2(a[12], a[13]); hi.w = pack_bf16x2(a[14], a[15]);
  auto put = [&](__nv_bfloat16* r) {
    *reinterpret_cast<uint4*>(r) = lo;
    *reinterpret_cast<uint4*>(r + Xp * 8) = hi;
  };
  auto row = [&](__nv_bfloat16* r) {
    put(r);
    if (!ghosts) return;
    if (x == 0) put(r + nx * 8);
    if (x == nx - 1) put(r - nx * 8);
  };
  row(q);
  if (!ghosts) return;
  const bool y0 = y == 0, y1 = y == ny - 1, z0 = z == 0, z1 = z == nz - 1;
  if (!(y0 || y1 || z0 || z1)) return;
  const ptrdiff_t sy = (ptrdiff_t)ny * Xp * 16, sz = (ptrdiff_t)nz * Yp * Xp * 16;
  if (y0) row(q + sy);
  if (y1) row(q - sy);
  if (z0) {
    row(q + sz);
    if (y0) row(q + sz + sy);
    if (y1) row(q + sz - sy);
  }
  if (z1) {
    row(q - sz);
    if (y0) row(q - sz + sy);
    if (y1) row(q - sz - sy);
  }
}

__device__ __forceinline__ void set_abort(int* status, volatile int* flag, int code) {
  *flag = 1;
  atomicExch(status, code);
}

// --------------------------------------------------------------------------
// Forward / dgrad convolution.

// Global data an epilogue reads besides the accumulators: the stored
// pre-activation (dgrad) or the solver's psi (residual).  Loaded for every
// row of a plane before any of them is computed, so the latencies overlap.
struct EpiAux {
  uint4 lo, hi;
  float2 psi;
};

__device__ __forceinline__ size_t psi_index(const ConvParams& p, int x, int y, int z) {
  return ((size_t)(z + p.psi_gh) * p.psi_Ny + (y + p.psi_gh)) * p.psi_Nx + (x + p.psi_gh);
}

// off: the site's element offset in an activation buffer.
template <int EPI>
__device__ __forceinline__ void epi_load(const ConvParams& p, int x, int y, int z, size_t off,
                                         EpiAux& a) {
  if (EPI == EPI_DGELU) {
    a.lo = *reinterpret_cast<const uint4*>(p.pre_in + off);
    a.hi = *reinterpret_cast<const uint4*>(p.pre_in + off + p.Xp * 8);
  } else if (EPI == EPI_RESID) {
    a.psi = reinterpret_cast<const float2*>(p.psi)[psi_index(p, x, y, z)];
  }
}

__device__ __forceinline__ float4 lds_float4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}

// bias: shared-memory address of the 16 biases.
template <int EPI>
__device__ __forceinline__ void conv_epilogue(const ConvParams& p, const float (&acc)[16],
                                              uint32_t bias, const EpiAux& aux, int x, int y,
                                              int z, size_t off) {
  if (EPI == EPI_GELU || EPI == EPI_GELU_PRE) {
    float pre[16], a[16];
    float4 b;
#pragma unroll
    for (int c = 0; c < 16; c += 2) {
      if (c % 4 == 0) b = lds_float4(bias + c * 4);
      const float2 v = __fadd2_rn(make_float2(acc[c], acc[c + 1]),
                                  c % 4 == 0 ? make_float2(b.x, b.y) : make_float2(b.z, b.w));
      const float2 g = gelu2(v);
      pre[c] = v.x;
      pre[c + 1] = v.y;
      a[c] = g.x;
      a[c + 1] = g.y;
    }
    if (EPI == EPI_GELU_PRE) store_act16(p.pre_out + off, p.Xp, p.Yp, p.nx, p.ny, p.nz, x, y, z, pre, false);
    store_act16(p.act_out + off, p.Xp, p.Yp, p.nx, p.ny, p.nz, x, y, z, a, true);
  } else if (EPI == EPI_DGELU) {
    float g[16];
    const uint32_t w[8] = {aux.lo.x, aux.lo.y, aux.lo.z, aux.lo.w, aux.hi.x, aux.hi.y, aux.hi.z, aux.hi.w};
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
      const float2 r = __fmul2_rn(make_float2(acc[2 * i], acc[2 * i + 1]), gelu_grad2(f));
      g[2 * i] = r.x;
      g[2 * i + 1] = r.y;
    }
    store_act16(p.act_out + off, p.Xp, p.Yp, p.nx, p.ny, p.nz, x, y, z, g, true);
  } else if (EPI == EPI_DELTA) {
    const size_t s = ((size_t)z * p.ny + y) * p.nx + x;
    const float4 b = lds_float4(bias);
    reinterpret_cast<float2*>(p.delta)[s] =
        make_float2((acc[0] + b.x) * p.out_scale, (acc[1] + b.y) * p.out_scale);
  } else {  // EPI_RESID: psi += delta on the solver's field, its periodic ghosts too
    const float4 b = lds_float4(bias);
    float2 v = aux.psi;
    v.x += (acc[0] + b.x) * p.out_scale;
    v.y += (acc[1] + b.y) * p.out_scale;
    float2* f = reinterpret_cast<float2*>(p.psi);
    int gx[2], gy[2], gz[2];
    ghost_targets(x, p.nx, 1, p.psi_gh, gx[0], gx[1]);
    ghost_targets(y, p.ny, 1, p.psi_gh, gy[0], gy[1]);
    ghost_targets(z, p.nz, 1, p.psi_gh, gz[0], gz[1]);
    auto row = [&](int yt, int zt) {
      float2* r = f + psi_index(p, 0, yt, zt);
      r[x] = v;
      if (gx[0] != NO_GHOST) r[gx[0]] = v;
      if (gx[1] != NO_GHOST) r[gx[1]] = v;
    };
    auto plane = [&](int zt) {
      row(y, zt);
      if (gy[0] != NO_GHOST) row(gy[0], zt);
      if (gy[1] != NO_GHOST) row(gy[1], zt);
    };
    plane(z);
    if (gz[0] != NO_GHOST) plane(gz[0]);
    if (gz[1] != NO_GHOST) plane(gz[1]);
  }
}

template <int EPI, int CO>
__global__ void __launch_bounds__(F_THREADS, 1)
conv_fwd_kernel(const __grid_constant__ ConvParams p) {
  constexpr int CW = OutShape<CO>::CW, NB = OutShape<CO>::NB, WTB = OutShape<CO>::WTB;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // 4 KB after the ring: an A operand of 128 sites reads past shorter rows (what
  // it finds there goes to accumulator lanes past the row, which nothing reads)
  unsigned char* wsm = ring + FSLOTS * p.slot_bytes + 4096;
  uint64_t* full = reinterpret_cast<uint64_t*>(wsm + W_TILES * WTB);
  uint64_t* empty = full + FSLOTS;
  uint64_t* accf = empty + FSLOTS;  // [2] MMAs of one input plane into a half done
  uint64_t* acce = accf + 2;        // [2] a half's finished output plane is drained
  uint64_t* drain = acce + 2;
  uint64_t* wfull = drain + 1;      // the weights have arrived
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(wfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* bias_s = reinterpret_cast<float*>(full + F_BIAS_OFF / 8);  // [16]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < FSLOTS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int h = 0; h < 2; h++) {
      mbar_init(&accf[h], 1);
      mbar_init(&acce[h], F_EPI_WARPS / 2);
    }
    mbar_init(drain, 1);
    mbar_init(wfull, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  fence_proxy_async();
  if (warp == 1) tc::tmem_alloc(smem_u32(tmem_holder), F_TMEM_COLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  const uint64_t lim = p.wait_limit_ns;
  const uint32_t row_bytes = (uint32_t)p.Xp * 16;
  if (warp >= 2) {  // the whole allocation starts at zero
    const int q = warp & 3;
    for (int a = (warp - 2) >> 2; a < (int)F_TMEM_COLS / 16; a += HROWS)
      tc::st_32x32b_x16_zero(tmem + ((uint32_t)(32 * q) << 16) + a * 16);
    tc::wait_st();
  }
  after_previous();
  if (threadIdx.x < 16) bias_s[threadIdx.x] = p.bias ? p.bias[threadIdx.x] : 0.0f;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();

  if (warp == 0) {
    if (tc::elect_one()) {
      const size_t row_elems = (size_t)p.Hin * p.Xp * 8;
      const size_t plane_elems = (size_t)p.Yp * row_elems;
      mbar_arrive_expect_tx(wfull, W_TILES * WTB);
      tc::bulk_load(smem_u32(wsm), p.w, W_TILES * WTB, smem_u32(wfull));
      uint32_t g = 0;
      for (int it = blockIdx.x; it < p.nitems && !*abort_flag; it += gridDim.x) {
        const int slab = it % p.nslab, zc = it / p.nslab;
        const int y0 = slab * TYF, z0 = zc * p.zchunk;
        const int nout = min(z0 + p.zchunk, p.nz) - z0;
        for (int pl = 0; pl < nout + 2; pl++, g++) {
          const uint32_t slot = g % FSLOTS, cyc = g / FSLOTS;
          if (cyc > 0 && !mbar_wait_bounded(&empty[slot], (cyc - 1) & 1, lim)) {
            set_abort(p.status, abort_flag, 1);
            break;
          }
          // rows y0 .. y0+TYF+1 (padded) of plane z0+pl: one contiguous range
          const uint32_t bytes = (uint32_t)min(TYF + 2, p.Yp - y0) * (uint32_t)(row_elems * 2);
          mbar_arrive_expect_tx(&full[slot], bytes);
          tc::bulk_load(smem_u32(ring + slot * p.slot_bytes),
                        p.in + (size_t)(z0 + pl) * plane_elems + (size_t)y0 * row_elems, bytes,
                        smem_u32(&full[slot]));
        }
      }
      const uint32_t first = g > FSLOTS ? g - FSLOTS : 0;
      for (uint32_t q = first; q < g; q++)
        if (!mbar_wait_bounded(&full[q % FSLOTS], (q / FSLOTS) & 1, lim)) {
          set_abort(p.status, abort_flag, 1);
          break;
        }
      if (!mbar_wait_bounded(wfull, 0, lim)) set_abort(p.status, abort_flag, 1);
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr int BROW = OSLOTS * CW;  // B rows / D columns per output row
      const uint32_t idesc1 = tc::idesc_bf16_f32(128, OutShape<CO>::n_of(1), false, false);
      const uint32_t idesc2 = tc::idesc_bf16_f32(128, OutShape<CO>::n_of(2), false, false);
      const uint32_t idesc3 = tc::idesc_bf16_f32(128, OutShape<CO>::n_of(3), false, false);
      const uint32_t lbo_a = p.Hin == 2 ? row_bytes : 0;
      const uint32_t ring_s = smem_u32(ring), w_s = smem_u32(wsm);
      const uint64_t bdesc0 = tc::smem_desc(w_s, NB * 16, 128);
      const uint64_t adesc0 = tc::smem_desc(ring_s, lbo_a, 128);
      const uint32_t row_step = (uint32_t)p.Hin * row_bytes;
      uint32_t g = 0;  // input planes
      if (!mbar_wait_bounded(wfull, 0, lim)) set_abort(p.status, abort_flag, 1);
      for (int it = blockIdx.x; it < p.nitems && !*abort_flag; it += gridDim.x) {
        const int slab = it % p.nslab, zc = it / p.nslab;
        const int y0 = slab * TYF, z0 = zc * p.zchunk;
        const int nout = min(z0 + p.zchunk, p.nz) - z0;
        const int nin = min(TYF, p.ny - y0) + 2;  // input rows y0-1 .. y0+nrows
        for (int t = 0; t < nout + 2 && !*abort_flag; t++, g++) {
          const int j = z0 - 1 + t;  // input plane (may be -1: its ghost plane)
          bool ok = mbar_wait_bounded(&full[g % FSLOTS], (g / FSLOTS) & 1, lim);
          if (ok && g > 0) ok = mbar_wait_bounded(&acce[0], (g - 1) & 1, lim);
          if (!ok) {
            set_abort(p.status, abort_flag, 1);
            break;
          }
          tc::fence_after_sync();
          const uint64_t ab = adesc0 + ((g % FSLOTS) * p.slot_bytes >> 4);
          const uint64_t bb = bdesc0 + (uint64_t)(((j + 3) % 3) * 3 * WTB / 16);
          bool second = false;  // the second half's accumulators are free
#pragma unroll
          for (int i = 0; i < TYF + 2; i++) {
            // input row i feeds slab rows i-2 .. i: keep those inside [0, TYF)
            const int jlo = i < 2 ? 2 - i : 0;
            const int jhi = i > TYF - 1 ? TYF + 1 - i : 2;
            const int cnt = jhi - jlo + 1;
            const uint32_t idesc = cnt == 3 ? idesc3 : (cnt == 2 ? idesc2 : idesc1);
            const uint32_t d = tmem + (uint32_t)((i - 2 + jlo) * BROW);
            const uint64_t b = bb + (uint64_t)(jlo * BROW * 16 / 16);
            if (!second && (i - 2 + jlo) * BROW + OutShape<CO>::n_of(cnt) > HROWS * BROW) {
              if (g > 0 && !mbar_wait_bounded(&acce[1], (g - 1) & 1, lim)) {
                ok = false;
                break;
              }
              tc::fence_after_sync();
              second = true;
            }
            if (i < nin) {
#pragma unroll
              for (int dx = 0; dx < 3; dx++)
                tc::mma_bf16(d, ab + ((i * row_step + dx * 16) >> 4), b + (uint64_t)(dx * WTB / 16),
                             idesc, 1u);
            }
            if (i == HROWS + 1) tc::commit(smem_u32(&accf[0]));  // its rows have all they get
          }
          if (!ok) {
            set_abort(p.status, abort_flag, 1);
            break;
          }
          tc::commit(smem_u32(&accf[1]));
          tc::commit(smem_u32(&empty[g % FSLOTS]));
        }
      }
      tc::commit(smem_u32(drain));
      if (!mbar_wait_bounded(drain, 0, lim)) set_abort(p.status, abort_flag, 1);
    }
  } else {
    // a warp has two rows of one half, HROWS / 2 apart; the warps of one half
    // compute while those of the other wait or drain
    const int q = warp & 3, h = ((warp - 2) >> 2) & 1, r0 = h * HROWS + ((warp - 2) >> 3);
    constexpr int KROW = HROWS / 2;
    const int x = 32 * q + lane;
    const uint32_t bias = smem_u32(bias_s);
    const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(r0 * OSLOTS * CW);
    const size_t plane = (size_t)p.Yp * p.Xp * 16;  // of an activation buffer
    uint32_t e = 0;  // input planes
    for (int it = blockIdx.x; it < p.nitems && !*abort_flag; it += gridDim.x) {
      const int slab = it % p.nslab, zc = it / p.nslab;
      const int y0 = slab * TYF + r0, z0 = zc * p.zchunk;
      const int nout = min(z0 + p.zchunk, p.nz) - z0;
      const uint32_t off0 = (uint32_t)((y0 + 1) * 2 * p.Xp + x + 1) * 8;
      bool stop = false;
      for (int t = 0; t < nout + 2 && !stop; t++, e++) {
        const int zo = z0 - 2 + t;  // output plane finished by input plane zo + 1
        const uint32_t so = (uint32_t)((zo + 3) % 3);
        const bool last = t == nout + 1;
        EpiAux aux[2];
        float v[2][16];
        bool mine[2];
        size_t off[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          mine[k] = zo >= z0 && y0 + k * KROW < p.ny && x < p.nx;
          off[k] = (size_t)(zo + 1) * plane + off0 + (uint32_t)(k * KROW * p.Xp * 16);
          if (mine[k]) epi_load<EPI>(p, x, y0 + k * KROW, zo, off[k], aux[k]);
        }
        if (!mbar_wait_bounded(&accf[h], e & 1, lim)) {
          set_abort(p.status, abort_flag, 1);
          stop = true;
          break;
        }
        tc::fence_after_sync();
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const uint32_t tr = tq + (uint32_t)(k * KROW * OSLOTS * CW);
          if (zo >= z0 && y0 + k * KROW < p.ny) {
            if (CW == 16) tc::ld_32x32b_x16(tr + so * CW, v[k]);
            else tc::ld_32x32b_x2(tr + so * CW, v[k]);
          }
#pragma unroll
          for (int ds = 0; ds < 3; ds++) {
            if (ds > 0 && !last) break;  // at the chunk's end: junk of the planes past it
            const uint32_t col = (so + ds) % 3 * CW;
            if (CW == 16) tc::st_32x32b_x16_zero(tr + col);
            else tc::st_32x32b_x2_zero(tr + col);
          }
        }
        tc::wait_st();
        tc::fence_before_sync();
        __syncwarp();
        // the next plane's MMAs run under the arithmetic
        if (lane == 0) mbar_arrive(&acce[h]);
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (mine[k])
            conv_epilogue<EPI>(p, v[k], bias, aux[k], x, y0 + k * KROW, zo, off[k]);
      }
      if (stop) break;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, F_TMEM_COLS);
  }
}

// --------------------------------------------------------------------------
// Weight gradient.

// The role and the share of (slab, plane) positions, planes running fastest, of
// one CTA.
struct WShare {
  int t0, nt;      // first (dz, dx) tap and their number
  int dz0;         // its taps need X planes z + dz0 and z + dz0 + 1 (padded)
  int pos, end;
};
__device__ __forceinline__ WShare wgrad_share(const WgradParams& p) {
  const bool r0 = (int)blockIdx.x < p.role0;
  const int n = r0 ? p.role0 : (int)gridDim.x - p.role0;
  const int i = r0 ? (int)blockIdx.x : (int)blockIdx.x - p.role0;
  const long long total = (long long)p.nslab * p.nz;
  WShare s;
  s.t0 = r0 ? 0 : W_TAPS0;
  s.nt = r0 ? W_TAPS0 : 9 - W_TAPS0;
  s.dz0 = s.t0 / 3;
  s.pos = (int)(i * total / n);
  s.end = (int)((i + 1) * total / n);
  return s;
}

__global__ void __launch_bounds__(W_THREADS, 1) conv_wgrad_kernel(const __grid_constant__ WgradParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* xring = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* dring = xring + WSLOTS * p.xslot_bytes;
  uint64_t* xfull = reinterpret_cast<uint64_t*>(dring + DSLOTS * p.dslot_bytes);
  uint64_t* xempty = xfull + WSLOTS;
  uint64_t* dfull = xempty + WSLOTS;
  uint64_t* dempty = dfull + DSLOTS;
  uint64_t* drain = dempty + DSLOTS;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WShare sh = wgrad_share(p);
  const bool bias = (int)blockIdx.x < p.role0;  // this role sums the bias gradient
  if (threadIdx.x == 0) {
    for (int s = 0; s < WSLOTS; s++) {
      mbar_init(&xfull[s], 1);
      mbar_init(&xempty[s], 1);
    }
    for (int s = 0; s < DSLOTS; s++) {
      mbar_init(&dfull[s], 1);
      mbar_init(&dempty[s], bias ? 1 + W_EPI_WARPS : 1);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) tc::tmem_alloc(smem_u32(tmem_holder), W_TMEM_COLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  const uint64_t lim = p.wait_limit_ns;
  const uint32_t row_bytes = (uint32_t)p.Xp * 16;
  if (warp >= 2) {  // the accumulators start at zero (every MMA accumulates)
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    for (int a = 0; a < W_TAPS0 * W_NCOL / 16; a++) tc::st_32x32b_x16_zero(tq + a * 16);
    tc::wait_st();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  after_previous();

  if (warp == 0) {
    if (tc::elect_one()) {
      const size_t row_elems = (size_t)2 * p.Xp * 8;
      const size_t plane_elems = (size_t)p.Yp * row_elems;
      uint32_t gx = 0, gd = 0;
      auto load_x = [&](int y0, int zpad) -> bool {
        const uint32_t slot = gx % WSLOTS, cyc = gx / WSLOTS;
        if (cyc > 0 && !mbar_wait_bounded(&xempty[slot], (cyc - 1) & 1, lim)) return false;
        const uint32_t bytes = (uint32_t)min(XROWS, p.Yp - y0) * (uint32_t)(row_elems * 2);
        mbar_arrive_expect_tx(&xfull[slot], bytes);
        tc::bulk_load(smem_u32(xring + slot * p.xslot_bytes),
                      p.x + (size_t)zpad * plane_elems + (size_t)y0 * row_elems, bytes,
                      smem_u32(&xfull[slot]));
        gx++;
        return true;
      };
      auto load_d = [&](int y0, int nrows, int zpad) -> bool {
        const uint32_t slot = gd % DSLOTS, cyc = gd / DSLOTS;
        if (cyc > 0 && !mbar_wait_bounded(&dempty[slot], (cyc - 1) & 1, lim)) return false;
        const uint32_t bytes = (uint32_t)nrows * (uint32_t)(row_elems * 2);
        mbar_arrive_expect_tx(&dfull[slot], bytes);
        tc::bulk_load(smem_u32(dring + slot * p.dslot_bytes),
                      p.dy + (size_t)zpad * plane_elems + (size_t)(y0 + 1) * row_elems, bytes,
                      smem_u32(&dfull[slot]));
        gd++;
        return true;
      };
      bool ok = true;
      for (int pos = sh.pos; pos < sh.end && ok && !*abort_flag;) {
        const int slab = pos / p.nz, z0 = pos - slab * p.nz;
        const int len = min(p.nz - z0, sh.end - pos);
        const int y0 = slab * TYW, nrows = min(TYW, p.ny - y0);
        ok = load_x(y0, z0 + sh.dz0);
        for (int o = 0; o < len && ok && !*abort_flag; o++)
          ok = load_x(y0, z0 + o + sh.dz0 + 1) && load_d(y0, nrows, z0 + o + 1);
        pos += len;
      }
      if (!ok) set_abort(p.status, abort_flag, 1);
      const uint32_t fx = gx > WSLOTS ? gx - WSLOTS : 0;
      for (uint32_t q = fx; q < gx; q++)
        if (!mbar_wait_bounded(&xfull[q % WSLOTS], (q / WSLOTS) & 1, lim)) {
          set_abort(p.status, abort_flag, 1);
          break;
        }
      const uint32_t fd = gd > DSLOTS ? gd - DSLOTS : 0;
      for (uint32_t q = fd; q < gd; q++)
        if (!mbar_wait_bounded(&dfull[q % DSLOTS], (q / DSLOTS) & 1, lim)) {
          set_abort(p.status, abort_flag, 1);
          break;
        }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      const uint32_t xring_s = smem_u32(xring), dring_s = smem_u32(dring);
      uint32_t gx0 = 0, gd = 0, xw = 0;
      const int nxc = p.nx / 16;
      for (int pos = sh.pos; pos < sh.end && !*abort_flag;) {
        const int slab = pos / p.nz, z0 = pos - slab * p.nz;
        const int len = min(p.nz - z0, sh.end - pos);
        const int nrows = min(TYW, p.ny - slab * TYW);
        const uint32_t idesc = tc::idesc_bf16_f32(128, 16 * nrows, true, true);
        for (int o = 0; o < len && !*abort_flag; o++, gd++) {
          bool ok = true;
          while (ok && xw < gx0 + o + 2) {
            ok = mbar_wait_bounded(&xfull[xw % WSLOTS], (xw / WSLOTS) & 1, lim);
            if (ok) xw++;
          }
          ok = ok && mbar_wait_bounded(&dfull[gd % DSLOTS], (gd / DSLOTS) & 1, lim);
          if (!ok) {
            set_abort(p.status, abort_flag, 1);
            break;
          }
          tc::fence_after_sync();
          const uint32_t xb0 = xring_s + ((gx0 + o) % WSLOTS) * p.xslot_bytes;
          const uint32_t xb1 = xring_s + ((gx0 + o + 1) % WSLOTS) * p.xslot_bytes;
          const uint32_t db = dring_s + (gd % DSLOTS) * p.dslot_bytes;
          for (int xc = 0; xc < nxc; xc++) {
            const uint64_t bdesc =
                tc::smem_desc(db + (uint32_t)(1 + 16 * xc) * 16, 128, row_bytes);
#pragma unroll
            for (int a = 0; a < W_TAPS0; a++) {
              if (a >= sh.nt) break;
              const int t = sh.t0 + a, dz = t / 3, dx = t - 3 * dz;
              const uint32_t xb = dz == sh.dz0 ? xb0 : xb1;
              const uint64_t adesc =
                  tc::smem_desc(xb + (uint32_t)(16 * xc + dx) * 16, 128, row_bytes);
              tc::mma_bf16(tmem + a * W_NCOL, adesc, bdesc, idesc, 1u);
            }
          }
          tc::commit(smem_u32(&xempty[(gx0 + o) % WSLOTS]));
          tc::commit(smem_u32(&dempty[gd % DSLOTS]));
        }
        if (*abort_flag) break;
        tc::commit(smem_u32(&xempty[(gx0 + len) % WSLOTS]));
        gx0 += len + 1;
        pos += len;
      }
      tc::commit(smem_u32(drain));
      if (!mbar_wait_bounded(drain, 0, lim)) set_abort(p.status, abort_flag, 1);
    }
  } else if (bias) {
    // bias gradient: warp w sums the (row, half) runs 4 k + w of every dY tile
    // (its half is w & 1), lanes along x
    const int w = warp - 2;
    float acc[8] = {};
    uint32_t gd = 0;
    for (int pos = sh.pos; pos < sh.end && !*abort_flag;) {
      const int slab = pos / p.nz, z0 = pos - slab * p.nz;
      const int len = min(p.nz - z0, sh.end - pos);
      const int nrows = min(TYW, p.ny - slab * TYW);
      for (int o = 0; o < len && !*abort_flag; o++, gd++) {
        if (!mbar_wait_bounded(&dfull[gd % DSLOTS], (gd / DSLOTS) & 1, lim)) {
          set_abort(p.status, abort_flag, 1);
          break;
        }
        const unsigned char* d = dring + (gd % DSLOTS) * p.dslot_bytes;
        for (int q = w; q < 2 * nrows; q += 4)
          for (int x = lane; x < p.nx; x += 32) {
            const uint4 v = *reinterpret_cast<const uint4*>(d + (size_t)q * row_bytes + (x + 1) * 16);
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[c]));
              acc[2 * c] += f.x;
              acc[2 * c + 1] += f.y;
            }
          }
        __syncwarp();
        if (lane == 0) mbar_arrive(&dempty[gd % DSLOTS]);
      }
      pos += len;
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    }
    // (through the holder's spare words: 4 warps x 8 floats)
    float* bs = reinterpret_cast<float*>(tmem_holder + 4);
    if (lane == 0)
#pragma unroll
      for (int c = 0; c < 8; c++) bs[8 * w + c] = acc[c];
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const bool good = !*abort_flag;
  float* red = reinterpret_cast<float*>(xring);  // [8 xrow][3 dy][16 co][16 ci], the ring is idle
  for (int a = 0; a < sh.nt; a++) {
    if (warp >= 2) {
      const int q = warp & 3, xrow = 2 * q + (lane >> 4), ci = lane & 15;
      const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16) + a * W_NCOL;
#pragma unroll
      for (int jj = -2; jj < 2; jj++) {  // dY rows this warp's two X rows meet
        const int j = 2 * q + jj;
        if (j < 0 || j >= TYW) continue;
        float v[16];
        tc::ld_32x32b_x16(tq + j * CH, v);
        const int dy = xrow - j;
        if (dy >= 0 && dy < 3)
#pragma unroll
          for (int co = 0; co < CH; co++) red[((xrow * 3 + dy) * CH + co) * CH + ci] = v[co];
      }
    }
    __syncthreads();
    float* out = p.partials + (size_t)blockIdx.x * W_PART + a * 3 * CH * CH;
    for (int i = threadIdx.x; i < 3 * CH * CH; i += W_THREADS) {
      const int dy = i / (CH * CH);
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < TYW; j++) t += red[(j + dy) * 3 * CH * CH + i];
      out[i] = good ? t : 0.f;
    }
    __syncthreads();
  }
  if (bias && threadIdx.x < CH) {
    const float* bs = reinterpret_cast<const float*>(tmem_holder + 4);
    const int h = threadIdx.x >> 3, c = threadIdx.x & 7;
    p.bpartials[blockIdx.x * CH + threadIdx.x] = good ? bs[8 * h + c] + bs[8 * (h + 2) + c] : 0.f;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, W_TMEM_COLS);
  }
}

// --------------------------------------------------------------------------
// Element-wise and reduction kernels.

// Solver field (gh ghosts, pitches Nx, Ny; complex of TS) -> first-layer input
// (channels Re, Im, 0, ...; H halves), ghosts included.  Every padded site
// reads its periodic interior source (the solver keeps only the face ghosts
// a star stencil needs, not edges and corners).  One warp per padded (y, z) row,
// four records a lane in flight; bound by the 16 (or 32) bytes written per site
// (128^3: 12.2 us with a block of 128 threads per row of 130, 11.1 so).
template <typename TS>
__global__ void pack_input_kernel(const TS* psi, int Nx, int Ny, int gh, int nx, int ny, int nz,
                                  __nv_bfloat16* act, int H) {
  const int Xp = nx + 2, Yp = ny + 2, rows = Yp * (nz + 2);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  using V = typename VT<TS>::T;
  after_previous();
  for (int row = blockIdx.x * nw + (threadIdx.x >> 5); row < rows; row += gridDim.x * nw) {
    const int yp = row % Yp, zp = row / Yp;
    const int y = yp == 0 ? ny - 1 : (yp == ny + 1 ? 0 : yp - 1);
    const int z = zp == 0 ? nz - 1 : (zp == nz + 1 ? 0 : zp - 1);
    const V* src = reinterpret_cast<const V*>(psi) + ((size_t)(z + gh) * Ny + (y + gh)) * Nx + gh;
    uint4* dst = reinterpret_cast<uint4*>(act) + (size_t)row * H * Xp;
    for (int x0 = lane; x0 < Xp; x0 += 128) {
      V v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int xp = x0 + 32 * q;
        if (xp < Xp) v[q] = src[xp == 0 ? nx - 1 : (xp == nx + 1 ? 0 : xp - 1)];
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int xp = x0 + 32 * q;
        if (xp >= Xp) break;
        dst[xp] = make_uint4(pack_bf16x2((float)v[q].x, (float)v[q].y), 0, 0, 0);
        if (H == 2) dst[Xp + xp] = zero;
      }
    }
  }
}

// Loss of one training pair and the gradient with respect to the last
// layer's output: e = u + delta - target, loss = sum |e|^2 / n,
// dL/d(out_c) = 2 e_c out_scale / n into channels 0, 1 of g (others 0).
template <typename TS, typename TT>
__global__ void loss_kernel(const float* delta, const TS* u, int Nx, int Ny, int gh,
                            const TT* target, int nx, int ny, int nz, float out_scale, __nv_bfloat16* g,
                            double* partials) {
  __shared__ double red[32];
  const int Xp = nx + 2, Yp = ny + 2;
  const size_t n = (size_t)nx * ny * nz;
  const double inv_n = 1.0 / (double)n;
  double acc = 0.0;
  after_previous();
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
       s += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(s % nx);
    const size_t t = s / nx;
    const int y = (int)(t % ny), z = (int)(t / ny);
    const size_t q = ((size_t)(z + gh) * Ny + (y + gh)) * Nx + (x + gh);
    const double er = (double)u[2 * q] + (double)delta[2 * s] - (double)target[2 * s];
    const double ei = (double)u[2 * q + 1] + (double)delta[2 * s + 1] - (double)target[2 * s + 1];
    acc += er * er + ei * ei;
    float a[16] = {};
    a[0] = (float)(2.0 * er * inv_n * out_scale);
    a[1] = (float)(2.0 * ei * inv_n * out_scale);
    store_act16(g + act_index(Xp, Yp, x + 1, y + 1, z + 1, 0), Xp, Yp, nx, ny, nz, x, y, z, a, true);
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    partials[blockIdx.x] = t;
  }
}

// dW[tap][co][ci] (fp32) of one layer from the wgrad partials (one block per
// tap; four groups of threads take every fourth CTA of the tap's role, added in
// a fixed order), and db from the channel sums (the last block).
__global__ void __launch_bounds__(1024) grad_finalize_kernel(const float* wpart, int nblk,
                                                              int role0, const float* bpart,
                                                              float* dw, float* db) {
  __shared__ float s[4][256];
  const int c = threadIdx.x & 255, g = threadIdx.x >> 8;
  after_previous();
  if (blockIdx.x == NTAP) {
    if (threadIdx.x < 16) {
      float t = 0.f;
      for (int b = 0; b < role0; b++) t += bpart[b * 16 + threadIdx.x];
      db[threadIdx.x] = t;
    }
    return;
  }
  const int tap = blockIdx.x, dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
  const int zx = dz * 3 + dx;
  const int a = zx < W_TAPS0 ? zx : zx - W_TAPS0;
  const int b0 = zx < W_TAPS0 ? 0 : role0, b1 = zx < W_TAPS0 ? role0 : nblk;
  float t = 0.f;
#pragma unroll 8
  for (int b = b0 + g; b < b1; b += 4) t += wpart[(size_t)b * W_PART + (a * 3 + dy) * 256 + c];
  s[g][c] = t;
  __syncthreads();
  if (g == 0) dw[tap * 256 + c] = (s[0][c] + s[1][c]) + (s[2][c] + s[3][c]);
}

// Adam (Kingma & Ba) on the masked parameters of all layers.
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v,
                            const unsigned char* __restrict__ mask, int n, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !mask[i]) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// fp32 weights [L][27][16 co][16 ci] -> bf16 B tiles [L][rot][dx][2 halves]
// [144 rows][8] (layout of the forward kernel's stacked B operand), K =
// input channel 8h + c.  The dgrad tiles hold the mirrored tap with co and
// ci exchanged (the adjoint convolution).
__global__ void pack_weights_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wf,
                                    __nv_bfloat16* __restrict__ wt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NLAYER * W_TILES * 2 * NSTACK * 8) return;
  const int c = i % 8, n = (i / 8) % NSTACK, h = (i / (8 * NSTACK)) % 2,
            tile = (i / (16 * NSTACK)) % W_TILES, l = i / (16 * NSTACK * W_TILES);
  const int rot = tile / 3, dx = tile % 3;
  const int co = n % 16, sj = n / 16, s = sj % 3, jrow = sj / 3;
  const int dz = 2 - (((s - rot + 1) % 3 + 3) % 3);
  const int tap = dz * 9 + (2 - jrow) * 3 + dx;
  const int k = 8 * h + c;
  const size_t base = (size_t)l * NTAP * 256;
  wf[i] = __float2bfloat16_rn(w[base + (size_t)tap * 256 + co * 16 + k]);
  wt[i] = __float2bfloat16_rn(w[base + (size_t)(NTAP - 1 - tap) * 256 + k * 16 + co]);
}

// The last layer (2 output channels) in the N = 32 layout of
// conv_fwd_kernel<*, 2>: [rot][dx][2 halves][32 rows][8], row n = (jrow*3 + s)*2
// + co for n < 18, zero rows above.
__global__ void pack_out2_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wf2) {
  constexpr int NB = OutShape<2>::NB;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= W_TILES * 2 * NB * 8) return;
  const int c = i % 8, n = (i / 8) % NB, h = (i / (8 * NB)) % 2, tile = i / (16 * NB);
  const int rot = tile / 3, dx = tile % 3;
  float v = 0.0f;
  if (n < 18) {
    const int co = n % 2, sj = n / 2, s = sj % 3, jrow = sj / 3;
    const int dz = 2 - (((s - rot + 1) % 3 + 3) % 3);
    const int tap = dz * 9 + (2 - jrow) * 3 + dx;
    v = w[(size_t)(NLAYER - 1) * NTAP * 256 + (size_t)tap * 256 + co * 16 + 8 * h + c];
  }
  wf2[i] = __float2bfloat16_rn(v);
}

// 2:1 restriction (2x2x2 average) of a solver field (gh ghosts) to a dense
// complex array of TO on the coarse grid.
template <typename TS, typename TO>
__global__ void restrict_kernel(const TS* __restrict__ f, int Nx, int Ny, int gh, int nxc,
                                int nyc, int nzc, TO* __restrict__ out) {
  const size_t n = (size_t)nxc * nyc * nzc;
  for (size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
       s += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(s % nxc);
    const size_t t = s / nxc;
    const int y = (int)(t % nyc), z = (int)(t / nyc);
    double re = 0.0, im = 0.0;
    for (int c = 0; c < 2; c++)
      for (int b = 0; b < 2; b++)
        for (int a = 0; a < 2; a++) {
          const size_t q =
              ((size_t)(2 * z + c + gh) * Ny + (2 * y + b + gh)) * Nx + (2 * x + a + gh);
          re += (double)f[2 * q];
          im += (double)f[2 * q + 1];
        }
    out[2 * s] = (TO)(0.125 * re);
    out[2 * s + 1] = (TO)(0.125 * im);
  }
}

}  // namespace cnn
}  // namespace gpe
