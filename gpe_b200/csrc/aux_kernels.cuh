// aux_kernels.cuh -- state transfer, scaling and reduction kernels.
#pragma once

#include <type_traits>

#include "device_utils.cuh"
#include "vec2.cuh"

namespace gpe {

// What a step hands back to the host (page-locked memory).
struct StepResult {
  double norm;
  int status;
};

struct Geom {
  int nx, ny, nz;  // interior
  int Nx, Ny;      // padded pitches
  int bcs;
  int gh;            // ghost layers on every side
  int zg_lo, zg_hi;  // fill z ghosts below / above locally
};

__device__ __forceinline__ size_t padded_index(const Geom& g, int i, int j,
                                               int k) {
  return ((size_t)(k + g.gh) * g.Ny + (size_t)(j + g.gh)) * g.Nx + (size_t)(i + g.gh);
}

// One warp per row of a field: rows r, r + (all warps), ... of `nrows`.
#define GPE_FOR_ROWS(r, nrows)                                        \
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   \
       r < (nrows); r += gridDim.x * (blockDim.x >> 5))

// Row copies with conversion: a pair of sites per lane where both rows start on
// a pair's alignment and the types agree (16-byte accesses for complex64), one
// site otherwise; four accesses in flight per lane.
template <typename TO, typename TI>
__device__ __forceinline__ void copy_row(TO* __restrict__ d, const TI* __restrict__ s, int n,
                                         int lane) {
  using VI = typename VT<TI>::T;
  int first = 0;
  if (std::is_same<TO, float>::value && std::is_same<TI, float>::value &&
      ((reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(s)) & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(s);
    float4* d4 = reinterpret_cast<float4*>(d);
#pragma unroll 4
    for (int i = lane; i < n / 2; i += 32) d4[i] = s4[i];
    first = n & ~1;
  }
#pragma unroll 4
  for (int i = first + lane; i < n; i += 32) {
    const VI v = reinterpret_cast<const VI*>(s)[i];
    st_one<TO>(d + 2 * i, (TO)v.x, (TO)v.y);
  }
}

// Dense interior array (any complex type TI) -> padded field of TS, with the
// boundary ghosts filled, edges included (the caller's halo exchange,
// src/gpe.f90:165-174).  One warp per padded row, which it gathers from the
// interior row it is an image of: every store is in row order.  HBM-bound.
template <typename TS, typename TI>
__global__ void unpack_kernel(const TI* __restrict__ src, TS* __restrict__ dst, Geom g) {
  using VI = typename VT<TI>::T;
  const int lane = threadIdx.x & 31;
  const int gh = g.gh, Nz = g.nz + 2 * gh;
  GPE_FOR_ROWS(r, g.Ny * Nz) {
    const int kp = r / g.Ny, jp = r - kp * g.Ny;
    const int k = kp - gh, j = jp - gh;
    if ((k < 0 && !g.zg_lo) || (k >= g.nz && !g.zg_hi)) continue;  // a neighbour sends these
    const int ks = ghost_source(k, g.nz, g.bcs), js = ghost_source(j, g.ny, g.bcs);
    const TI* s = src + 2 * ((size_t)ks * g.ny + js) * (size_t)g.nx;
    TS* d = dst + 2 * ((size_t)r * g.Nx + gh);
    copy_row<TS, TI>(d, s, g.nx, lane);
    if (lane < 2 * gh) {
      const int i = lane < gh ? lane - gh : g.nx + lane - gh;
      const VI v = reinterpret_cast<const VI*>(s)[ghost_source(i, g.nx, g.bcs)];
      st_one<TS>(d + 2 * i, (TS)v.x, (TS)v.y);
    }
  }
}

// Every boundary ghost of a field from its own interior, `depth` deep, edges
// included.  Rows that lie in the y or z ghosts are copied whole, one per
// warp; of the interior rows four per warp, eight lanes each, copy the
// x ghosts.
template <typename TS>
__device__ __forceinline__ void fill_ghost_rows(TS* f, const Geom& g, int depth,
                                                int block, int nblocks) {
  using V = typename VT<TS>::T;
  V* F = reinterpret_cast<V*>(f);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int warps = nblocks * nw, me = block * nw + (threadIdx.x >> 5);
  // whole rows: z-ghost planes (2 depth of ny + 2 depth rows), then the y-ghost
  // rows of the interior planes
  const int Yd = g.ny + 2 * depth, zrows = 2 * depth * Yd, whole = zrows + 2 * depth * g.nz;
  for (int r = me; r < whole; r += warps) {
    int j, k;
    if (r < zrows) {
      const int kk = r / Yd;
      k = kk < depth ? kk - depth : g.nz + kk - depth;
      j = r - kk * Yd - depth;
    } else {
      const int q = r - zrows;
      k = q / (2 * depth);
      const int jj = q - k * 2 * depth;
      j = jj < depth ? jj - depth : g.ny + jj - depth;
    }
    const size_t from =
        padded_index(g, 0, ghost_source(j, g.ny, g.bcs), ghost_source(k, g.nz, g.bcs));
    const size_t to = padded_index(g, 0, j, k);
    // 16 bytes a lane (rows start an even number of complexes in)
    constexpr int W = 16 / (int)sizeof(V);
    const float4* s4 = reinterpret_cast<const float4*>(F + from);
    float4* d4 = reinterpret_cast<float4*>(F + to);
#pragma unroll 4
    for (int i = lane; i < g.nx / W; i += 32) d4[i] = s4[i];
    if (W > 1 && lane < g.nx % W) F[to + g.nx - 1] = F[from + g.nx - 1];
    if (lane < 2 * depth) {
      const int i = lane < depth ? lane - depth : g.nx + lane - depth;
      F[to + i] = F[from + ghost_source(i, g.nx, g.bcs)];
    }
  }
  const int rows = g.ny * g.nz, sub = lane >> 3, l = lane & 7;
  const int i = l < depth ? l - depth : g.nx + l - depth;
  const int is = ghost_source(i, g.nx, g.bcs);
#pragma unroll 4
  for (int r4 = me; r4 * 4 < rows; r4 += warps) {
    const int r = r4 * 4 + sub;
    if (r < rows && l < 2 * depth) {
      const int k = r / g.ny, j = r - k * g.ny;
      const size_t at = padded_index(g, 0, j, k);
      F[at + i] = F[at + is];
    }
  }
}

template <typename TS>
__global__ void fill_ghosts_kernel(TS* f, Geom g, int depth) {
  after_previous();
  fill_ghost_rows<TS>(f, g, depth, blockIdx.x, gridDim.x);
}

// Fixed-order reduction of slot `slot` of the per-CTA partials by one block
// (sum, or max for op 1); the result is s[0] for every thread on return.
__device__ __forceinline__ void reduce_partials(const double* partials, int nblk,
                                                int slot, int op, double* s) {
  double a = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    const double v = partials[2 * (size_t)b + slot];
    a = op ? fmax(a, v) : a + v;
  }
  s[threadIdx.x] = a;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      const double v = s[threadIdx.x + w];
      s[threadIdx.x] = op ? fmax(s[threadIdx.x], v) : s[threadIdx.x] + v;
    }
    __syncthreads();
  }
}

// The end of a step in pairs, blocks of 1024 threads: block 0 reduces the norm
// as finalize_kernel does, the others fill the new psi's ghosts.
template <typename TS>
__global__ void __launch_bounds__(1024) ghosts_norm_kernel(TS* f, Geom g, int depth,
                                                            const double* partials, int nblk,
                                                            double scale, double* out,
                                                            double* series, StepResult* res,
                                                            const int* status) {
  __shared__ double s[1024];
  after_previous();
  if (blockIdx.x > 0) {
    fill_ghost_rows<TS>(f, g, depth, blockIdx.x - 1, gridDim.x - 1);
    return;
  }
  reduce_partials(partials, nblk, 0, 0, s);
  if (threadIdx.x == 0) {
    const double r = s[0] * scale;
    out[0] = r;
    if (series) *series = r;
    if (res) {
      res->norm = r;
      res->status = *status;
    }
  }
}

// The ghosts of one field per member of a batch, nblocks blocks a member (all along
// the grid's x, which has room for any number of members).
struct GhostRun {
  void* field;
  Geom g;
};
template <typename TS>
__global__ void batch_ghosts_kernel(const GhostRun* __restrict__ runs, int depth, int nblocks) {
  const int run = blockIdx.x / nblocks;
  const GhostRun r = runs[run];
  fill_ghost_rows<TS>(static_cast<TS*>(r.field), r.g, depth, blockIdx.x - run * nblocks, nblocks);
}

// Padded field -> dense interior array of TO, one warp per row.
template <typename TS, typename TO>
__global__ void pack_kernel(const TS* __restrict__ src, TO* __restrict__ dst, Geom g) {
  const int lane = threadIdx.x & 31;
  GPE_FOR_ROWS(r, g.ny * g.nz) {
    const int k = r / g.ny, j = r - k * g.ny;
    copy_row<TO, TS>(dst + 2 * (size_t)r * g.nx, src + 2 * padded_index(g, 0, j, k), g.nx, lane);
  }
}

// f[q] = op(f[q]) for a whole padded field: 16 bytes a thread and access, four
// in flight (rows are a multiple of four complexes).  128^3 complex64: 13.4 us one
// scalar at a time, 8.8 so.
template <typename TS, typename F>
__device__ __forceinline__ void for_scalars(TS* f, size_t nscalars, F op) {
  constexpr int W = 16 / (int)sizeof(TS);
  struct alignas(16) Vec {
    TS v[W];
  };
  Vec* fv = reinterpret_cast<Vec*>(f);
  const size_t n = nscalars / W, step = (size_t)gridDim.x * blockDim.x;
#pragma unroll 4
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += step) {
    Vec a = fv[q];
#pragma unroll
    for (int k = 0; k < W; k++) a.v[k] = op(a.v[k]);
    fv[q] = a;
  }
}

// renormalise (src/variables.f90:698-709): f = (sqrt(nn) f) / sqrt(norm)
// over the whole padded buffer, ghosts included (they stay exact copies).
template <typename TS>
__global__ void scale_kernel(TS* __restrict__ f, size_t nscalars, double snn,
                             double sn) {
  for_scalars(f, nscalars, [=](TS v) { return (TS)(((double)v * snn) / sn); });
}

// The same rescaling with the factor sqrt(target / current) read on the
// device (both norms left in device memory by earlier reductions).
template <typename TS>
__global__ void rescale_to_kernel(TS* f, size_t nscalars, const double* target,
                                  const double* current) {
  after_previous();
  const double s = sqrt(target[0] / current[0]);
  for_scalars(f, nscalars, [=](TS v) { return (TS)((double)v * s); });
}

// Weighted |psi|^2 per CTA into partials[2*blk] (get_norm without a stencil).
template <typename TS>
__global__ void norm_kernel(const TS* f, Geom g, const double* __restrict__ wx,
                            const double* __restrict__ wy, const double* __restrict__ wz,
                            double* partials) {
  __shared__ double s[32];
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  after_previous();
  GPE_FOR_ROWS(r, g.ny * g.nz) {
    const int k = r / g.ny, j = r - k * g.ny;
    const typename VT<TS>::T* row =
        reinterpret_cast<const typename VT<TS>::T*>(f) + padded_index(g, 0, j, k);
    const double wyj = wy[j], wzk = wz[k];
#pragma unroll 4
    for (int i = lane; i < g.nx; i += 32) {
      const typename VT<TS>::T v = row[i];
      const double a = (double)v.x, b = (double)v.y;
      acc += (wx[i] * wyj) * wzk * (a * a + b * b);
    }
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s[w];
    partials[2 * blockIdx.x] = t;
    partials[2 * blockIdx.x + 1] = 0.0;
  }
}

// Fixed-order reduction of partials[2*b + slot], b < nblk, by one CTA of
// 1024 threads.  op 0 = sum, 1 = max.  out[0] = result * scale, written to
// *series too when it is non-null, and with the status word to *res.
__global__ void finalize_kernel(const double* partials, int nblk, int slot, int op,
                                double scale, double* out, double* series, StepResult* res,
                                const int* status) {
  __shared__ double s[1024];
  after_previous();
  reduce_partials(partials, nblk, slot, op, s);
  if (threadIdx.x == 0) {
    const double r = s[0] * scale;
    out[0] = r;
    if (series) *series = r;
    if (res) {
      res->norm = r;
      res->status = *status;
    }
  }
}

// ---------------------------------------------------------------------------
// rkqs step control on the device (src/solve.f90:158-244).  A step is: begin
// (first attempt's dt), then attempts of the six Cash-Karp stages, each
// followed by rk45_control_kernel, until one is accepted.  The stage kernels
// read dt from `dt_r, dt_i, dt0_r, dt0_i` (contiguous, in this order).

struct DevTime {
  double dt_r, dt_i, dt0_r, dt0_i;  // this attempt's dt, the step's first dt
  double t, im_t;
  double errmax, did_r, did_i;       // last accepted attempt
  double errcon;                     // (5 / safety)^(1 / dt_increase)
  int attempts, underflow, halt, steps;  // halt: 0, or the GPE status code
  int real_time, pad;
};

// Sets the while node's condition (when it is one) and starts a step.
__global__ void rk45_begin_kernel(DevTime* T, cudaGraphConditionalHandle h, int use_cond) {
  if (threadIdx.x != 0) return;
  T->attempts = 0;
  T->dt0_r = T->dt_r;
  T->dt0_i = T->dt_i;
  if (use_cond) cudaGraphSetConditional(h, T->halt ? 0u : 1u);
}

// After an attempt whose error maximum (over all sites, already reduced
// across slabs) is scal[3] and whose trial-state norm is scal[0]: accept and
// advance t, dt (recording the step in the series), or shrink dt and retry.
// The arithmetic is the reference's: errmax <= 1 accepts; a rejected dt
// shrinks to max(safety dt errmax^dt_decrease, dt / 10) along the time
// direction; an accepted one grows to safety dt errmax^dt_increase, or 5 dt
// when errmax <= errcon; t advances by the accepted dt and im_t by the new
// |Im dt|.
__device__ void rk45_control(DevTime* T, const double* __restrict__ scal,
                             double* __restrict__ s_norm, double* __restrict__ s_dt,
                             int* __restrict__ s_att, int cap, cudaGraphConditionalHandle h,
                             int use_cond) {
  const double safety = 0.9, dt_decrease = -0.25, dt_increase = -0.20;
  if (T->halt) {
    if (use_cond) cudaGraphSetConditional(h, 0u);
    return;
  }
  const double errmax = scal[3];
  T->attempts += 1;
  T->errmax = errmax;
  bool done = false;
  // the error maximum skips NaN sites (fmax, as maxval does), so a state
  // that went non-finite shows in the fused norm of the trial state
  if (!isfinite(errmax) || !isfinite(scal[0])) {
    T->halt = 5;  // GPE_ERR_NAN
    done = true;
  } else if (errmax <= 1.0) {
    const double dr = T->dt_r, di = T->dt_i;
    double nr, ni;
    if (errmax > T->errcon) {
      const double f = pow(errmax, dt_increase);
      nr = (safety * dr) * f;
      ni = (safety * di) * f;
    } else {
      nr = 5.0 * dr;
      ni = 5.0 * di;
    }
    T->t = T->t + dr;
    T->did_r = dr;
    T->did_i = di;
    T->dt_r = nr;
    T->dt_i = ni;
    T->im_t = T->im_t + fabs(ni);
    const int k = T->steps;
    if (k < cap) {
      if (s_norm) s_norm[k] = scal[0];
      if (s_dt) s_dt[k] = dr;
      if (s_att) s_att[k] = T->attempts;
    }
    T->steps = k + 1;
    done = true;
  } else {
    const double dr = T->dt_r, di = T->dt_i;
    const double f = pow(errmax, dt_decrease);
    const double tr = (safety * dr) * f, ti = (safety * di) * f;
    const double mag = fmax(hypot(tr, ti), 0.1 * hypot(dr, di));
    if (T->real_time) {
      T->dt_r = mag;
      T->dt_i = 0.0;
      if (T->t + mag == T->t) T->underflow = 1;
    } else {
      T->dt_r = 0.0;
      T->dt_i = -mag;
    }
    if (T->attempts > 10000) {
      T->halt = 8;  // GPE_ERR_UNDERFLOW
      done = true;
    }
  }
  if (use_cond) cudaGraphSetConditional(h, done ? 0u : 1u);
}

__global__ void rk45_control_kernel(DevTime* T, const double* __restrict__ scal,
                                    double* __restrict__ s_norm, double* __restrict__ s_dt,
                                    int* __restrict__ s_att, int cap,
                                    cudaGraphConditionalHandle h, int use_cond) {
  if (threadIdx.x == 0) rk45_control(T, scal, s_norm, s_dt, s_att, cap, h, use_cond);
}

// A context with no neighbours: the attempt's two reductions (error maximum
// into scal[3], trial-state norm into scal[0], each as finalize_kernel forms
// it) and the step control in one launch of 1024 threads.
__global__ void rk45_reduce_control_kernel(const double* __restrict__ partials, int nblk,
                                           double err_scale, double norm_scale,
                                           double* __restrict__ scal, DevTime* T,
                                           double* __restrict__ s_norm,
                                           double* __restrict__ s_dt, int* __restrict__ s_att,
                                           int cap, cudaGraphConditionalHandle h,
                                           int use_cond) {
  __shared__ double s[1024];
  reduce_partials(partials, nblk, 1, 1, s);
  if (threadIdx.x == 0) scal[3] = s[0] * err_scale;
  __syncthreads();
  reduce_partials(partials, nblk, 0, 0, s);
  if (threadIdx.x == 0) {
    scal[0] = s[0] * norm_scale;
    rk45_control(T, scal, s_norm, s_dt, s_att, cap, h, use_cond);
  }
}

// Slab group: combine d_scal[idx] of n members in member order (sum, or max
// for op 1) and write the result back to every member.
__global__ void combine_scalars_kernel(double* const* __restrict__ scal, int n, int idx,
                                       int op) {
  if (threadIdx.x != 0) return;
  double a = scal[0][idx];
  for (int m = 1; m < n; m++) {
    const double v = scal[m][idx];
    a = op ? fmax(a, v) : a + v;
  }
  for (int m = 0; m < n; m++) scal[m][idx] = a;
}

// Batched ensembles: one CTA per run sums slot 0 of the partials of every
// work item of that run (fixed item order), times scale[r]; out[r] gets the
// value and, when series is non-null, series[r * cap + *counter] too.
__global__ void batch_finalize_kernel(const double* __restrict__ partials,
                                      const int* __restrict__ item_run, int nitems,
                                      const double* __restrict__ scale,
                                      double* __restrict__ out,
                                      double* __restrict__ series, int cap,
                                      const int* __restrict__ counter) {
  __shared__ double s[256];
  const int r = blockIdx.x;
  double a = 0.0;
  for (int i = threadIdx.x; i < nitems; i += blockDim.x)
    if (item_run[i] == r) a += partials[2 * (size_t)i];
  s[threadIdx.x] = a;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double v = s[0] * scale[r];
    out[r] = v;
    if (series) series[(size_t)r * cap + *counter] = v;
  }
}

__global__ void bump_counter_kernel(int* counter) { *counter = *counter + 1; }

// Failure-detection probe: waits, bounded by limit_ns, on an mbarrier phase
// that nothing completes, then records the timeout in *status exactly as
// the stage kernels do.
__global__ void wait_probe_kernel(unsigned long long limit_ns, int* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait_bounded(&bar, 0, limit_ns)) atomicExch(status, 1);
}

// A sum held as an unevaluated pair, about 106 bits: add() by Knuth's two-sum.
// hi alone is the plain sum, so an infinity or NaN shows there as it would.
struct Sum2 {
  double hi, lo;
  __device__ __forceinline__ double value() const { return isfinite(hi) ? hi + lo : hi; }
  __device__ __forceinline__ void add(double x) {
    const double s = hi + x, b = s - hi;
    lo += (hi - (s - b)) + (x - b);
    hi = s;
  }
  __device__ __forceinline__ void add(const Sum2& o) {
    add(o.hi);
    lo += o.lo;
  }
};

// mass (src/variables.f90:590-610) and momentum (:615-694) in one pass:
// per block, [8] partials = (hi, lo) of { sum |psi|^2, and for d = x, y, z the
// weighted sum of (Re psi - 1) Im(d conj psi) - Im psi Re(d psi) }.  First
// derivatives use the face ghosts: c1 (f+1 - f-1) + c2 (f+2 - f-2).
// A block owns 32 x 8 sites in (x, y) and marches a chunk of z: the z
// neighbours come from a register queue, the x and y ones from L1, so DRAM is
// read about once.  Bound by FP64 and L1 (256^3 complex128: 296 us with every
// neighbour fetched by its own 64-bit index).
// Neighbouring sites carry momentum of one sign, so the partial sums of a block
// are far larger than the total they cancel to, and rounding them costs digits
// that scattered sites did not (momentum at 256^3: 2.5e-15 of its largest
// component against 1.5e-15): a thread adds DIAG_RUN planes plainly, and from
// there on every sum is a Sum2 (3.7e-16).  256^3, plain sums -> these: complex128
// 144 -> 129 us, complex64 137 both; three blocks per SM, unrolled by two in
// complex128 only (without the cap 126 registers and 191 us; complex64 unrolled
// 150).
constexpr int DIAG_RUN = 8;
constexpr int DIAG_PARTIALS = 8;  // doubles a block
struct DiagArgs {
  Geom g;
  double c1[3], c2[3];
  const double* w[3];
  int tx, ty, zchunk;  // tiles in x and y, planes per block
};
template <typename TS, bool FOURTH>
__global__ void __launch_bounds__(256, 3) diag_kernel(const TS* __restrict__ f,
                                                       DiagArgs p,
                                                       double* __restrict__ partials) {
  using V = typename VT<TS>::T;
  __shared__ Sum2 red[4][8];
  constexpr int R = FOURTH ? 2 : 1, UNROLL = sizeof(TS) == 8 ? 2 : 1;
  const V* F = reinterpret_cast<const V*>(f);
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int tile = blockIdx.x % (p.tx * p.ty), chunk = blockIdx.x / (p.tx * p.ty);
  const int i = (tile % p.tx) * 32 + lane, j = (tile / p.tx) * 8 + row;
  const int z0 = chunk * p.zchunk, z1 = min(z0 + p.zchunk, p.g.nz);
  const int sy = p.g.Nx;
  const size_t sz = (size_t)p.g.Nx * p.g.Ny;
  Sum2 sum[4] = {};
  if (i < p.g.nx && j < p.g.ny) {
    const double wxy = p.w[0][i] * p.w[1][j];
    const V* c = F + padded_index(p.g, i, j, z0);
    V q[2 * R + 1];  // planes z - R .. z + R
#pragma unroll
    for (int d = 0; d < 2 * R; d++) q[d] = *(c + (ptrdiff_t)(d - R) * (ptrdiff_t)sz);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll UNROLL
    for (int z = z0; z < z1; z++, c += sz) {
      q[2 * R] = c[(size_t)R * sz];
      const double re = (double)q[R].x, im = (double)q[R].y;
      acc[0] += re * re + im * im;
      const double w = wxy * p.w[2][z];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        V p1, m1, p2, m2;
        if (a == 2) {
          p1 = q[R + 1];
          m1 = q[R - 1];
          p2 = q[2 * R];
          m2 = q[0];
        } else {
          const int s = a == 0 ? 1 : sy;
          p1 = c[s];
          m1 = c[-s];
          p2 = FOURTH ? c[2 * s] : p1;
          m2 = FOURTH ? c[-2 * s] : m1;
        }
        double dr = p.c1[a] * ((double)p1.x - (double)m1.x);
        double di = p.c1[a] * ((double)p1.y - (double)m1.y);
        if (FOURTH) {
          dr += p.c2[a] * ((double)p2.x - (double)m2.x);
          di += p.c2[a] * ((double)p2.y - (double)m2.y);
        }
        // Im(d conj psi) = -Im(d psi)
        acc[1 + a] += w * (-(re - 1.0) * di - im * dr);
      }
#pragma unroll
      for (int d = 0; d < 2 * R; d++) q[d] = q[d + 1];
      if (((z - z0) & (DIAG_RUN - 1)) == DIAG_RUN - 1 || z == z1 - 1)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          sum[v].add(acc[v]);
          acc[v] = 0.0;
        }
    }
  }
#pragma unroll
  for (int v = 0; v < 4; v++) {
    Sum2 t = sum[v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      t.add(Sum2{__shfl_down_sync(0xffffffffu, t.hi, o), __shfl_down_sync(0xffffffffu, t.lo, o)});
    if (lane == 0) red[v][row] = t;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    Sum2 t = red[threadIdx.x][0];
    for (int w = 1; w < 8; w++) t.add(red[threadIdx.x][w]);
    double* out = partials + (size_t)DIAG_PARTIALS * blockIdx.x + 2 * threadIdx.x;
    out[0] = t.hi;
    out[1] = t.lo;
  }
}

// [nblk][4] pairs -> out[0..3] * scale, fixed order (one CTA of 1024).
__global__ void __launch_bounds__(1024) diag_finalize_kernel(const double* __restrict__ partials,
                                                              int nblk, double scale,
                                                              double* __restrict__ out) {
  __shared__ Sum2 s[1024];
  // value v of blocks b, b + 256, ...: thread 4 b + v, so loads are contiguous
  Sum2 a = {};
#pragma unroll 4
  for (int q = threadIdx.x; q < 4 * nblk; q += 1024)
    a.add(Sum2{partials[2 * q], partials[2 * q + 1]});
  s[threadIdx.x] = a;
  __syncthreads();
  for (int w = 512; w >= 4; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x].add(s[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x < 4) out[threadIdx.x] = s[threadIdx.x].value() * scale;
}

}  // namespace gpe
