// internal.h -- library-internal access between translation units (not part
// of the C-ABI).
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <string>

#include "gpe_gpu.h"

namespace gpe {

// The resident psi of a context: padded field (gh ghosts per side, pitches
// Nx >= nx + 2 gh, Ny = ny + 2 gh), complex of es bytes.
struct FieldView {
  void* psi;
  int nx, ny, nz, Nx, Ny;
  int gh;
  int es;
  int bcs;
  int dev;
  int single_domain;
  cudaStream_t stream;
  int* status;  // the context's device status word (wait timeouts)
  double dx, dy, dz;  // grid spacings, 2 xr / (nx - 1) etc.
  double xr, yr, zr;  // box half-widths
  void* stage;        // dense staging buffer, nx ny nz elements of 16 bytes
  bool overlap;       // launches on the stream may overlap (stream_overlap in gpe_gpu.cu)
};

// Whether a correction network can work on a grid: rows of nx sites (a multiple
// of an MMA's 16, up to its 128 rows), complex of es bytes, boundary bcs.  Asked by
// the network's own checks and by rk4, which keeps its order of summation there.
inline bool network_nx(int nx) { return nx >= 16 && nx <= 128 && nx % 16 == 0; }
inline bool network_fits(int nx, int es, int bcs) { return network_nx(nx) && es == 8 && bcs == 1; }

// Lets every launch of fn take as much dynamic shared memory as a block may
// have.  The limit is the function's, shared by all contexts, threads and
// launches of the process, while what a launch needs depends on its grid: a
// limit set to one launch's need would refuse a larger one of another context.
// One read of the attributes where the limit is there already.
inline cudaError_t allow_dynamic_smem(const void* fn) {
  constexpr int BLOCK_SMEM = 227 * 1024;
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, fn);
  if (e != cudaSuccess) return e;
  const int most = BLOCK_SMEM - (int)a.sharedSizeBytes;
  if (a.maxDynamicSharedSizeBytes >= most) return cudaSuccess;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

// Launches fn, which begins with after_previous(), so that its blocks are set
// up while the kernel before it in the stream ends (programmatic dependent
// launch).  Where kernels last some microseconds the gap between two of them
// counts: an rk2 step (two launches) of 40^3 14.4 -> 9.8 us, an rk4 step in pairs
// (four) of 32^3 24.7 -> 15.9, one stage at a time (five) of 64^3 32.9 -> 21.7.
template <typename... P, typename... A>
cudaError_t launch_overlapped(bool overlap, void (*fn)(P...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(a)...);
}
// The same for a kernel held as an untyped entry.
inline cudaError_t launch_overlapped(bool overlap, const void* fn, dim3 grid, dim3 block,
                                     void** args, size_t smem, cudaStream_t st) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// A timed region on a context's stream (recorded only while the context's
// timing is on; collected by gpe_gpu_get_timing under `family`).
struct TimedRegion {
  cudaEvent_t a = nullptr, b = nullptr;
  int family = 0;
  int64_t sites = 0;
};

// Per-context state of another translation unit, owned by the context and
// deleted with it (with the context's device current, its stream drained).
struct Extension {
  virtual ~Extension() = default;
};

}  // namespace gpe

// Fills *v; marks the context's cached norm stale (the caller may write psi).
int gpe_internal_field_view(gpe_ctx* c, gpe::FieldView* v);
// fn(arg, c) is called after every completed step of c (enqueueing work on
// c's stream); null detaches.
void gpe_internal_set_post_step(gpe_ctx* c, int (*fn)(void*, gpe_ctx*), void* arg);
void gpe_internal_set_last_error(const std::string& msg);
// Records msg as the context's last error and returns code.
int gpe_internal_fail(gpe_ctx* c, int code, const std::string& msg);
// The context's extension slots (0 spectral, 1 vortex line length).
constexpr int GPE_EXT_SPECTRAL = 0, GPE_EXT_VORTEX = 1, GPE_EXT_SLOTS = 2;
std::unique_ptr<gpe::Extension>& gpe_internal_extension(gpe_ctx* c, int slot);
// Dense staging buffer (x fastest, elements of the field's own es bytes) ->
// psi with the boundary ghosts filled; invalidates the cached norm.
int gpe_internal_load_stage(gpe_ctx* c);
void gpe_internal_time_begin(gpe_ctx* c, gpe::TimedRegion* r, int family, int64_t sites);
void gpe_internal_time_end(gpe_ctx* c, gpe::TimedRegion* r);
// Enqueues psi *= sqrt(norm of the last step / norm of psi now) (the norm
// kept through a post-step correction).
int gpe_internal_restore_norm(gpe_ctx* c);
// Adds n to the context's launch counter (kernels enqueued by other units).
void gpe_internal_count_launches(gpe_ctx* c, int64_t n);
