// Host-side internals shared by the library's translation units: the
// per-thread status, the device status word, device properties and TMA
// tensor-map encoding through the driver entry point (no link-time libcuda).
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <utility>

#include "phpc_gemm.h"

namespace phpc {

// Per-thread status of the last public call.
void set_last_error(int code);
int get_last_error();

// Device status word (a file-scope __device__ int, one per device). Kernels
// receive its device address and record timeouts there.
int* device_status_ptr();

// Properties of the current device, cached per device ordinal.
struct DeviceInfo {
  int ordinal;
  int sm_count;
  int cc_major, cc_minor;
  size_t smem_optin;
};
const DeviceInfo* current_device();

inline int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }

// Launches a kernel; with `dependent` it may come up while the kernel before it
// on the stream finishes (programmatic dependent launch: the kernel calls
// pdl_wait before it touches global memory). Only for a kernel that directly
// follows one of this library's own on the stream. Such a kernel takes no
// __restrict__ pointers: its inputs are still being written when it starts, and
// the qualifier would let the compiler read them through the non-coherent path
// or ahead of the wait.
template <class... P, class... A>
cudaError_t launch_dependent(bool dependent, void (*kern)(P...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Whether a GEMM of `steps` K-steps a tile is short enough for dependent
// launches around it: up to 80 K-steps an SM. A dependent launch takes the SMs
// in the order they fall free instead of the regular one, and a long kernel
// loses more by that (blocks that share data in L2 end up on different halves
// of the GPU) than the set-up it hides: N = 1024 (44 K-steps an SM) 65.9 ->
// 63.5 us, but 1537 x 1000 x 2311 (178) 161 -> 167-170, 4096 x 512 x 4096 330
// -> 361, 3xBF16 at 32768 x 4096 x 8192 8.84 -> 9.12 ms with every launch
// dependent.
inline bool short_gemm(int m, int n, int64_t steps, int sms) {
  return (int64_t)ceil_div(m, 128) * ceil_div(n, 256) * steps <= (int64_t)80 * sms;
}

// A value of 1 and up kept per device ordinal (a kernel attribute, an
// occupancy): 0 until it is stored. Devices beyond the table are asked anew.
struct PerDevice {
  static constexpr int kDevices = 64;
  std::atomic<int> v[kDevices] = {};
  int get(int ordinal) const { return ordinal >= 0 && ordinal < kDevices ? v[ordinal].load(std::memory_order_acquire) : 0; }
  void set(int ordinal, int value) {
    if (ordinal >= 0 && ordinal < kDevices) v[ordinal].store(value, std::memory_order_release);
  }
};

// cuTensorMapEncodeTiled, resolved once through cudaGetDriverEntryPointByVersion.
bool encode_tiled(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base, const uint64_t* dims,
                  const uint64_t* strides_bytes /* rank-1 entries */, const uint32_t* box, CUtensorMapSwizzle swz);

#define PHPC_CUDA_TRY(expr)                                                                        \
  do {                                                                                             \
    cudaError_t _e = (expr);                                                                       \
    if (_e != cudaSuccess) {                                                                       \
      if (getenv("PHPC_VERBOSE"))                                                                  \
        fprintf(stderr, "phpc: %s failed at %s:%d: %s\n", #expr, __FILE__, __LINE__, cudaGetErrorString(_e)); \
      return PHPC_ERR_CUDA;                                                                        \
    }                                                                                              \
  } while (0)

// Library-internal launchers (device pointers, asynchronous on `stream`).
bool fp64_pipe_is_dfma();
int dgemm_dmma(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
               int64_t ldc, int gw, int gh, int kpanel, cudaStream_t stream);
int dgemm_ozaki(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
                int64_t ldc, int s, void* ws, size_t ws_bytes, cudaStream_t stream, int bn);
size_t ozaki_workspace_bytes(int m, int k, int n, int s);
size_t ozaki2_workspace_bytes(int m, int k, int n, int nmod);
int dgemm_ozaki2(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
                 int64_t ldc, int nmod, void* ws, size_t ws_bytes, cudaStream_t stream, int bn);
int ozaki2_bits(int nmod, int k);
int ozaki2_prepare2(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, int nmod,
                    void* ws, size_t ws_bytes, cudaStream_t stream_a, cudaStream_t stream_b);
int ozaki2_multiply(int m, int k, int n, int nmod, const void* ws, size_t ws_bytes, cudaStream_t stream, int bn);
// Row-panel pieces of the modular scheme (device pointers to row 0 of the full
// m-row operands; the workspace is that of the full m x k x n problem).
int ozaki2_prepare_a_rows(int m, int r0, int rows, int k, int n, const double* dA, int64_t lda, int nmod, void* ws,
                          size_t ws_bytes, cudaStream_t stream);
int ozaki2_prepare_b(int m, int k, int n, const double* dB, int64_t ldb, int nmod, void* ws, size_t ws_bytes,
                     cudaStream_t stream);
int ozaki2_multiply_rows(int m, int r0, int rows, int k, int n, int nmod, const void* ws, size_t ws_bytes,
                         cudaStream_t stream, int bn);
// Column-panel pieces (dB: column 0 of the full k x n operand): B's scan and
// split of columns [c0, c0 + cols), and the residue GEMMs of the block of rows
// [r0, r0 + rows) x columns [c0, c0 + cols).
int ozaki2_prepare_b_cols(int m, int k, int n, int c0, int cols, const double* dB, int64_t ldb, int nmod, void* ws,
                          size_t ws_bytes, cudaStream_t stream);
int ozaki2_multiply_block(int m, int r0, int rows, int c0, int cols, int k, int n, int nmod, const void* ws,
                          size_t ws_bytes, cudaStream_t stream, int bn, bool dependent = false);
int ozaki2_reconstruct_rows(int m, int r0, int rows, int k, int n, double* dC, int64_t ldc, int nmod, const void* ws,
                            size_t ws_bytes, cudaStream_t stream, bool dependent = false);
int ozaki2_reconstruct(int m, int k, int n, double* dC, int64_t ldc, int nmod, const void* ws, size_t ws_bytes,
                       cudaStream_t stream);
int ozaki2_grids(int m, int k, int n, int nmod, const void* ws, size_t ws_bytes, int* ea, int* eb, int* ba, int* bb);
int ozaki_prepare2(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, int s, void* ws,
                   size_t ws_bytes, cudaStream_t stream_a, cudaStream_t stream_b);
int ozaki_multiply(int m, int k, int n, double* dC, int64_t ldc, int s, const void* ws, size_t ws_bytes,
                   cudaStream_t stream, int bn);
// Device memory pool of the host entry points (one per device, grow-only
// unless PHPC_POOL_KEEP=0): buffers of one call are reused by the next.
cudaMemPool_t host_api_pool();
// A second stream of this host thread on the current device, for work that
// can run beside the caller's stream (nullptr if it cannot be created).
cudaStream_t side_stream();
// Makes `to` wait for the work submitted to `from` so far (an event; valid
// under stream capture, where it adds `to` to the captured graph).
bool stream_fork(cudaStream_t from, cudaStream_t to);
// Creates this thread's side stream and fork event (call before a capture).
bool side_stream_ready();
int default_slices(int m, int k, int n);
// Number of moduli of the modular scheme for this shape, or 0 for the digit
// scheme (default_slices slices).
int default_moduli(int m, int k, int n);
int default_bn(int m, int k, int n);
int digit_bn(int m, int k, int n);       // the digit GEMM's tile width
int digit_cluster(int m, int k, int n);  // and CTAs per cluster
int modular_bn(int m, int k, int n, int moduli);
int default_grouped_bn(const phpc_gemm_problem* problems, int count);
int default_group_rows(int m, int k, int n);
int default_cluster(int m, int k, int n, int moduli);
// Pipeline depths: K-stages of the tcgen05 engine's shared-memory ring for
// the FP64-accurate GEMMs (0 = the deepest ring that fits), of the 3xBF16
// FP32 GEMM, and of the plain FP64 GEMM (2 .. 6).
int default_stages(int m, int k, int n);
int default_plain_stages(int m, int k, int n);
// 3xBF16 FP32 GEMM: tile width, raster height and stages from the table's
// "f32" entries (PHPC_F32_BN / PHPC_GROUP_ROWS / PHPC_STAGES override).
struct F32Tune {
  int bn, group_rows, stages;
};
F32Tune default_f32(int m, int k, int n);
bool residue_wide_split(int m, int k, int n, int moduli, const DeviceInfo* dev);
bool f32_narrow_split(int m, int k, int n, const DeviceInfo* dev);
constexpr int kF32SplitSteps = 48;  // K-steps (six products of each 64 of K) from which the 3xBF16 GEMM splits K
// Stages of the grouped GEMM (the "grouped" entry's fifth field; 0 = deepest).
int default_grouped_stages(const phpc_gemm_problem* problems, int count);

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Row stride (in BF16 elements) of an operand plane K long. TMA needs 16-byte
// rows; rows that start off a 32-byte sector cost the GEMM a fifth sector per
// 128-byte box row and 1.6x its time (m = n = 3000: 695 us at K = 3000 or
// 3016, 466 at 3040, 442 at 3008; whole 128-byte lines are another 5 %), so
// rows are padded to 128 bytes, short ones (where that could double a plane)
// to 32. A workspace that holds only the 16-byte layout still gets that one.
inline int64_t plane_ld(int k, bool padded) {
  const int64_t to = !padded ? 8 : k >= 256 ? 64 : 16;
  return (k + to - 1) / to * to;
}


}  // namespace phpc
