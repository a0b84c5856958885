// Error plumbing shared by the C-ABI entry points: every entry returns 0 on success or a negative
// code, and leaves a message retrievable with mpsa_last_error().  No exception crosses the
// boundary and nothing here allocates device memory.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#define MPSA_OK 0
#define MPSA_ERR_BAD_ARG (-1)
#define MPSA_ERR_UNSUPPORTED (-2)
#define MPSA_ERR_LAUNCH (-3)
#define MPSA_ERR_TIMEOUT (-4)

namespace mpsa {
int set_error(int code, const char* fmt, ...);
int check_launch(const char* what);
int sm_count();                       // of the current device

// Opt-in for more than 48 KB of dynamic shared memory: a per-device attribute of a kernel, set by the first launch on
// each device (ID tells the kernels of one function type apart).
template <int ID, typename F>
bool allow_smem(F* kernel, int bytes) {
  constexpr int kMaxDevices = 64;
  static std::atomic<bool> done[kMaxDevices];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev >= 0 && dev < kMaxDevices && done[dev].load(std::memory_order_acquire)) return true;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (dev >= 0 && dev < kMaxDevices) done[dev].store(true, std::memory_order_release);
  return true;
}

// A launch that may start (dependent) while the kernel before it on the stream, whosever it is, still runs: once every CTA of that one has
// ended or let its dependents go.  The kernel must call grid_dependency_wait() before it touches memory that anything before it on the
// stream may write or read, in every CTA that does, and every launch after it has to be able to rely on that: see overlaps_previous.
template <typename... P, typename... A>
void launch_dependent(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, bool dependent, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);     // an error is reported by check_launch
}

// Whether the first launch of a call may be a dependent one of whatever is before it on the stream: its CTAs then set up, and wait in
// grid_dependency_wait(), under that kernel's tail.  A wait is for the one kernel before, so what follows has to know everything earlier to
// be complete when that one is: the first kernels of a call (preparation, column sums, product) wait in every thread, and only then let
// their dependents go.  Two later ones let them go before they wait, and wait all the same before they end: the preparation behind the
// column sums, which starts only when those have seen the end of everything before them, and nvfp4_quant_kernel behind the preparation.
// Not while the stream is captured: a
// graph node with several predecessors takes ordinary edges.  Back to back: NVFP4
// 1500 x 4096 x 4096 18.5 -> 17.2 us, routed attention over 1024 tokens 28.4 -> 27.4.
inline bool overlaps_previous(cudaStream_t st) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &c) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return c == cudaStreamCaptureStatusNone;
}

// One call of the fused forward (see mpsa_attn_fwd for the operands).  map null: the band rule (band, uniform) instead.
struct AttnCall {
  const void *q8 = nullptr, *q8_sf = nullptr, *q4 = nullptr, *q4_sf = nullptr;
  const void *k8 = nullptr, *k8_sf = nullptr, *k4 = nullptr, *k4_sf = nullptr;
  const void *vt = nullptr, *vt8 = nullptr, *v8_sf = nullptr, *vt4 = nullptr, *v4_sf = nullptr;
  int pv_mode = 0;
  const void* map = nullptr;
  long long map_sb = 0, map_sh = 0;
  int band = 1, uniform = 0;            // uniform: 0 no, 1 MXFP8, 2 FP4
  bool route = false;                   // online router inside (map_rw: the map it writes)
  float tau = 0.0f;
  void *map_rw = nullptr, *stat_out = nullptr;
  void* out = nullptr;
  int out_dtype = 0;
  void* lse = nullptr;
  int B = 0, Hq = 0, Hkv = 0, S = 0, Skv = 0, D = 0, Skv_pad = 0, causal = 0, fp8_fmt = 1, fp4_kind = 0;
  bool need8 = true, need4 = true;      // operand formats the map can select; the pointers of the other may be null
  bool depth64 = false;                 // the upper 64 of the 128 depth elements of Q and K are zero blocks
  float fp4_scale = 0.0f;
  const void *ts_q = nullptr, *ts_k = nullptr;   // NVFP4: the two tensor scales in device memory, instead of fp4_scale
  int* range_flag = nullptr;
  int* counter = nullptr;               // a device word, zero on entry: work items are handed out in turn (fixed schedule without it)
  void* partial = nullptr;              // attn_split_bytes() of device memory, 256-byte aligned: lets the forward divide an item's keys among CTAs
  bool after_prep = false;              // the kernel before this one on the stream is prep_launch's
  const void *acc_in = nullptr, *lse_in = nullptr;
  int* status = nullptr;
};
int attn_forward(const AttnCall& c, cudaStream_t st);
long long attn_split_bytes(const AttnCall& c);   // 0: this call divides no item (acc_in and lse go without a division)
// partial column sums of x [B,H,L,D], [B*H, nchunk, D] floats, nchunk = col_sum_chunks(L)
int col_sum_chunks(int L);
int col_sums(const void* x, int in_dtype, int B, int H, int L, int D, long long xs_b, long long xs_h, long long xs_l, float* part,
             int nchunk, cudaStream_t st);
// NVFP4 codes and E4M3 scale tiles of x [B,H,L,D] (16-bit, D a multiple of 64), given the bits of amax |x * s| in device memory;
// launched as a dependent of the kernel before it
int nvfp4_quant(const void* x, int in_dtype, int B, int H, int L, int D, long long xs_b, long long xs_h, long long xs_l, float s,
                unsigned* amax, void* codes, void* scales, float* tensor_scale, cudaStream_t st);
}  // namespace mpsa
