// Internal declarations shared by the translation units behind include/cct_b200.h.
#pragma once
#include <atomic>
#include <cuda_runtime.h>
#include <stdint.h>
#include <functional>
#include <initializer_list>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cct_b200.h"
#include "half_pairs.cuh"

struct cct_ctx;

// What a program (cct_program_begin) does with a context's calls concerns the thread that does it alone; other threads' calls
// on the same context are carried out on the context's stream meanwhile.
struct Recording {  // between cct_program_begin and _end: this thread's bridge calls on `ctx` are kept in `calls`
  cct_ctx* ctx = nullptr;
  std::vector<std::function<int()>>* calls = nullptr;
  bool live = false;  // and carried out as well
};
inline thread_local Recording recording_here;
inline thread_local cudaStream_t capture_here = nullptr;  // set while this thread captures a program: its launches go there

// The stream a context's work is enqueued on, as seen from this thread.
struct CtxStream {
  cudaStream_t own = nullptr;
  CtxStream& operator=(cudaStream_t s) { own = s; return *this; }
  operator cudaStream_t() const { return capture_here ? capture_here : own; }
};

struct cct_ctx {
  int device = 0;
  CtxStream stream;
  bool owns_stream = false;
  // Side streams of the host-buffer entry points: uploads and downloads overlap each other and the kernels.
  cudaStream_t copy_in = nullptr, copy_out = nullptr;
  int sm_count = 148;
  // SMs the persistent kernels leave free while gradient reductions are in flight on the communicator's stream
  // (set by cct_allreduce_sum_begin, cleared by cct_comm_wait): NCCL's CTAs take whole SMs, and a persistent grid
  // sized for every SM would otherwise run its displaced CTAs as a second wave.
  int reserved_sms = 0;
  int launch_sms() const { return sm_count - reserved_sms > 0 ? sm_count - reserved_sms : 1; }
  // Set when a communicator of more than one rank is created on this context: plans created afterwards size their
  // work-unit counts (split counts, channel tilings) for the SMs that remain while reductions are in flight, because
  // that is when the backward kernels of a multi-GPU job run.
  int comm_sms = 0;
  int planning_sms() const { return sm_count - comm_sms > 0 ? sm_count - comm_sms : 1; }
  // One word in mapped pinned host memory that kernels set when a bounded wait runs out; read by cct_sync().
  volatile int* status_host = nullptr;
  int* status_dev = nullptr;
  std::string last_error;
  std::atomic<cudaStream_t> spare_stream{nullptr};  // for the next capture of a program
  int timed_plans = 0;  // plans whose kernel timing is switched on: programs then run call by call
};

// First line of every recordable entry point: `call` is the entry point with its own arguments.
inline int record_call(std::function<int()> call) {
  const Recording here = recording_here;
  try {
    here.calls->push_back(call);
  } catch (...) {
    return CCT_ERR_NOMEM;
  }
  if (!here.live) return CCT_OK;
  recording_here = Recording{};  // an entry point may use others
  const int rc = call();
  recording_here = here;
  return rc;
}
#define CCT_RECORD(context, call)                                                    \
  if ((context) && recording_here.ctx == (context)) {                                \
    try {                                                                            \
      return record_call([=]() -> int { return call; });                             \
    } catch (...) {                                                                  \
      return CCT_ERR_NOMEM;                                                          \
    }                                                                                \
  }

// Whether `n` words at `out` lie outside all of `others` (address and words; null: none).
inline bool apart(const void* out, size_t n, std::initializer_list<std::pair<const void*, size_t>> others) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(out);
  for (const auto& o : others) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(o.first);
    if (o.first && a < b + o.second * 4 && b < a + n * 4) return false;
  }
  return true;
}

// Blocks of the first of two jobs, of `a` and `b` tiles, in one launch over `slots` resident blocks: one per tile where there are slots for all,
// else the slots in proportion to the tiles; 0 where there are more than two tiles for each of them.
inline int share_slots(long long slots, long long a, long long b) {
  if (a + b > 2 * slots) return 0;
  const long long mine = a + b <= slots ? a : slots * a / (a + b);
  return (int)(mine < 1 ? 1 : mine);
}

#define CCT_CUDA(ctx, call)                                                                   \
  do {                                                                                        \
    cudaError_t e__ = (call);                                                                 \
    if (e__ != cudaSuccess) {                                                                 \
      (ctx)->last_error = std::string(#call) + ": " + cudaGetErrorString(e__);                \
      return e__ == cudaErrorMemoryAllocation ? CCT_ERR_NOMEM : CCT_ERR_CUDA;                 \
    }                                                                                         \
  } while (0)

// Programmatic dependent launch: every kernel of the library starts with pdl_wait() - the persistent
// ones once barriers, tensor memory and the plan's constant tables are set up - (griddepcontrol.wait: returns once
// the kernel before it in the stream has completed and its writes are visible) and is launched with the programmatic
// stream-serialisation attribute, so the launch itself - grid set-up, parameter upload - overlaps the tail of its
// predecessor instead of following it.  No kernel signals its dependents early: the order of execution stays the
// stream's order.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline std::atomic<uint64_t> kernel_launches{0};  // cct_kernel_launches
inline thread_local uint64_t thread_launches = 0; // those of this thread, captured ones included

// `cluster` blocks (a divisor of the grid's x) form a thread-block cluster.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(unsigned cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                      cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  kernel_launches.fetch_add(1, std::memory_order_relaxed);
  ++thread_launches;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  return launch_pdl_cluster(1, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}
#endif

#define CCT_CHECK_LAUNCH(ctx) CCT_CUDA(ctx, cudaGetLastError())

// Optional per-kernel-group timing with CUDA events on the context's stream (measurement only).
struct PhaseTimer {
  static constexpr int kSlots = 5;  // 0 forward, 1 wgrad, 2 wgrad reduce (with the repacking for dgrad), 3 dgrad, 4 forward repack
  bool enabled = false;
  cudaEvent_t ev[2 * kSlots] = {};
  bool have[kSlots] = {};
  void begin(int slot, cudaStream_t s) {
    if (enabled) cudaEventRecord(ev[2 * slot], s);
  }
  void end(int slot, cudaStream_t s) {
    if (enabled) {
      cudaEventRecord(ev[2 * slot + 1], s);
      have[slot] = true;
    }
  }
};

// Geometry of one convolution layer, resolved once per plan.
struct ConvGeom {
  int B, D, n, o, k, s, p, g;
  int m;       // output size
  int Dg, og;  // per-group depths
  int bias;
};

// ---- SIMT fp32 path (conv_simt.cu) ----
int simt_conv_forward(cct_ctx* ctx, const ConvGeom& G, const float* X, const float* W, const float* bias, float* Y,
                      int relu, PhaseTimer* t);
int simt_conv_backward(cct_ctx* ctx, const ConvGeom& G, const float* X, const float* W, const float* dY, float* dX,
                       float* dW, float* db, PhaseTimer* t);

// ---- tcgen05 3xTF32 path (conv_umma.cu) ----
// dY as the weight gradient's operand: rows of one channel over all images (`row_len` floats, a multiple of 32), the values and
// behind them, `lo` floats on, their low parts; the plane sums for the bias gradient, or null.
struct DyRows {
  float* rows = nullptr;
  size_t lo = 0, row_len = 0;
  float* plane_sums = nullptr;
  int channels = 0, batch = 0;
  const HalfScales* half = nullptr;  // set, and X and dY ok: pairs of fp16 of scaled dY in place of the low parts (half_word)
};
struct UmmaPlan;  // opaque: tables, packed weights, split-K scratch
// `tensor_only`: every pass on the tensor cores, however small the layer (CCT_ALGO_UMMA_3XTF32 by name); otherwise small
// layers take the fp32 kernels of conv_small.cuh.
int umma_plan_create(cct_ctx* ctx, const ConvGeom& G, bool tensor_only, UmmaPlan** out);
void umma_plan_destroy(cct_ctx* ctx, UmmaPlan* p);
size_t umma_plan_workspace_bytes(const UmmaPlan* p);
bool umma_supported(const ConvGeom& G);
// `batch` > 0 restricts a call to the first `batch` images of the tensors it is given; `repack` = rewrite the packed
// weight operand from W first (needed once per new W).  `pack_W`: the weight gradient's last launch does that for the data
// gradient.
int umma_conv_forward(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* bias, float* Y,
                      int relu, PhaseTimer* t, int batch = 0, bool repack = true);
int umma_conv_backward(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* dY, float* dX,
                       float* dW, float* db, PhaseTimer* t, bool scaled = false);
// Whether umma_conv_backward takes dY in the form of `rows` (then dY = null), written there by the kernel that makes it.
bool umma_dy_rows(const UmmaPlan* p, DyRows* rows);
// Where dY is what pooling P's windows (k x k, stride s) makes of dP, the scales come from dP, which is smaller; before that kernel (whose rows need
// them); umma_conv_backward is `scaled` then.
int umma_pooled_scales(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* W, const float* dP, const float* P, const int32_t* idx, int k, int s,
                       bool dgrad);
int umma_conv_wgrad(cct_ctx* ctx, UmmaPlan* p, const float* X, const float* dY, float* dW, float* db, PhaseTimer* t,
                    const float* pack_W = nullptr);
int umma_conv_dgrad(cct_ctx* ctx, UmmaPlan* p, const float* W, const float* dY, float* dX, PhaseTimer* t, int batch,
                    bool repack);

// ---- max pooling forward with the plane staged in shared memory (layers.cu)
// pool_relu_backward_pooled for windows of 3x3 with stride 2, into rows; CCT_ERR_UNSUPPORTED (and no error text) for others.
int pool_relu_backward_rows(cct_ctx* ctx, const float* P, const int32_t* idx, const float* dP, const DyRows& out, int planes,
                            int n, int k, int s);
int pool_relu_backward_pooled(cct_ctx* ctx, const float* P, const int32_t* idx, const float* dP, float* dA, int planes,
                              int n, int k, int s);
int maxpool_forward_staged(cct_ctx* ctx, const float* X, float* Y, int32_t* idx, int planes, int n, int m, int k, int s);

// ---- index arithmetic of the pooling kernels
// x / d for x * d < 2^32 as one multiply-high: inv = floor(2^32 / d) + 1 (host side, fast_div_magic); inv == 0 means
// "divide".  The GPU has no integer divider, and these kernels would otherwise spend more on index arithmetic than on
// memory.
__device__ __forceinline__ uint32_t fast_div(uint32_t x, uint32_t d, uint32_t inv) {
  return inv ? __umulhi(x, inv) : x / d;
}
// Magic for fast_div: valid when max_x * d < 2^32 and d > 1, else 0 (plain division).
inline uint32_t fast_div_magic(uint64_t max_x, uint32_t d) {
  return (d > 1 && max_x * d < (1ull << 32)) ? (uint32_t)((1ull << 32) / d) + 1u : 0u;
}
