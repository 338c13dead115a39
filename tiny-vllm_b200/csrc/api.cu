// C ABI of libb200q: argument validation, kernel-family choice, launches.
// Nothing here allocates device memory, synchronises, or falls back to a CPU path.
#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cstdint>

#include "common.h"

namespace b200q {

// Device-side status word: a kernel whose bounded wait gave up writes a non-zero code here.
__device__ int g_device_status = 0;

namespace {
std::atomic<int> g_last_cuda_error{0};
std::atomic<uint64_t> g_launches{0};

// Debug knobs of the calling thread (common.h): value and "is set" per knob.
struct Knobs {
  int value[B200Q_KNOB_COUNT];
  bool set[B200Q_KNOB_COUNT];
};
thread_local Knobs t_knobs{};

constexpr int kMaxDevices = 64;

struct DeviceInfo {
  std::atomic<int> ready{0};
  int cc_major = 0;
  int sms = 0;
  int* status_ptr = nullptr;
};
DeviceInfo g_dev[kMaxDevices];

DeviceInfo* device_info() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  DeviceInfo& d = g_dev[dev];
  if (d.ready.load(std::memory_order_acquire) == 0) {
    int major = 0, sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    void* p = nullptr;
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&p, g_device_status);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      return nullptr;
    }
    d.cc_major = major;
    d.sms = sms;
    d.status_ptr = static_cast<int*>(p);
    d.ready.store(1, std::memory_order_release);
  }
  return &d;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_dims(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return B200Q_ERR_BAD_SHAPE;
  if (static_cast<long long>(M) * N > INT_MAX || static_cast<long long>(M) * K > INT_MAX ||
      static_cast<long long>(N) * K > INT_MAX)
    return B200Q_ERR_BAD_SHAPE;
  if ((K % 16) != 0) return B200Q_ERR_UNSUPPORTED_SHAPE;
  return B200Q_OK;
}

// Kernel family when nothing is forced; figures from graph-replayed chains of launches.
// * Few tokens: the weight-streaming mma.sync family — the kernels that hold the weights in registers where
//   they are the fastest, the ring-fed persistent ones for larger matrices (gemm_bulk_decode.cu).
// * Long rows of a narrow matrix (K > 4096, too few channels for the rings): tcgen05 with K split over clusters
//   (128 x 8192 at 16 tokens: 3.4 against 5.7 us W8A8, 4.4 against 7.1 W8A16).
// * Everything else: tcgen05.  Its single-CTA kernel for mid sizes wants 16-byte output pieces; with an odd
//   channel count up to 32 tokens stay on the streaming kernels.
int auto_path(int M, int N, int K, bool a16) {
  if (M <= debug_knob(B200Q_KNOB_SIMT_MAX_M, 0)) return B200Q_PATH_SIMT_STREAM;
  if (reg_decode_preferred(M, N, K, a16)) return B200Q_PATH_MMA_STREAM;
  if (M <= 16) {
    if (bulk_decode_applicable(M, N, K, a16)) return B200Q_PATH_MMA_STREAM;
    // long K, or a matrix that the ring leaves to them: the tcgen05 kernels
    return (K > 4096 || (a16 && bulk_decode_yields(M, N, K))) && (N % 8) == 0 ? B200Q_PATH_UMMA : B200Q_PATH_MMA_STREAM;
  }
  return M <= 32 && (N % 8) != 0 ? B200Q_PATH_MMA_STREAM : B200Q_PATH_UMMA;
}

int resolve_path(int op, int M, int N, int K) {
  const int forced = debug_knob(B200Q_KNOB_FORCE_PATH, B200Q_PATH_AUTO);
  if (forced != B200Q_PATH_AUTO) return forced;
  return auto_path(M, N, K, op == B200Q_OP_W8A16);
}

int run_w8a8(GemmArgs& a) {
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  a.status = d->status_ptr;
  const int path = resolve_path(B200Q_OP_W8A8, a.M, a.N, a.K);
  if (path == B200Q_PATH_SIMT_STREAM) {
    cudaError_t e = launch_w8a8_simt(a);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      return B200Q_ERR_LAUNCH;
    }
    return B200Q_OK;
  }
  if (path == B200Q_PATH_MMA_STREAM) {
    if (!mma_decode_applicable(a.M)) return B200Q_ERR_UNSUPPORTED_SHAPE;
    cudaError_t e = bulk_decode_applicable(a.M, a.N, a.K, false) ? launch_w8a8_bulk_decode(a)
                    : reg_decode_applicable(a.M, a.N, a.K)     ? launch_w8a8_reg_decode(a, false)
                                                               : launch_w8a8_mma_decode(a);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      return B200Q_ERR_LAUNCH;
    }
    return B200Q_OK;
  }
  if (path == B200Q_PATH_UMMA && umma_pair_applicable(a.M, a.N, a.K, a.acc_out != nullptr))
    return launch_w8a8_umma_pair(a);
  if (path == B200Q_PATH_UMMA && umma_mid_applicable(a.M, a.N, a.K))
    return launch_umma_mid(a);
  if (path == B200Q_PATH_UMMA || path == B200Q_PATH_UMMA_SWAP) {
    UmmaPlan plan;
    if (!umma_make_plan(B200Q_OP_W8A8, a.M, a.N, a.K, path == B200Q_PATH_UMMA_SWAP, &plan))
      return B200Q_ERR_UNSUPPORTED_SHAPE;
    return launch_w8a8_umma(a, plan);
  }
  return B200Q_ERR_BAD_ARGUMENT;
}

// Workspace that run_w8a8 insists on: only the persistent single-CTA kernel with its K split through memory.
size_t w8a8_workspace_needed(int M, int N, int K) {
  const int path = resolve_path(B200Q_OP_W8A8, M, N, K);
  if (path != B200Q_PATH_UMMA && path != B200Q_PATH_UMMA_SWAP) return 0;
  if (path == B200Q_PATH_UMMA && (umma_pair_applicable(M, N, K, false) || umma_mid_applicable(M, N, K))) return 0;
  UmmaPlan plan;
  return umma_make_plan(B200Q_OP_W8A8, M, N, K, path == B200Q_PATH_UMMA_SWAP, &plan) ? plan.ws_bytes : 0;
}

// One kernel for quantisation and GEMM, where each CTA can afford to read all tokens' rows.
bool dynamic_is_fused(int M, int N, int K) {
  return resolve_path(B200Q_OP_W8A8, M, N, K) == B200Q_PATH_MMA_STREAM &&
         !bulk_decode_applicable(M, N, K, false) && reg_decode_dynamic_applicable(M, N, K);
}

// b200q_act_quant_i8 with the choice of `carve` and `early` (common.h)
int run_act_quant(const void* x, int64_t ldx, int x_dtype, int8_t* xq, float* a_scales, int M, int K,
                  Carveout carve, bool early, void* stream) {
  if (x == nullptr || xq == nullptr || a_scales == nullptr) return B200Q_ERR_NULL_POINTER;
  if (M <= 0 || K <= 0 || static_cast<long long>(M) * K > INT_MAX) return B200Q_ERR_BAD_SHAPE;
  if (x_dtype != B200Q_DTYPE_F16 && x_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if ((K % 16) != 0 || ldx < K || (ldx % 8) != 0) return B200Q_ERR_UNSUPPORTED_SHAPE;
  if (!aligned16(x) || !aligned16(xq) || (reinterpret_cast<uintptr_t>(a_scales) & 3u) != 0)
    return B200Q_ERR_MISALIGNED;
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  cudaError_t e =
      launch_act_quant(x, ldx, x_dtype, xq, a_scales, M, K, early, carve, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return B200Q_ERR_LAUNCH;
  }
  return B200Q_OK;
}

size_t dynamic_code_offset(int M) { return (static_cast<size_t>(M) * 4 + 255) / 256 * 256; }

}  // namespace

bool pdl_enabled() { return debug_knob(B200Q_KNOB_NO_PDL, 0) == 0; }

int debug_knob(int knob, int dflt) {
  if (knob < 0 || knob >= B200Q_KNOB_COUNT) return dflt;
  return t_knobs.set[knob] ? t_knobs.value[knob] : dflt;
}

int sm_count() {
  DeviceInfo* d = device_info();
  return d != nullptr && d->sms > 0 ? d->sms : 148;
}

int device_cc_major() {
  DeviceInfo* d = device_info();
  return d != nullptr ? d->cc_major : 0;
}

int* device_status_ptr() {
  DeviceInfo* d = device_info();
  return d != nullptr ? d->status_ptr : nullptr;
}

void note_cuda_error(cudaError_t e) { g_last_cuda_error.store(static_cast<int>(e)); }
void count_launch(int n) { g_launches.fetch_add(static_cast<uint64_t>(n)); }

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_act_quant_i8(const void* x, int64_t ldx, int x_dtype, int8_t* xq, float* a_scales, int M,
                       int K, void* stream) {
  return run_act_quant(x, ldx, x_dtype, xq, a_scales, M, K, DEFAULT_SPLIT, false, stream);
}

int b200q_w8a8_gemm(const int8_t* xq, const float* a_scales, const int8_t* qweight,
                    const float* w_scales, const void* bias, void* y, int M, int N, int K,
                    int out_dtype, void* workspace, size_t workspace_bytes, void* stream) {
  if (xq == nullptr || a_scales == nullptr || qweight == nullptr || w_scales == nullptr ||
      y == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (out_dtype != B200Q_DTYPE_F16 && out_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (!aligned16(xq) || !aligned16(qweight) || !aligned16(y) || !aligned16(w_scales) ||
      (reinterpret_cast<uintptr_t>(a_scales) & 3u) != 0 ||
      (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0) ||
      (workspace != nullptr && !aligned16(workspace)))
    return B200Q_ERR_MISALIGNED;
  GemmArgs a{};
  a.x = xq;
  a.w = qweight;
  a.a_scales = a_scales;
  a.w_scales = w_scales;
  a.bias = bias;
  a.y = y;
  a.acc_out = nullptr;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = out_dtype;
  a.workspace = workspace;
  a.workspace_bytes = workspace_bytes;
  a.stream = static_cast<cudaStream_t>(stream);
  return run_w8a8(a);
}

int b200q_w8a8_gemm_allreduce(const int8_t* xq, const float* a_scales, const int8_t* qweight,
                              const float* w_scales, const void* bias, void* y, int M, int N,
                              int K, int out_dtype, void* const* peer_recv,
                              void* const* peer_flags, size_t recv_bytes, int rank, int world,
                              void* stream) {
  if (xq == nullptr || a_scales == nullptr || qweight == nullptr || w_scales == nullptr ||
      y == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (out_dtype != B200Q_DTYPE_F16 && out_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (!aligned16(xq) || !aligned16(qweight) || !aligned16(y) ||
      (reinterpret_cast<uintptr_t>(a_scales) & 3u) != 0 ||
      (reinterpret_cast<uintptr_t>(w_scales) & 3u) != 0 ||
      (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0))
    return B200Q_ERR_MISALIGNED;
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  GemmArgs a{};
  a.x = xq;
  a.w = qweight;
  a.a_scales = a_scales;
  a.w_scales = w_scales;
  a.bias = bias;
  a.y = y;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = out_dtype;
  a.status = d->status_ptr;
  a.stream = static_cast<cudaStream_t>(stream);
  return launch_w8a8_mma_decode_fused(a, peer_recv, peer_flags, recv_bytes, rank, world);
}

int b200q_w8a8_gemm_allreduce_tiled(const int8_t* xq, const float* a_scales, const int8_t* qweight,
                                    const float* w_scales, const void* bias, void* const* peer_y,
                                    int M, int N, int K, int out_dtype, void* const* peer_stage,
                                    size_t stage_bytes, void* const* peer_flags, int rank,
                                    int world, void* stream) {
  if (xq == nullptr || a_scales == nullptr || qweight == nullptr || w_scales == nullptr ||
      peer_y == nullptr || peer_stage == nullptr || peer_flags == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (out_dtype != B200Q_DTYPE_F16 && out_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (world < 1 || world > 8 || rank < 0 || rank >= world) return B200Q_ERR_BAD_ARGUMENT;
  if ((N % 8) != 0 || (M % (world * 256)) != 0) return B200Q_ERR_UNSUPPORTED_SHAPE;
  if (!aligned16(xq) || !aligned16(qweight) ||
      (reinterpret_cast<uintptr_t>(a_scales) & 3u) != 0 ||
      (reinterpret_cast<uintptr_t>(w_scales) & 3u) != 0 ||
      (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0))
    return B200Q_ERR_MISALIGNED;
  if (static_cast<size_t>(M) * N * 2 > stage_bytes) return B200Q_ERR_WORKSPACE;
  for (int r = 0; r < world; ++r) {
    if (peer_y[r] == nullptr || peer_stage[r] == nullptr || peer_flags[r] == nullptr)
      return B200Q_ERR_NULL_POINTER;
    if (!aligned16(peer_y[r]) || !aligned16(peer_stage[r])) return B200Q_ERR_MISALIGNED;
  }
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  GemmArgs a{};
  a.x = xq;
  a.w = qweight;
  a.a_scales = a_scales;
  a.w_scales = w_scales;
  a.bias = bias;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = out_dtype;
  a.status = d->status_ptr;
  a.stream = static_cast<cudaStream_t>(stream);
  // test hook: 1 = GEMM kernel only, 2 = sum-and-gather kernel only (two calls make one)
  const int only = debug_knob(B200Q_KNOB_TILED_ONLY, 0);
  if (!(only & 2)) {
    if (int rc = launch_w8a8_umma_pair_scatter(a, peer_stage, rank, world)) return rc;
  }
  if (only & 1) return B200Q_OK;
  return launch_tp_reduce_gather(peer_stage[rank], peer_y, peer_flags, rank, world, M, N,
                                 out_dtype, a.stream);
}

int b200q_w8a16_gemm_allreduce(const void* x, const int8_t* qweight, const float* scales,
                               const void* bias, void* y, int M, int N, int K, int x_dtype,
                               void* const* peer_recv, void* const* peer_flags,
                               size_t recv_bytes, int rank, int world, void* stream) {
  if (x == nullptr || qweight == nullptr || scales == nullptr || y == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (x_dtype != B200Q_DTYPE_F16 && x_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (!aligned16(x) || !aligned16(qweight) || !aligned16(y) ||
      (reinterpret_cast<uintptr_t>(scales) & 3u) != 0 ||
      (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0))
    return B200Q_ERR_MISALIGNED;
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  GemmArgs a{};
  a.x = x;
  a.w = qweight;
  a.w_scales = scales;
  a.bias = bias;
  a.y = y;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = x_dtype;
  a.status = d->status_ptr;
  a.stream = static_cast<cudaStream_t>(stream);
  return launch_w8a16_mma_decode_fused(a, peer_recv, peer_flags, recv_bytes, rank, world);
}

int b200q_w8a8_gemm_i32(const int8_t* xq, const int8_t* qweight, int32_t* acc, int M, int N, int K,
                        void* workspace, size_t workspace_bytes, void* stream) {
  if (xq == nullptr || qweight == nullptr || acc == nullptr) return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (!aligned16(xq) || !aligned16(qweight) || !aligned16(acc) ||
      (workspace != nullptr && !aligned16(workspace)))
    return B200Q_ERR_MISALIGNED;
  GemmArgs a{};
  a.x = xq;
  a.w = qweight;
  a.acc_out = acc;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = B200Q_DTYPE_BF16;
  a.workspace = workspace;
  a.workspace_bytes = workspace_bytes;
  a.stream = static_cast<cudaStream_t>(stream);
  return run_w8a8(a);
}

int b200q_w8a16_gemm(const void* x, const int8_t* qweight, const float* scales, const void* bias,
                     void* y, int M, int N, int K, int x_dtype, void* workspace,
                     size_t workspace_bytes, void* stream) {
  if (x == nullptr || qweight == nullptr || scales == nullptr || y == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (x_dtype != B200Q_DTYPE_F16 && x_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (!aligned16(x) || !aligned16(qweight) || !aligned16(y) || !aligned16(scales) ||
      (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0) ||
      (workspace != nullptr && !aligned16(workspace)))
    return B200Q_ERR_MISALIGNED;
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  GemmArgs a{};
  a.x = x;
  a.w = qweight;
  a.w_scales = scales;
  a.bias = bias;
  a.y = y;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = x_dtype;
  a.workspace = workspace;
  a.workspace_bytes = workspace_bytes;
  a.status = d->status_ptr;
  a.stream = static_cast<cudaStream_t>(stream);
  const int path = resolve_path(B200Q_OP_W8A16, M, N, K);
  if (path == B200Q_PATH_SIMT_STREAM) {
    cudaError_t e = launch_w8a16_simt(a);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      return B200Q_ERR_LAUNCH;
    }
    return B200Q_OK;
  }
  if (path == B200Q_PATH_MMA_STREAM) {
    if (!mma_decode_applicable(M)) return B200Q_ERR_UNSUPPORTED_SHAPE;
    cudaError_t e = bulk_decode_applicable(M, N, K, true) ? launch_w8a16_bulk_decode(a)
                    : reg_decode_applicable(M, N, K)    ? launch_w8a16_reg_decode(a)
                                                        : launch_w8a16_mma_decode(a);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      return B200Q_ERR_LAUNCH;
    }
    return B200Q_OK;
  }
  if (path == B200Q_PATH_UMMA && umma16_mid_applicable(M, N, K)) return launch_umma16_mid(a);
  if (path == B200Q_PATH_UMMA && umma16_pair_applicable(M, N, K)) return launch_w8a16_umma_pair(a);
  if (path == B200Q_PATH_UMMA && umma16_ts_applicable(M, N, K)) return launch_w8a16_umma_ts(a);
  if (path == B200Q_PATH_UMMA || path == B200Q_PATH_UMMA_SWAP) {
    UmmaPlan plan;
    if (!umma16_make_plan(M, N, K, path == B200Q_PATH_UMMA_SWAP, &plan))
      return B200Q_ERR_UNSUPPORTED_SHAPE;
    return launch_w8a16_umma(a, plan);
  }
  return B200Q_ERR_BAD_ARGUMENT;
}

size_t b200q_w8a8_dynamic_scratch_bytes(int M, int N, int K) {
  if (check_dims(M, N, K) != B200Q_OK || dynamic_is_fused(M, N, K)) return 0;
  return dynamic_code_offset(M) + static_cast<size_t>(M) * K;
}

int b200q_w8a8_dynamic_gemm(const void* x, const int8_t* qweight, const float* w_scales,
                            const void* bias, void* y, int M, int N, int K, int x_dtype,
                            void* scratch, size_t scratch_bytes, void* workspace,
                            size_t workspace_bytes, void* stream) {
  if (x == nullptr || qweight == nullptr || w_scales == nullptr || y == nullptr)
    return B200Q_ERR_NULL_POINTER;
  if (int rc = check_dims(M, N, K)) return rc;
  if (x_dtype != B200Q_DTYPE_F16 && x_dtype != B200Q_DTYPE_BF16) return B200Q_ERR_BAD_ARGUMENT;
  if (!aligned16(x) || !aligned16(qweight) || !aligned16(y) || !aligned16(w_scales) || !aligned16(scratch) ||
      !aligned16(workspace) || (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 1u) != 0))
    return B200Q_ERR_MISALIGNED;
  if (!dynamic_is_fused(M, N, K)) {
    // what could refuse the GEMM refuses the call before the quantiser is launched
    if (scratch == nullptr || scratch_bytes < dynamic_code_offset(M) + static_cast<size_t>(M) * K)
      return B200Q_ERR_WORKSPACE;
    const size_t need = w8a8_workspace_needed(M, N, K);
    if (need > 0 && (workspace == nullptr || workspace_bytes < need)) return B200Q_ERR_WORKSPACE;
    // scales first, codes behind them
    float* a_s = static_cast<float*>(scratch);
    int8_t* xq = static_cast<int8_t*>(scratch) + dynamic_code_offset(M);
    const Carveout carve = resolve_path(B200Q_OP_W8A8, M, N, K) != B200Q_PATH_MMA_STREAM || bulk_decode_applicable(M, N, K, false)
                               ? MAX_SHARED : DEFAULT_SPLIT;
    if (int rc = run_act_quant(x, K, x_dtype, xq, a_s, M, K, carve, true, stream)) return rc;
    return b200q_w8a8_gemm(xq, a_s, qweight, w_scales, bias, y, M, N, K, x_dtype, workspace,
                           workspace_bytes, stream);
  }
  DeviceInfo* d = device_info();
  if (d == nullptr) return B200Q_ERR_LAUNCH;
  if (d->cc_major != 10) return B200Q_ERR_UNSUPPORTED_ARCH;
  GemmArgs a{};
  a.x = x;
  a.w = qweight;
  a.w_scales = w_scales;
  a.bias = bias;
  a.y = y;
  a.M = M;
  a.N = N;
  a.K = K;
  a.dtype = x_dtype;
  a.stream = static_cast<cudaStream_t>(stream);
  const cudaError_t e = launch_w8a8_reg_decode(a, true);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return B200Q_ERR_LAUNCH;
  }
  return B200Q_OK;
}

size_t b200q_workspace_bytes(int op, int M, int N, int K) {
  if (op == B200Q_OP_W8A16 && check_dims(M, N, K) == B200Q_OK &&
      resolve_path(op, M, N, K) == B200Q_PATH_UMMA) {
    if (!umma16_mid_applicable(M, N, K) && umma16_pair_applicable(M, N, K)) return umma16_pair_workspace_bytes(N, K);
  }
  if (op != B200Q_OP_W8A8 && op != B200Q_OP_W8A16) return 0;
  if (check_dims(M, N, K) != B200Q_OK) return 0;
  const int path = resolve_path(op, M, N, K);
  if (path != B200Q_PATH_UMMA && path != B200Q_PATH_UMMA_SWAP) return 0;
  // (an upper bound at sizes where gemm_umma_mid.cu, which needs none, takes over the W8A8 problem)
  if (path == B200Q_PATH_UMMA && op == B200Q_OP_W8A16 && umma16_mid_applicable(M, N, K)) return 0;
  if (path == B200Q_PATH_UMMA && op == B200Q_OP_W8A16 && umma16_ts_applicable(M, N, K)) return 0;
  UmmaPlan plan;
  const bool ok = op == B200Q_OP_W8A8
                      ? umma_make_plan(op, M, N, K, path == B200Q_PATH_UMMA_SWAP, &plan)
                      : umma16_make_plan(M, N, K, path == B200Q_PATH_UMMA_SWAP, &plan);
  return ok ? plan.ws_bytes : 0;
}

const char* b200q_select_path(int op, int M, int N, int K) {
  if (op == B200Q_OP_ACT_QUANT) {
    if (M <= 0 || K <= 0 || (K % 16) != 0) return "unsupported_shape";
    if (act_quant_long_row(K)) return "act_quant_long_row";
    return row_shape(M, K >> 3).g == 32 ? "act_quant_warp_per_row" : "act_quant_multiwarp_row";
  }
  if (op != B200Q_OP_W8A8 && op != B200Q_OP_W8A16) return "invalid_op";
  if (check_dims(M, N, K) != B200Q_OK) return "unsupported_shape";
  const int path = resolve_path(op, M, N, K);
  const bool a16 = op == B200Q_OP_W8A16;
  switch (path) {
    case B200Q_PATH_SIMT_STREAM:
      return a16 ? "simt_stream_w8a16" : "simt_stream_dp4a";
    case B200Q_PATH_MMA_STREAM:
      if (bulk_decode_applicable(M, N, K, a16))
        return a16 ? "bulk_ring_w8a16_persistent" : "bulk_ring_s8_persistent";
      return a16 ? "mma_stream_w8a16_splitk" : "mma_stream_s8_splitk";
    case B200Q_PATH_UMMA:
      if (!a16 && umma_pair_applicable(M, N, K, false)) return "umma_i8_pair_tokens256";
      // the single-CTA kernels of a scheme (gemm_umma_mid.cu and gemm_umma.cu; gemm_umma_mid_w8a16.cu and
      // gemm_umma_w8a16.cu) are one family
      if (a16 && !umma16_mid_applicable(M, N, K)) {
        if (umma16_pair_applicable(M, N, K)) return "umma_f16_pair_expand_once_tokens256";
        if (umma16_ts_applicable(M, N, K)) return "umma_f16_tmem_weights_channels256";
      }
      return a16 ? "umma_f16_expand_tokens128" : "umma_i8_tokens128";
    case B200Q_PATH_UMMA_SWAP:
      return a16 ? "umma_f16_expand_channels128_splitk" : "umma_i8_channels128_splitk";
    default:
      return "invalid_path";
  }
}

const char* b200q_strerror(int code) {
  switch (code) {
    case B200Q_OK:
      return "ok";
    case B200Q_ERR_NULL_POINTER:
      return "a required pointer is NULL";
    case B200Q_ERR_BAD_SHAPE:
      return "M, N or K is not positive or too large";
    case B200Q_ERR_UNSUPPORTED_SHAPE:
      return "unsupported shape (K must be a multiple of 16; row pitch rules)";
    case B200Q_ERR_MISALIGNED:
      return "a pointer is not sufficiently aligned (16 bytes)";
    case B200Q_ERR_WORKSPACE:
      return "workspace missing or smaller than b200q_workspace_bytes()";
    case B200Q_ERR_UNSUPPORTED_ARCH:
      return "device is not compute capability 10.x (B200)";
    case B200Q_ERR_LAUNCH:
      return "a CUDA call failed (see b200q_last_cuda_error)";
    case B200Q_ERR_BAD_ARGUMENT:
      return "unknown op, dtype or path id";
    case B200Q_ERR_DEVICE_TIMEOUT:
      return "a bounded device-side wait gave up";
    case B200Q_ERR_SCRATCH_LIMIT:
      return "problem needs more scratch than the library's built-in 8 MiB array; "
             "use b200q_w8a8_gemm with a caller-owned workspace";
    default:
      return "unknown error code";
  }
}

int b200q_last_cuda_error(void) { return g_last_cuda_error.load(); }

int b200q_device_status(void) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_device_status, sizeof(int));
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return -1;
  }
  if (v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
  }
  return v;
}

int b200q_check_status(int* status_word) {
  const int v = b200q_device_status();
  if (status_word != nullptr) *status_word = v;
  if (v < 0) return B200Q_ERR_LAUNCH;
  return v == 0 ? B200Q_OK : B200Q_ERR_DEVICE_TIMEOUT;
}

int b200q_version(void) { return B200Q_VERSION; }

int b200q_debug_force_path(int path) {
  if (path < B200Q_PATH_AUTO || path > B200Q_PATH_MMA_STREAM) return -1;
  const int prev = debug_knob(B200Q_KNOB_FORCE_PATH, B200Q_PATH_AUTO);
  t_knobs.value[B200Q_KNOB_FORCE_PATH] = path;
  t_knobs.set[B200Q_KNOB_FORCE_PATH] = path != B200Q_PATH_AUTO;
  return prev;
}

int b200q_debug_set(int knob, int value) {
  if (knob < 0 || knob >= B200Q_KNOB_COUNT) return -1;
  t_knobs.value[knob] = value;
  t_knobs.set[knob] = true;
  return 0;
}

void b200q_debug_reset(void) { t_knobs = Knobs{}; }

int b200q_debug_mid_plan(int op, int M, int N, int K, int* plan) {
  if (plan == nullptr || (op != B200Q_OP_W8A8 && op != B200Q_OP_W8A16) || check_dims(M, N, K) != B200Q_OK) return 0;
  if (resolve_path(op, M, N, K) != B200Q_PATH_UMMA) return 0;
  MidShape s;
  if (op == B200Q_OP_W8A8 ? umma_pair_applicable(M, N, K, false) || !umma_mid_shape(M, N, K, &s)
                          : !umma16_mid_shape(M, N, K, &s))
    return 0;
  const int v[6] = {s.tokens, s.channels, s.cluster, s.tmem_cols, s.smem_bytes, s.ctas};
  for (int i = 0; i < 6; ++i) plan[i] = v[i];
  return 1;
}

uint64_t b200q_debug_maps_encoded(void) { return maps_encoded(); }

uint64_t b200q_launch_count(void) { return g_launches.load(); }

}  // extern "C"
