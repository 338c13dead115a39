// Internal declarations shared by the translation units of libb200q.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/b200q.h"

namespace b200q {

// One linear-layer problem, in the vocabulary of the layer: M tokens, K input
// features, N output channels.
struct GemmArgs {
  const void* x;          // int8 [M,K] (W8A8) or f16/bf16 [M,K] (W8A16)
  const int8_t* w;        // int8 [N,K]
  const float* a_scales;  // fp32 [M]  (W8A8 only)
  const float* w_scales;  // fp32 [N]
  const void* bias;       // [N] in `dtype`, or nullptr
  void* y;                // [M,N] in `dtype`            (nullptr in int32 mode)
  int32_t* acc_out;       // [M,N] raw accumulators      (int32 mode only)
  int M, N, K;
  int dtype;              // B200Q_DTYPE_*
  void* workspace;
  size_t workspace_bytes;
  int* status;            // device status word of the current device
  cudaStream_t stream;
};

// Tiling of one problem onto the tcgen05 kernel.  "A side" is the operand that
// fills the 128 rows of the UMMA tile, "B side" the one that fills its columns.
struct UmmaPlan {
  int swap;          // 0: A = tokens, B = channels; 1: A = channels, B = tokens
  int rows_a, rows_b;
  int bn;            // B-side tile (UMMA N), multiple of 32, <= 256
  int tiles_a, tiles_b;
  int k_blocks;      // ceil(K_bytes / 128)
  int splits;        // split-K factor
  int kb_per_split;
  int stages;        // shared-memory ring depth
  int conv_bufs;     // W8A16 only: ring depth of the converted (16-bit) weight tiles
  int cluster;       // CTAs per cluster that split K and reduce through shared memory (1 = off)
  int partial_bytes; // shared memory for the partial tiles the cluster leader receives
  int tmem_cols;     // power of two >= 2 * bn
  int grid;          // CTAs launched (persistent)
  size_t smem_bytes;
  size_t ws_bytes;   // counters + split-K partials (0 when splits == 1)
};

constexpr size_t kCounterBytes = 16384;  // zero-initialised tile counters at workspace start

// Shared memory of an SM, and what a CTA takes beyond its own.  The CTA-pair kernel allocates all of an SM's tensor memory
// for a cluster, so no CTA of another cluster that allocates some may be beside it (the residency rule of
// umma_mid_common.cuh): it asks for kPairSmem, and such a CTA for kClusterSmemMin at least.  The 9 KB that are left hold the
// CTAs of the kernels that quantise activations.
constexpr int kSmSharedBytes = 228 * 1024, kCtaSharedExtra = 1024;
constexpr int kPairSmem = 218 * 1024, kClusterSmemMin = 12 * 1024;
static_assert(kPairSmem + kClusterSmemMin + 2 * kCtaSharedExtra > kSmSharedBytes, "a cluster beside the CTA-pair kernel");

// Number of SMs of the current device (cached).
int sm_count();

// Row-wise kernels: threads per row (32 to 256) and 16-byte chunks per thread.  While all rows fit the GPU at
// once, what counts is the chain of one thread: as few chunks as one wave of threads allows.  Beyond, four
// chunks keep enough bytes in flight at a moderate register count.  (us, one chunk / this rule / always four:
// quantiser, K = 1024, 512 tokens 2.2 / 2.2 / 2.9, 1999 3.1 / 3.2 / 4.5, 8192 7.9 / 6.8 / 6.8; RMSNorm, K = 2048,
// 256 tokens 3.4 / 3.4 / 4.1, 8192 28.6 / 22.5 / 22.5.)
struct RowShape {
  int g, c;
};
inline RowShape row_shape(int M, int nchunk) {
  const long long wave = static_cast<long long>(sm_count()) * 2048;
  int c = 1;
  while (c < 4 && static_cast<long long>(M) * nchunk > c * wave) ++c;
  int g = 32;
  while (g < 256 && g * c < nchunk) g *= 2;
  return {g, (nchunk + g - 1) / g};
}

// Compute-capability major of the current device (0 on error) and the device address of
// its status word (nullptr on error); both cached per device.
int device_cc_major();
int* device_status_ptr();

// An SM divides its memory between L1 and shared memory by the kernel that starts on it and cannot change that while
// CTAs run.  A kernel that would leave most of it to L1, and stands between two that need nearly all of it as shared memory,
// keeps the second one off its SMs until it has ended; so does one with less of its own.  MAX_SHARED asks for the division
// that those need: for the tcgen05 (from 33 tokens on) and ring kernels and for what quantises their activations (256 tokens of the 0.6B
// model, W8A8, 376 -> 359 us), not for the kernels that live on L1 (16 tokens, weights in registers, 129 -> 157 us).
enum Carveout { DEFAULT_SPLIT = 0, MAX_SHARED = 1 };

// act_quant.cu: rows too long for a thread group's registers are read twice
inline bool act_quant_long_row(int K) { return K > 256 * 8 * 8; }
// early: the next kernel takes the codes as activations and may start at once; carve: what suits that kernel
cudaError_t launch_act_quant(const void* x, int64_t ldx, int x_dtype, int8_t* xq, float* a_scales,
                             int M, int K, bool early, Carveout carve, cudaStream_t stream);

// gemm_simt.cu
cudaError_t launch_w8a8_simt(const GemmArgs& a);
cudaError_t launch_w8a16_simt(const GemmArgs& a);

// gemm_mma_decode.cu: weight-streaming mma.sync kernels for M <= 64
bool mma_decode_applicable(int M);
cudaError_t launch_w8a8_mma_decode(const GemmArgs& a);
cudaError_t launch_w8a16_mma_decode(const GemmArgs& a);
// The same kernels with the row-parallel sum over peer memory fused in; return B200Q_* codes.
int launch_w8a8_mma_decode_fused(const GemmArgs& a, void* const* peer_recv,
                                 void* const* peer_flags, size_t recv_bytes, int rank, int world);
int launch_w8a16_mma_decode_fused(const GemmArgs& a, void* const* peer_recv,
                                  void* const* peer_flags, size_t recv_bytes, int rank, int world);

// gemm_reg_decode.cu: few tokens, the weights in registers before the activations exist;
// applicable = can run, preferred = is the fastest; `dynamic`: a.x holds 16-bit activations that the kernel quantises itself
bool reg_decode_applicable(int M, int N, int K);
bool reg_decode_preferred(int M, int N, int K, bool a16);
bool reg_decode_dynamic_applicable(int M, int N, int K);
cudaError_t launch_w8a8_reg_decode(const GemmArgs& a, bool dynamic);
cudaError_t launch_w8a16_reg_decode(const GemmArgs& a);

// gemm_bulk_decode.cu: persistent decode kernels for large matrices; a producer warp streams
// weights and activations through a shared-memory ring of bulk asynchronous copies
bool bulk_decode_applicable(int M, int N, int K, bool a16);
bool bulk_decode_yields(int M, int N, int K);
cudaError_t launch_w8a8_bulk_decode(const GemmArgs& a);
cudaError_t launch_w8a16_bulk_decode(const GemmArgs& a);

// gemm_umma.cu
bool umma_make_plan(int op, int M, int N, int K, int swap, UmmaPlan* plan);
// Returns a B200Q_* code.
int launch_w8a8_umma(const GemmArgs& a, const UmmaPlan& plan);

// gemm_umma.cu: TMA descriptor of a dense row-major matrix viewed as bytes [rows, row_bytes],
// box = box_bytes (128: 128-byte swizzle, 64: 64-byte swizzle) x box_rows, zero fill outside.
// box_blocks > 0: a 3-D view [row_bytes / box_bytes][rows][box_bytes] of the whole blocks of a row,
// whose box holds that many blocks of box_bytes x box_rows.
// make_tensor_map encodes on every call (activations and outputs: their addresses change from
// call to call); get_tensor_map keeps the result in a per-process cache (weights: same
// address for the life of the model).
bool make_tensor_map(const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
                     uint32_t box_bytes, CUtensorMap* out, uint32_t box_blocks = 0);
bool get_tensor_map(const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
                    uint32_t box_bytes, CUtensorMap* out, uint32_t box_blocks = 0);
uint64_t maps_encoded();   // how many descriptors this process has encoded

// Test and tuning hooks (B200Q_KNOB_* of b200q.h).  Every knob is unset (the built-in
// behaviour) until the CALLING THREAD sets it through b200q_debug_set(); nothing is read from
// the environment, so a stray variable can never change what a kernel computes.
int debug_knob(int knob, int dflt);
// Limit of one wait on a peer GPU in SM cycles: about a second unless a test shortened it.
inline long long peer_wait_limit_cycles() {
  const int k = debug_knob(B200Q_KNOB_WAIT_CYCLES, 0);
  return k > 0 ? static_cast<long long>(k) : 2000000000LL;
}

// gemm_umma_pair.cu: CTA-pair (cta_group::2) variant for prefill-sized W8A8 problems
bool umma_pair_applicable(int M, int N, int K, bool raw_int32_out);
int launch_w8a8_umma_pair(const GemmArgs& a);
// Row-parallel prefill: the pair kernel writing its partial tiles to the owners' staging areas
// (reduce-scatter under the main loop), and the kernel that sums and gathers them.
int launch_w8a8_umma_pair_scatter(const GemmArgs& a, void* const* peer_stage, int rank,
                                  int world);
int launch_tp_reduce_gather(const void* stage, void* const* peer_y,
                            void* const* peer_ctl, int rank, int world, int M, int N, int dtype,
                            cudaStream_t stream);

// gemm_umma_pair.cu: W8A16 prefill route — weights expanded once per call into the
// workspace, then the 16-bit CTA-pair kernel
bool umma16_pair_applicable(int M, int N, int K);
size_t umma16_pair_workspace_bytes(int N, int K);
int launch_w8a16_umma_pair(const GemmArgs& a);

// gemm_umma_mid.cu, gemm_umma_mid_w8a16.cu: tens to hundreds of tokens (W8A8: up to a wave of 128 x 128 tiles; W8A16: 2.6
// waves, at most 2048 tokens), one tile per CTA, K split over a cluster
bool umma_mid_applicable(int M, int N, int K);
int launch_umma_mid(const GemmArgs& a);
bool umma16_mid_applicable(int M, int N, int K);
int launch_umma16_mid(const GemmArgs& a);
// How these kernels would cut a problem (tests); false where they cannot.
struct MidShape {
  int tokens, channels;   // of a tile
  int cluster, tmem_cols, smem_bytes, ctas;
};
bool umma_mid_shape(int M, int N, int K, MidShape* s);
bool umma16_mid_shape(int M, int N, int K, MidShape* s);

// gemm_umma_w8a16.cu
bool umma16_make_plan(int M, int N, int K, int swap, UmmaPlan* plan);
int launch_w8a16_umma(const GemmArgs& a, const UmmaPlan& plan);

// gemm_umma_w8a16_ts.cu: prefill variant with the expanded weights in tensor memory
bool umma16_ts_applicable(int M, int N, int K);
int launch_w8a16_umma_ts(const GemmArgs& a);

// Launches `kernel` so that it may overlap its start-up (barrier set-up, TMEM allocation,
// descriptor prefetch, launch latency, first weights) with the tail of the previous kernel in the
// stream (programmatic dependent launch).  Only for kernels that call ptx::grid_dependency_wait()
// before their first access to what that kernel, or one before it, may read or write.  Weights, their scales
// and the bias count as constants (b200q.h states the caller's side): they may be read before the
// wait.  A predecessor that does not call ptx::grid_launch_dependents() has then ended, and with it all
// that was ahead of it; so a kernel whose output may become somebody's weights must not call it
// (act_quant.cu).  B200Q_KNOB_NO_PDL turns the overlap off.
bool pdl_enabled();
template <typename... KArgs, typename... Args>
cudaError_t launch_clustered(Carveout carve, int cluster, bool overlap, void (*kernel)(KArgs...), dim3 grid,
                             dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (overlap && pdl_enabled()) ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (carve == MAX_SHARED) {
    cudaLaunchAttribute& c = attr[cfg.numAttrs++];
    c.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    c.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
  }
  if (cluster > 1) {  // grid.x must be a multiple of the cluster size
    cudaLaunchAttribute& c = attr[cfg.numAttrs++];
    c.id = cudaLaunchAttributeClusterDimension;
    c.val.clusterDim.x = static_cast<unsigned int>(cluster);
    c.val.clusterDim.y = 1;
    c.val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_maybe_overlapped(bool overlap, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                                    size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_clustered(DEFAULT_SPLIT, 1, overlap, kernel, grid, block, smem, stream,
                          static_cast<Args&&>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_overlapped(Carveout carve, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, Args&&... args) {
  return launch_clustered(carve, 1, true, kernel, grid, block, smem, stream, static_cast<Args&&>(args)...);
}

void note_cuda_error(cudaError_t e);
void count_launch(int n = 1);

}  // namespace b200q
