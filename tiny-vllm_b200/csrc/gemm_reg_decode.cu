// Decode kernels for at most 16 tokens over matrices that fit the register files of the GPU (a few MB):
// the whole weight matrix is in registers before the activations exist.
//
// A decode step is a chain of dependent launches of a few microseconds, so what counts is what happens
// between the end of one kernel and the end of the next.  Weights are constants: every CTA loads its
// weights (32 KB: 8 pieces of 16 bytes per lane) and, for W8A16, expands them to 16 bits BEFORE it waits for
// the kernel that produces its activations (griddepcontrol.wait), and lets its own successor start at
// once; 128 registers per thread leave room for two CTAs per SM, so that the successor can do the
// same.  After the wait there is one trip to L2 for the activations, the MMAs, a reduction over
// the CTA's warps in shared memory and the store.
//
//   * a CTA owns 8 NT channels and all of K, cut over its 8 warps into BLK blocks of 64 each: NT x BLK = 8
//     pieces per lane, NT = 4 for K <= 1024 (each activation fragment feeds four MMA tiles), 2 for
//     K <= 2048, 1 beyond;
//   * within a block lane (g = lane / 4, t = lane % 4) owns elements [16 t, 16 t + 16) of weight row g and of
//     token rows g and g + 8.  Which physical k sits in which MMA slot does not matter as long as both
//     operands agree, so neither needs a shuffle (as in gemm_mma_decode.cu);
//   * REG_A8_DYN takes 16-bit activations and quantises them itself, into shared memory, with the arithmetic
//     of act_quant.cu (same codes, same scales), instead of a kernel and a launch of their own.
//
// Arithmetic as in gemm_mma_decode.cu: exact int32 sums, then (float(acc) * a_s[m]) * w_s[n] + b[n]
// (nanovllm/quantization/csrc/w8a8_gemm.cu:165-183, 387-390); fp32 sums of x * float(q), then
// acc * s[n] + b[n] (nanovllm/quantization/csrc/int8_weight_only_gemm.cu:258-292).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "act_quant_device.cuh"
#include "common.h"
#include "expand_device.cuh"
#include "mma_device.cuh"
#include "ptx_sm100.cuh"

namespace b200q {
namespace {

enum { REG_A16 = 0, REG_A8 = 1, REG_A8_RAW = 2, REG_A8_DYN = 3 };

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kCodePad = 64; // spreads the rows of codes over the banks
constexpr int kBlock = 64;   // K elements of a block: one 16-byte piece of weights per lane

struct RegParams {
  const void* x;            // int8 codes or 16-bit activations [M, K]
  const int8_t* w;          // [N, K]
  const float* a_s;         // [M] (REG_A8)
  const float* w_s;         // [N]
  const void* bias;         // [N] or nullptr
  void* out;                // [M, N]
  int M, N, K;
};

// What the previous kernel wrote: ordinary loads, which stay behind the wait.  (A non-coherent load,
// __ldg, is taken for one of constant memory and may be moved ahead of it: chains of dependent
// launches then read stale activations.)
__device__ __forceinline__ uint4 load_or_zero(const void* p, bool ok) {
  return ok ? *reinterpret_cast<const uint4*>(p) : make_uint4(0u, 0u, 0u, 0u);
}

// Constants of the layer: volatile loads keep their place ahead of the wait (ordinary ones sink to their
// first use, and a scale fetched from HBM after the MMAs costs a microsecond).
__device__ __forceinline__ uint4 ldg_weights(const int8_t* p, bool ok) {
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (ok)
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
  return v;
}
__device__ __forceinline__ float ldg_scale(const float* p, bool ok) {
  float v = 0.f;
  if (ok) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
template <typename T>
__device__ __forceinline__ float ldg_bias(const void* bias, int n, bool ok) {
  uint16_t v = 0;
  if (ok) asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(static_cast<const T*>(bias) + n));
  return to_float<T>(*reinterpret_cast<const T*>(&v));
}

// Per-token quantisation of x [M, K] into the CTA's shared memory, value for value what act_quant.cu
// writes to memory.  8 / G rows at a time, G warps to a row (all eight for a single token); loops
// instead of unrolled code, because an instruction that runs once per launch costs its fetch.
template <typename T>
__device__ __forceinline__ void quantise_rows(const RegParams& p, uint8_t* codes, float* s_max, float* s_scale) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int shift = p.M == 1 ? 3 : p.M == 2 ? 2 : p.M <= 4 ? 1 : 0;       // G = 1 << shift
  const int sub = warp & ((1 << shift) - 1), step = 32 << shift;
  const int nchunk = p.K >> 3;                                            // 16 bytes of x
#pragma unroll 1
  for (int row = warp >> shift; row < p.M; row += kWarps >> shift) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + static_cast<size_t>(row) * p.K);
    AbsMax2<T> m;
#pragma unroll 4
    for (int i = sub * 32 + lane; i < nchunk; i += step) {
      const uint4 v = src[i];
      m.add(v.x);
      m.add(v.y);
      m.add(v.z);
      m.add(v.w);
    }
    float amax = warp_max(m.value());
    if (shift > 0) {   // then there is one pass, and all warps of the row are in it
      if (lane == 0) s_max[warp] = amax;
      ptx::named_bar_sync(1 + (warp >> shift), step);
      for (int i = 0; i < (1 << shift); ++i) amax = fmaxf(amax, s_max[(warp & ~((1 << shift) - 1)) + i]);
    }
    const float scale = fmaxf(__fdiv_rn(amax, 127.0f), 1e-8f), inv = __frcp_rn(scale);
    if (sub == 0 && lane == 0) s_scale[row] = scale;
    uint2* dst = reinterpret_cast<uint2*>(codes + row * (p.K + kCodePad));
#pragma unroll 2
    for (int i = sub * 32 + lane; i < nchunk; i += step) dst[i] = quant8<T>(src[i], scale, inv);   // from L1
  }
  __syncthreads();
}

// HI: token rows 8-15 exist (M > 8).
template <int KIND, typename T, int NT, int BLK, bool HI>
__global__ void __launch_bounds__(kThreads, 2) reg_decode_kernel(const RegParams p) {
  constexpr bool k16 = KIND == REG_A16;                    // 16-bit operands, fp32 sums
  constexpr bool kX16 = KIND == REG_A16 || KIND == REG_A8_DYN;
  constexpr int kCh = 8 * NT;
  __shared__ uint32_t red[kWarps][16 * kCh];
  __shared__ float s_max[kWarps], s_scale[16];              // REG_A8_DYN
  extern __shared__ __align__(16) uint8_t s_codes[];        // REG_A8_DYN: [M][K + kCodePad]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kCh;
  const int k0 = warp * (BLK * kBlock) + 16 * t;           // this lane's first element

  // ------------------------------------------------ before the wait: weights, scales
  uint4 wv[NT][BLK];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int n = n0 + 8 * j + g;
    const int8_t* row = p.w + static_cast<size_t>(n < p.N ? n : 0) * p.K;
#pragma unroll
    for (int b = 0; b < BLK; ++b) wv[j][b] = ldg_weights(row + k0 + b * kBlock, n < p.N && k0 + b * kBlock < p.K);
  }
  ptx::grid_launch_dependents();
  constexpr int kOut = 16 * kCh / kThreads > 0 ? 16 * kCh / kThreads : 1;   // outputs per thread
  float o_scale[kOut], o_bias[kOut];
#pragma unroll
  for (int i = 0; i < kOut; ++i) {
    const int n = n0 + (threadIdx.x + i * kThreads) % kCh;
    o_scale[i] = ldg_scale(p.w_s + n, KIND != REG_A8_RAW && n < p.N);
    o_bias[i] = ldg_bias<T>(p.bias, n, p.bias != nullptr && n < p.N);
  }
  uint2 e[k16 ? NT : 1][k16 ? BLK : 1][4];                 // expanded weights
  if (k16) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int b = 0; b < BLK; ++b) {
        e[j][b][0] = expand4<T>(wv[j][b].x);
        e[j][b][1] = expand4<T>(wv[j][b].y);
        e[j][b][2] = expand4<T>(wv[j][b].z);
        e[j][b][3] = expand4<T>(wv[j][b].w);
      }
  }
  // (never taken: it ends a basic block, so that the expansion is not scheduled behind the wait to save
  // registers — 2.3 against 1.7 us on 4096 x 1024)
  if (p.M < 0) ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();                             // activations, and the output's memory

  // ------------------------------------------------------------- activations, MMAs
  constexpr int kElem = kX16 ? 2 : 1;
  // 16 tokens at a time (one pass up to 16): the weights stay where they are
#pragma unroll 1
  for (int tok0 = 0; tok0 < p.M; tok0 += 16) {
  const bool lo_ok = tok0 + g < p.M, hi_ok = HI && tok0 + g + 8 < p.M;
  const char* x_lo = static_cast<const char*>(p.x) + (static_cast<size_t>(tok0 + g) * p.K + k0) * kElem;
  const char* x_hi = x_lo + static_cast<size_t>(8) * p.K * kElem;

  float facc[NT][4];
  int iacc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      facc[j][i] = 0.f;
      iacc[j][i] = 0;
    }

  if (k16) {
    // blocks whose activations are requested together: 16 registers a block (8 without HI)
    constexpr int kBatch = BLK < (HI ? 2 : 4) ? BLK : (HI ? 2 : 4);
#pragma unroll
    for (int b0 = 0; b0 < BLK; b0 += kBatch) {
      uint4 xl[kBatch][2], xh[kBatch][2];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int off = (b0 + i) * kBlock;
        const bool k_ok = b0 + i < BLK && k0 + off < p.K;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          xl[i][h] = load_or_zero(x_lo + off * 2 + 16 * h, lo_ok && k_ok);
          xh[i][h] = load_or_zero(x_hi + off * 2 + 16 * h, hi_ok && k_ok);
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        if (b0 + i >= BLK) break;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint2(&w)[4] = e[k16 ? j : 0][k16 ? b0 + i : 0];
          mma_16<T>(facc[j], xl[i][0].x, xh[i][0].x, xl[i][0].y, xh[i][0].y, w[0].x, w[0].y);
          mma_16<T>(facc[j], xl[i][0].z, xh[i][0].z, xl[i][0].w, xh[i][0].w, w[1].x, w[1].y);
          mma_16<T>(facc[j], xl[i][1].x, xh[i][1].x, xl[i][1].y, xh[i][1].y, w[2].x, w[2].y);
          mma_16<T>(facc[j], xl[i][1].z, xh[i][1].z, xl[i][1].w, xh[i][1].w, w[3].x, w[3].y);
        }
      }
    }
  } else {
    if (KIND == REG_A8_DYN) quantise_rows<T>(p, s_codes, s_max, s_scale);
#pragma unroll
    for (int b = 0; b < BLK; ++b) {
      const bool k_ok = k0 + b * kBlock < p.K;
      uint4 a, c = make_uint4(0u, 0u, 0u, 0u);
      if (KIND == REG_A8_DYN) {
        const uint8_t* row = s_codes + g * (p.K + kCodePad) + k0 + b * kBlock;
        a = lo_ok && k_ok ? *reinterpret_cast<const uint4*>(row) : make_uint4(0u, 0u, 0u, 0u);
        if (hi_ok && k_ok) c = *reinterpret_cast<const uint4*>(row + 8 * (p.K + kCodePad));
      } else {
        a = load_or_zero(x_lo + b * kBlock, lo_ok && k_ok);
        c = load_or_zero(x_hi + b * kBlock, hi_ok && k_ok);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        // bytes 0-7 feed the first k32 step, bytes 8-15 the second
        mma_s8(iacc[j], a.x, c.x, a.y, c.y, wv[j][b].x, wv[j][b].y);
        mma_s8(iacc[j], a.z, c.z, a.w, c.w, wv[j][b].z, wv[j][b].w);
      }
    }
  }

  // C fragment: [0..1] = (token g, channels 2t, 2t + 1 of the tile), [2..3] = token g + 8
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (!HI && i >= 2) continue;
      red[warp][(g + (i >> 1) * 8) * kCh + 8 * j + 2 * t + (i & 1)] =
          k16 ? __float_as_uint(facc[j][i]) : static_cast<uint32_t>(iacc[j][i]);
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOut; ++i) {
    const int o = threadIdx.x + i * kThreads;
    const int tok = tok0 + o / kCh, n = n0 + o % kCh;
    if (o >= 16 * kCh || tok >= p.M || n >= p.N) continue;
    const size_t at = static_cast<size_t>(tok) * p.N + n;
    if (k16) {
      float sum = 0.f;
#pragma unroll
      for (int wi = 0; wi < kWarps; ++wi) sum = __fadd_rn(sum, __uint_as_float(red[wi][o]));   // fixed order
      reinterpret_cast<T*>(p.out)[at] = from_float<T>(__fadd_rn(__fmul_rn(sum, o_scale[i]), o_bias[i]));
    } else {
      int sum = 0;
#pragma unroll
      for (int wi = 0; wi < kWarps; ++wi) sum += static_cast<int>(red[wi][o]);
      if (KIND == REG_A8_RAW) {
        reinterpret_cast<int32_t*>(p.out)[at] = sum;
      } else {
        const float a_s = KIND == REG_A8_DYN ? s_scale[tok] : p.a_s[tok];
        reinterpret_cast<T*>(p.out)[at] = from_float<T>(
            __fadd_rn(__fmul_rn(__fmul_rn(static_cast<float>(sum), a_s), o_scale[i]), o_bias[i]));
      }
    }
  }
  if (tok0 + 16 < p.M) __syncthreads();   // the partial sums have been read
  }
}

template <int KIND, typename T, int NT, int BLK>
cudaError_t launch_hi(const RegParams& p, cudaStream_t stream) {
  const dim3 grid((p.N + 8 * NT - 1) / (8 * NT));
  const size_t smem = KIND == REG_A8_DYN ? static_cast<size_t>(p.M) * (p.K + kCodePad) : 0;
  return p.M > 8 ? launch_overlapped(DEFAULT_SPLIT, reg_decode_kernel<KIND, T, NT, BLK, true>, grid, dim3(kThreads), smem, stream, p)
                 : launch_overlapped(DEFAULT_SPLIT, reg_decode_kernel<KIND, T, NT, BLK, false>, grid, dim3(kThreads), smem, stream, p);
}

template <int KIND, typename T>
cudaError_t launch_reg(const RegParams& p, cudaStream_t stream) {
  if (p.K <= 512) return launch_hi<KIND, T, 4, 1>(p, stream);
  if (p.K <= 1024) return launch_hi<KIND, T, 4, 2>(p, stream);
  if (p.K <= 1536) return launch_hi<KIND, T, 2, 3>(p, stream);
  if (p.K <= 2048) return launch_hi<KIND, T, 2, 4>(p, stream);
  if (p.K <= 3072) return launch_hi<KIND, T, 1, 6>(p, stream);
  return launch_hi<KIND, T, 1, 8>(p, stream);
}

template <int KIND>
cudaError_t launch_kind(const RegParams& p, int dtype, cudaStream_t stream) {
  return dtype == B200Q_DTYPE_BF16 ? launch_reg<KIND, __nv_bfloat16>(p, stream)
                                   : launch_reg<KIND, __half>(p, stream);
}

RegParams params_of(const GemmArgs& a) {
  return RegParams{a.x, a.w, a.a_scales, a.w_scales, a.bias, a.acc_out != nullptr ? a.acc_out : a.y,
                   a.M, a.N, a.K};
}

}  // namespace

// K <= 4096: a warp's share of a row fits its registers.
bool reg_decode_applicable(int M, int N, int K) {
  return M >= 1 && M <= 64 && K <= kWarps * 8 * kBlock && debug_knob(B200Q_KNOB_NO_REG, 0) == 0;
}

// Where it is the fastest kernel (us, chains of launches, W8A8 / W8A16).
// * Up to 16 tokens and K <= 2048 always: 4096 x 1024 at 16 2.3 / 2.5 (register-streaming kernel without the early
//   weights: 3.5 / 4.2), 12288 x 2048 6.7 / 9.6 (ring: 7.7 / 12.8).  Longer rows leave one MMA tile per
//   activation fragment, so only while the matrix is one wave of CTAs: 2048 x 4096 3.1 / 4.4 (4.8 / 6.1), but
//   4096 x 4096 5.9 / 8.8 (5.3 / 8.9) and 5120 x 2560 5.7 / 8.5 (4.6 / 7.4).
// * 17 to 32 tokens take a second pass over the activations; the tcgen05 kernels are the rivals.  W8A8 at 32:
//   1024 x 2048 2.7 (3.4), 4096 x 1536 3.1 (4.5), but 6144 x 1024 3.8 (3.6).  W8A16: 4096 x 1024 at 32 3.6
//   (3.9), 1024 x 3072 at 24 4.1 (4.3) but at 32 4.7 (4.4), 1024 x 4096 at 17 5.0 (4.5), 4096 x 1024 at 40 4.5 (4.2).
bool reg_decode_preferred(int M, int N, int K, bool a16) {
  if (!reg_decode_applicable(M, N, K)) return false;
  const bool one_wave = static_cast<long long>(N) * K <= (17ll << 19);   // 8.5 MB
  if (M <= 16) return K <= 2048 || one_wave;
  if (!a16) return M <= 32 && one_wave && N <= 5120;
  // W8A16: until the tcgen05 kernel is ahead (that one needs whole groups of 8 channels)
  return one_wave && (M <= 24 ? K <= 3072 : M <= 32 ? K <= 2048 : M <= 48 && K <= 1536 && (N % 8) != 0);
}

// Every CTA quantises all tokens, so only few values: 8 tokens of 1024 3.6 us in all against 4.4 in two kernels, 16
// tokens 5.5 against 4.6.
bool reg_decode_dynamic_applicable(int M, int N, int K) {
  return M <= 16 && reg_decode_applicable(M, N, K) && M * K <= 8192;
}

cudaError_t launch_w8a16_reg_decode(const GemmArgs& a) {
  const cudaError_t e = launch_kind<REG_A16>(params_of(a), a.dtype, a.stream);
  if (e == cudaSuccess) count_launch();
  return e;
}

cudaError_t launch_w8a8_reg_decode(const GemmArgs& a, bool dynamic) {
  const RegParams p = params_of(a);
  const cudaError_t e = a.acc_out != nullptr ? launch_reg<REG_A8_RAW, __nv_bfloat16>(p, a.stream)
                        : dynamic            ? launch_kind<REG_A8_DYN>(p, a.dtype, a.stream)
                                             : launch_kind<REG_A8>(p, a.dtype, a.stream);
  if (e == cudaSuccess) count_launch();
  return e;
}

}  // namespace b200q
