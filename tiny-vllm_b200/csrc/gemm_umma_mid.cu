// Decode- and short-prompt-sized GEMMs (tens to hundreds of tokens) on tcgen05, both schemes:
//   W8A8   int8 x int8 -> int32 (kind::i8), (float(acc) * a_s[m]) * w_s[n] + b[n]
//          (nanovllm/quantization/csrc/w8a8_gemm.cu:165-183, 387-390)
//   W8A16  weights expanded int8 -> 16 bit on the way (exact), kind::f16, acc * s[n] + b[n]
//          (nanovllm/quantization/csrc/int8_weight_only_gemm.cu:258-292, 397-412)
//
// What bounds these sizes is not a rate but a chain: start-up, first weights from HBM, first
// activations from L2, (expansion,) MMAs, epilogue, and then the next launch.  Hence:
//   * the NEXT kernel of the stream is resident while this one runs: on the same SMs (two CTAs of at
//     most 112 KB) or, with a deeper ring, on the SMs that a grid of 64-128 CTAs leaves free.
//     Weights are constants: a CTA sets up, asks for its first weight tiles and expands them
//     before it waits for the kernel that produces its activations (griddepcontrol.wait),
//     and lets its own successor start at once.
//   * one output tile per CTA, 128 tokens x 32 to 256 channels, and K split over a cluster
//     of up to 8 CTAs, so that narrow layers fill the GPU too.  Every CTA of a cluster owns
//     128 / S of the token rows (row % S): the others write their partial sums for these rows
//     into its shared memory, and it adds them in rank order, scales, rounds and stores.
//     (A single leader would need S - 1 whole tiles of shared memory and do all of the work.)
//   * the expansion of W8A16 is a chain of latencies (wait, load, permute, store, fence, arrive),
//     not of work: two to four groups of warps take the K blocks in turn, so that their chains overlap.
//
// What a chain of such launches takes per launch (64 tokens, us; before: the persistent kernels, whose
// start-up and first loads do not overlap anything): W8A8 4096 x 1024 3.8 (5.9), 1024 x 3072 4.2
// (10.7), 768 x 4096 4.3 (8.5); W8A16 6.0 (9.9), 5.9 (12.9), 6.0 (16.0).  Of the 3.8 us, 0.9 pass between the
// predecessor's end and the release of the wait, 0.4 until the activations land, 1.5 in the
// MMAs (some 45 cycles each at 32-64 channels, and 400 per chunk of waits and set-up) and 0.6 in the epilogue.
//
// Warp roles (352 threads): warp 0 TMA of the activations, warp 1 UMMA, warps 2-9 expansion, then
// epilogue, warp 10 TMA of the weights.
// Every mbarrier wait is bounded; the cluster barrier is reached by every thread on every path.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.h"
#include "ptx_sm100.cuh"
#include "w8a16_device.cuh"

namespace b200q {
namespace {

enum { MID_I8 = 0, MID_I8_RAW = 1, MID_F16 = 2 };

constexpr int kMidTok = 128;                     // UMMA M: token rows of a tile
constexpr int kMidXTile = kMidTok * 128;         // bytes the UMMA reads per K block of activations
constexpr int kMidThreads = 352;
constexpr int kMidMaxStages = 12;
constexpr int kMidConvWarps = 8;
constexpr int kMidCtrlBytes = 768;
constexpr int kMidSmemTwo = 112 * 1024;          // two CTAs per SM
constexpr int kMidSmemOne = 226 * 1024;          // one, with a deep ring

struct MidParams {
  int M, N;
  int bn;                  // channels per tile
  int x_rows;              // token rows loaded per K block: 128, or M rounded up to 8
  int tiles_m;
  int kc;                  // K blocks (128 bytes of a 16-bit or int8 operand row) per chunk
  int chunks, chunks_per_split;
  int chunks_3d;           // chunks below this one come through the 3-D maps: one TMA instruction
  int splits;              // cluster size
  int stages, stage_bytes; // ring of chunks: activations and the weights the UMMA reads
  int raw_bytes;           // W8A16: a second ring of as many chunks of int8 weights
  int tmem_cols;
  int is_bf16;
  const float* a_scales;   // per token (W8A8)
  const float* w_scales;   // per channel
  const void* bias;        // per channel or nullptr
  void* out;
  int* status;
};

// Expansion warps that share a K block: groups of two where the ring has a stage for each group.
__device__ __forceinline__ int conv_warps_per_block(int stages) {
  return stages >= 4 ? 2 : stages >= 2 ? 4 : 8;
}

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c,
                                              uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Eight sums of one token row -> eight outputs, one 16-byte store (two for raw int32).
template <int KIND, typename T>
__device__ __forceinline__ void store8(const MidParams& p, const uint32_t (&w)[8], float a_s,
                                       const float* s_ws, const T* bias, int row, int col) {
  const size_t at = static_cast<size_t>(row) * p.N + col;
  if (KIND == MID_I8_RAW) {
    uint4* dst = reinterpret_cast<uint4*>(static_cast<int32_t*>(p.out) + at);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
    return;
  }
  uint32_t packed[4];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[h] = KIND == MID_F16 ? __uint_as_float(w[j + h])
                             : __fmul_rn(static_cast<float>(static_cast<int>(w[j + h])), a_s);
      v[h] = __fmul_rn(v[h], s_ws[j + h]);
      if (bias != nullptr) v[h] = __fadd_rn(v[h], to_float<T>(bias[col + j + h]));
    }
    packed[j / 2] = pack2_rn<T>(make_float2(v[0], v[1]));
  }
  *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + at) =
      make_uint4(packed[0], packed[1], packed[2], packed[3]);
}

template <int KIND, typename T>
__global__ void __launch_bounds__(kMidThreads, 2)
umma_mid_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                const __grid_constant__ CUtensorMap tmap_x3, const __grid_constant__ CUtensorMap tmap_w3,
                const MidParams p) {
  constexpr bool kExpand = KIND == MID_F16;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t raw_base = static_cast<uint32_t>(p.stages * p.stage_bytes);
  uint8_t* red = smem + raw_base + p.stages * p.raw_bytes;     // [S][rows_own][bn] 32-bit sums (S > 1)
  const int rows_own = (min(kMidTok, p.x_rows) + p.splits - 1) / p.splits;   // token rows a CTA owns
  const int x_blk = p.x_rows * 128;                            // bytes of one K block of activations
  float* s_ws = reinterpret_cast<float*>(red + (p.splits > 1 ? p.splits * rows_own * p.bn * 4 : 0));
  float* s_as = s_ws + p.bn;                                   // scales of the 128 token rows
  uint8_t* ctrl = reinterpret_cast<uint8_t*>(s_as + kMidTok);
  uint64_t* xfull = reinterpret_cast<uint64_t*>(ctrl);         // activations of a stage have landed
  uint64_t* wfull = xfull + kMidMaxStages;                     // weights of a stage have landed
  uint64_t* cfull = wfull + kMidMaxStages;                     // ... and are expanded (W8A16)
  uint64_t* empty = cfull + kMidMaxStages;                     // the MMAs that read a stage are done
  uint64_t* rempty = empty + kMidMaxStages;                    // int8 tile read (W8A16)
  uint64_t* tfull = rempty + kMidMaxStages;                    // accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(p.splits > 1 ? ptx::cluster_ctarank() : 0);
  const int tile = static_cast<int>(blockIdx.x) / p.splits;
  const int tile_m = tile % p.tiles_m, tile_n = tile / p.tiles_m;  // neighbours share the weights
  const int c0 = rank * p.chunks_per_split;
  const int n_ch = min(p.chunks, c0 + p.chunks_per_split) - c0;    // >= 1 by construction
  const uint32_t smem_base = ptx::smem_u32(smem);
  const bool aligned = (smem_base & 1023u) == 0u;
  const int w_blk = p.bn * 128;                                // one K block of the operand the MMA reads
  const uint32_t w_off = static_cast<uint32_t>(p.kc * x_blk);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(ptx::smem_u32(xfull + s), 1);
      ptx::mbar_init(ptx::smem_u32(wfull + s), 1);
      ptx::mbar_init(ptx::smem_u32(cfull + s), conv_warps_per_block(p.stages));
      ptx::mbar_init(ptx::smem_u32(empty + s), 1);
      ptx::mbar_init(ptx::smem_u32(rempty + s), conv_warps_per_block(p.stages));
    }
    ptx::mbar_init(ptx::smem_u32(tfull), 1);
    *abort_flag = aligned ? 0 : 2;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (p.splits > 1) cluster_arrive();   // "this CTA runs": awaited before the first remote store
  ptx::grid_launch_dependents();        // the successor does not touch our results before it waits
  const bool run = aligned;             // a misaligned shared window (never seen) skips all work

  if (warp == 0 || warp == kMidThreads / 32 - 1) {
    if (run) {
      // -------------------------------------------------------------- TMA producers
      // One warp per operand: the weights run ahead as far as their ring allows, first of all
      // ahead of the kernel that produces the activations.
      const bool weights = warp != 0;
      constexpr int kWK = kExpand ? kBlockK : 128;             // bytes of a weight row per block
      const CUtensorMap* map = weights ? &tmap_w : &tmap_x;      // a block at a time: the end of K
      const CUtensorMap* map3 = weights ? &tmap_w3 : &tmap_x3;   // whole chunks of whole blocks
      const int row0 = weights ? tile_n * p.bn : tile_m * kMidTok;
      const int k_step = weights ? kWK : 128;                  // bytes of a row per block
      const int blk = weights ? p.bn * kWK : x_blk;            // bytes of a block's tile
      const uint32_t dst0 = smem_base + (weights ? (kExpand ? raw_base : w_off) : 0u);
      const uint32_t dst_step = static_cast<uint32_t>(weights && kExpand ? p.raw_bytes : p.stage_bytes);
      uint64_t* full = weights ? wfull : xfull;
      uint64_t* free_bar = weights && kExpand ? rempty : empty;
      if (weights) {
        if (ptx::elect_one())
          for (int i = p.stages; i < n_ch && i < p.stages + 8 && c0 + i < p.chunks_3d; ++i)
            ptx::tma_prefetch_l2_3d(map3, 0, row0, (c0 + i) * p.kc);
      } else {
        ptx::grid_dependency_wait();
      }
      int stage = 0, issued = 0;
      uint32_t phase = 1;                                      // the first round waits for nobody
      for (; issued < n_ch; ++issued) {
        if (issued >= p.stages && !ptx::mbar_wait(ptx::smem_u32(free_bar + stage), phase, abort_flag)) break;
        if (ptx::elect_one()) {
          const uint32_t bar = ptx::smem_u32(full + stage), dst = dst0 + stage * dst_step;
          const int c = (c0 + issued) * p.kc;
          ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(p.kc * blk));
          if (c0 + issued < p.chunks_3d) {
            ptx::tma_load_3d(dst, map3, bar, 0, row0, c);
          } else {
            for (int b = 0; b < p.kc; ++b) ptx::tma_load_2d(dst + b * blk, map, bar, (c + b) * k_step, row0);
          }
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (*abort_flag != 0) {
        // a wait ran out: give the copies in flight a bounded time to land before the CTA ends
        for (int j = max(0, issued - p.stages); j < issued; ++j) {
          const uint32_t parity = static_cast<uint32_t>((j / p.stages) & 1);
          for (int tries = 0;
               tries < (1 << 16) && !ptx::mbar_try_wait(ptx::smem_u32(full + j % p.stages), parity); ++tries) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (run) {
      // ----------------------------------------------------------------- UMMA issuer
      // An iteration costs some 400 cycles of waits, fences and descriptor set-up whatever it issues,
      // more than the MMAs of one K block take: hence chunks of several blocks.
      const uint32_t idesc = kExpand
                                 ? ptx::umma_idesc(1u, p.is_bf16 ? 1u : 0u, kMidTok, static_cast<uint32_t>(p.bn))
                                 : ptx::umma_idesc(2u, 1u, kMidTok, static_cast<uint32_t>(p.bn));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < n_ch; ++i) {
        uint64_t* wready = kExpand ? cfull : wfull;
        if (!ptx::mbar_wait(ptx::smem_u32(wready + stage), phase, abort_flag) ||
            !ptx::mbar_wait(ptx::smem_u32(xfull + stage), phase, abort_flag)) {
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          uint64_t a_desc = ptx::umma_desc_k_sw128(smem_base + stage * p.stage_bytes);
          uint64_t b_desc = ptx::umma_desc_k_sw128(smem_base + stage * p.stage_bytes + w_off);
          for (int b = 0; b < p.kc; ++b) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {   // 32 bytes of K per instruction
              const uint32_t acc = (i > 0 || b > 0 || k > 0) ? 1u : 0u;
              if (kExpand) ptx::umma_f16_ss(tmem_base, a_desc + 2u * k, b_desc + 2u * k, idesc, acc);
              else ptx::umma_i8_ss(tmem_base, a_desc + 2u * k, b_desc + 2u * k, idesc, acc);
            }
            a_desc += static_cast<uint32_t>(x_blk >> 4);
            b_desc += static_cast<uint32_t>(w_blk >> 4);
          }
          ptx::umma_commit(ptx::smem_u32(empty + stage));
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok && ptx::elect_one()) ptx::umma_commit(ptx::smem_u32(tfull));
    }
  } else {
    const int cw = warp - 2, tid = threadIdx.x - 64;
    // channel scales: constants, fetched ahead of the wait
    if (KIND != MID_I8_RAW && tid < p.bn) {
      const int col = tile_n * p.bn + tid;
      s_ws[tid] = col < p.N ? __ldg(p.w_scales + col) : 0.f;
    }
    if (kExpand && run) {
      // -------------------------------------------------------------- expansion
      // A stage always belongs to the same group of warps: a group that has not seen the previous
      // use of a stage complete could not tell its barrier's phases apart.
      const int wpb = conv_warps_per_block(p.stages), groups = kMidConvWarps / wpb;
      const int group = cw / wpb, t = (cw - group * wpb) * 32 + lane;
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < n_ch; ++i, stage = stage + 1 == p.stages ? 0 : stage + 1) {
        if (i > 0 && stage == 0) phase ^= 1u;
        if (stage % groups != group) continue;
        if (!ptx::mbar_wait(ptx::smem_u32(wfull + stage), phase, abort_flag)) break;
        if (i >= p.stages && !ptx::mbar_wait(ptx::smem_u32(empty + stage), phase ^ 1u, abort_flag)) break;
        const uint8_t* raw = smem + raw_base + stage * p.raw_bytes;
        uint8_t* dst = smem + stage * p.stage_bytes + w_off;
#pragma unroll 2
        for (int u = t; u < p.kc * p.bn * 4; u += wpb * 32)    // blocks follow one another
          expand_quarter_row<T>(raw, dst, u >> 2, u & 3);
        ptx::fence_proxy_async_smem();   // generic-proxy writes -> visible to the UMMA reads
        __syncwarp();
        if (lane == 0) {
          ptx::mbar_arrive(ptx::smem_u32(cfull + stage));
          ptx::mbar_arrive(ptx::smem_u32(rempty + stage));
        }
      }
    }
    __syncwarp();
    ptx::grid_dependency_wait();         // a_scales come from the previous kernel, y may be in use by it
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                       // token row of the tile = TMEM lane
    const int grow = tile_m * kMidTok + row;
    const bool live = grow < p.M;
    float a_s = 1.f;
    if (KIND == MID_I8) {
      a_s = live ? p.a_scales[grow] : 0.f;   // while the main loop runs (not __ldg: it must stay behind the wait)
      if (cw < 4) s_as[row] = a_s;
    }
    const T* bias = reinterpret_cast<const T*>(p.bias);
    // ------------------------------------------------ partial sums -> the rows' owners
    if (p.splits > 1) cluster_wait();    // every CTA of the cluster runs: its memory may be written
    else ptx::named_bar_sync(1, 256);             // s_ws complete
    bool done = run && ptx::mbar_wait(ptx::smem_u32(tfull), 0u, abort_flag);
    done = __all_sync(0xFFFFFFFFu, done);
    if (done) {
      ptx::tc_fence_after_sync();
      const int shift = __ffs(p.splits) - 1;
      const int owner = row & (p.splits - 1), rl = row >> shift;
      const uint32_t mine = ptx::smem_u32(red) + static_cast<uint32_t>((rank * rows_own + rl) * p.bn) * 4u;
      const uint32_t dst = p.splits > 1 ? ptx::map_to_cta(mine, static_cast<uint32_t>(owner)) : mine;
      for (int c = cw >> 2; c < p.bn / 32; c += 2) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c * 32, v);
        ptx::tmem_ld_wait();
        if (!live) continue;
        if (p.splits > 1) {
#pragma unroll
          for (int j = 0; j < 8; ++j)    // 16-byte chunk c * 8 + j of the row, swizzled by the row
            st_cluster_v4(dst + static_cast<uint32_t>((c * 8 + (j ^ (rl & 7))) << 4), v[4 * j],
                          v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          continue;
        }
        // no split: straight from the registers, 8 channels (16 bytes) at a time
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          const int col = tile_n * p.bn + c * 32 + j;
          if (col >= p.N) break;         // N % 8 == 0
          const uint32_t w[8] = {v[j], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7]};
          store8<KIND, T>(p, w, a_s, s_ws + c * 32 + j, bias, grow, col);
        }
      }
    }
  }
  if (p.splits > 1 && (warp < 2 || warp == kMidThreads / 32 - 1)) {
    __syncwarp();
    cluster_wait();      // the arrival at the start
  }
  __syncwarp();
  ptx::tc_fence_before_sync();
  if (p.splits > 1) {
    cluster_arrive();    // release: this CTA's stores; after the wait nothing is written remotely
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }

  // ------------------------------------------------------ own rows: add, scale, round, store
  if (p.splits > 1) {
    const int gshift = __ffs(p.bn) - 4;      // bn / 8 groups of 8 channels per row: one 16-byte store
    const T* bias = reinterpret_cast<const T*>(p.bias);
    for (int u = threadIdx.x; u < (rows_own << gshift); u += kMidThreads) {
      const int rl = u >> gshift, cg = u - (rl << gshift);
      const int row = rl * p.splits + rank;
      const int grow = tile_m * kMidTok + row, col = tile_n * p.bn + cg * 8;
      if (grow >= p.M || col >= p.N) continue;   // N % 8 == 0
      const int j0 = ((2 * cg) & 7) ^ (rl & 7), j1 = ((2 * cg + 1) & 7) ^ (rl & 7);
      const int base = (2 * cg) & ~7;
      uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      for (int s = 0; s < p.splits; ++s) {       // rank order: results do not depend on the run
        const uint8_t* src = red + static_cast<size_t>((s * rows_own + rl) * p.bn) * 4;
        const uint4 a = *reinterpret_cast<const uint4*>(src + ((base + j0) << 4));
        const uint4 b = *reinterpret_cast<const uint4*>(src + ((base + j1) << 4));
        const uint32_t in[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          w[j] = s == 0 ? in[j]
                 : kExpand ? __float_as_uint(__fadd_rn(__uint_as_float(w[j]), __uint_as_float(in[j])))
                           : w[j] + in[j];
      }
      store8<KIND, T>(p, w, KIND == MID_I8 ? s_as[row] : 1.f, s_ws + cg * 8, bias, grow, col);
    }
  }
  if (threadIdx.x == 0 && *abort_flag != 0)
    atomicCAS(p.status, 0, 0xA00 | (*abort_flag << 4) | (static_cast<int>(blockIdx.x) << 12));
}

}  // namespace

// ------------------------------------------------------------------------------ host
namespace {

struct MidPlan {
  int bn, x_rows, splits, kc, chunks, chunks_per_split, tiles_m, tiles_n, stages, stage_bytes, raw_bytes;
  size_t smem;
};

bool mid_plan_for(int M, int N, int k_blocks, bool a16, int bn, int splits, int kc,
                  int smem_cap, MidPlan* pl) {
  pl->bn = bn;
  pl->kc = kc;
  pl->splits = splits;
  pl->chunks = (k_blocks + kc - 1) / kc;
  pl->chunks_per_split = (pl->chunks + splits - 1) / splits;
  if (pl->chunks_per_split * (splits - 1) >= pl->chunks) return false;   // a CTA without work
  pl->tiles_m = (M + kMidTok - 1) / kMidTok;
  pl->tiles_n = (N + bn - 1) / bn;
  pl->x_rows = M >= kMidTok ? kMidTok : (M + 7) / 8 * 8;
  pl->stage_bytes = kc * (pl->x_rows * 128 + bn * 128);
  pl->raw_bytes = a16 ? kc * bn * kRow8 : 0;
  const int ring_bytes = pl->stage_bytes + pl->raw_bytes;
  const int rows_own = (pl->x_rows + splits - 1) / splits;
  int fixed = (splits > 1 ? splits * rows_own * bn * 4 : 0) + bn * 4 + kMidTok * 4 + kMidCtrlBytes;
  // the UMMA reads 128 rows of activations whatever x_rows is: the last block's excess must still
  // lie inside the CTA's shared memory (what it holds only reaches accumulator rows nobody reads)
  fixed = std::max(fixed, (kc - 1) * pl->x_rows * 128 + kMidXTile - pl->stage_bytes);
  pl->stages = std::min({(smem_cap - fixed) / ring_bytes, kMidMaxStages, pl->chunks_per_split});
  if (pl->stages < 1 || (pl->stages < 2 && pl->chunks_per_split > 1)) return false;
  pl->smem = static_cast<size_t>(pl->stages) * ring_bytes + fixed;
  return true;
}

// Predicted time of one call in a stream of such calls, in microseconds.  The form follows what the
// kernel does (the three pipes overlap, hence the root of cubes); the coefficients are fitted to
// 5,600 measured configurations (13 shapes from 2 to 100 MB of weights, 24 to 512 tokens, both
// schemes): the configuration with the smallest prediction is on average 4 % slower than the
// best measured one.
double mid_cost(const MidPlan& pl, int M, double matrix_bytes, bool a16) {
  const double clk = 1850.0;   // cycles per microsecond
  const int ctas = pl.tiles_m * pl.tiles_n * pl.splits;
  const int per_sm = pl.smem <= kMidSmemTwo ? 2 : 1;
  // clusters of 4 and 8 do not fill every SM (a cluster lives inside one group of SMs)
  const int sms = sm_count() - (pl.splits == 8 ? 28 : pl.splits == 4 ? 12 : 0);
  const double passes = (ctas + sms - 1) / sms, waves = (ctas + sms * per_sm - 1) / (sms * per_sm);
  const double kb = pl.chunks_per_split * pl.kc;
  const double per_mma = pl.bn == 256 ? 130 : pl.bn == 128 ? 68 : pl.bn == 64 ? 51 : 43;   // cycles
  const double mma = 0.68 * kb * 4 * per_mma * passes;
  const double expand = a16 ? kb * pl.bn * kRow8 / 17.6 * passes : 0.0;
  const double weights = kb * pl.bn * (a16 ? 64 : 128) / 134.0 * passes;
  const double hbm = matrix_bytes / sm_count() / 26.6;
  double us = 2.34 + std::cbrt(mma * mma * mma + expand * expand * expand + weights * weights * weights +
                               hbm * hbm * hbm) / clk;
  // a ring shorter than the K loop goes round at the latency of a load
  us += 0.534 * waves * std::max(0, pl.chunks_per_split - pl.stages) / pl.stages;
  us += 0.135 * waves * pl.chunks_per_split;
  const double rows = std::min(M, kMidTok);
  if (pl.splits > 1) us += 0.416 + 0.04 * rows * pl.bn * 4 * passes / clk;
  us += 0.061 * rows * pl.bn * 2 * passes / clk;
  // start-up (1 us, and the first weights from HBM) hides under the previous kernel only as far as
  // both fit the GPU
  const double slots = static_cast<double>(sm_count()) * per_sm;
  us += 1.345 * std::min(1.0, std::max(0.0, (2.0 * ctas - slots) / slots)) + 1.676 * (waves - 1);
  return us;
}

bool search_plan(int M, int N, int K, bool a16, MidPlan* best) {
  const int k_blocks = a16 ? (K + kBlockK - 1) / kBlockK : (K + 127) / 128;
  const int want_bn = debug_knob(B200Q_KNOB_BN, 0), want_s = debug_knob(B200Q_KNOB_CLUSTER, 0);
  double best_cost = 1e30;
  for (int bn : {128, 64, 32, 256}) {
    if (want_bn != 0 && bn != want_bn) continue;
    for (int s : {1, 2, 4, 8}) {
      if (want_s != 0 && s != want_s) continue;
      for (int kc : {4, 2, 1}) {
        for (int cap : {kMidSmemOne, kMidSmemTwo}) {
          MidPlan pl;
          if (!mid_plan_for(M, N, k_blocks, a16, bn, s, kc, cap, &pl)) continue;
          const double cost = mid_cost(pl, M, static_cast<double>(N) * K, a16);
          if (cost < best_cost) {
            best_cost = cost;
            *best = pl;
          }
        }
      }
    }
  }
  return best_cost < 1e30;
}

// The search costs some 10 us of host time, more than the launch: its results are kept per thread, in a
// table of fixed size where a new shape replaces the one in its slot.
bool mid_plan(int M, int N, int K, bool a16, MidPlan* best) {
  if (debug_knob(B200Q_KNOB_BN, 0) != 0 || debug_knob(B200Q_KNOB_CLUSTER, 0) != 0)
    return search_plan(M, N, K, a16, best);
  struct Entry {
    int M, N, K, kind;   // kind: 0 = empty, 1 = W8A8, 2 = W8A16
    MidPlan plan;
  };
  constexpr unsigned kSlots = 1024;
  thread_local Entry table[kSlots];
  const unsigned h = static_cast<unsigned>(M) * 0x9E3779B1u ^ static_cast<unsigned>(N) * 0x85EBCA77u ^
                     static_cast<unsigned>(K) * 0xC2B2AE3Du;
  Entry& e = table[(h >> 16) % kSlots];
  const int kind = a16 ? 2 : 1;
  if (e.kind != kind || e.M != M || e.N != N || e.K != K) {
    Entry fresh{M, N, K, kind, {}};
    if (!search_plan(M, N, K, a16, &fresh.plan)) return false;
    e = fresh;
  }
  *best = e.plan;
  return true;
}

template <auto kernel>
cudaError_t launch_mid_kernel(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tx3,
                              const CUtensorMap& tw3, const MidParams& mp,
                              const MidPlan& pl, cudaStream_t stream) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmemOne);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_set[dev] = true;
  }
  return launch_clustered(pl.splits, true, kernel, dim3(pl.tiles_m * pl.tiles_n * pl.splits),
                          dim3(kMidThreads), pl.smem, stream, tx, tw, tx3, tw3, mp);
}

}  // namespace

// Up to 148 tiles of 128 x 128 outputs (one wave), where this kernel beats the persistent ones by
// 1.1 to 2.7 times at every measured shape (4096 x 1024 at 256 tokens: W8A8 4.8 against 6.2 us,
// W8A16 7.8 against 10.2; 1024 x 3072 at 64 tokens: 4.1 against 8.0 and 5.2 against 12.8; 768 x 4096 at
// 64: 4.2 against 8.5 and 5.9 against 16.0).  Beyond one wave their overlapped epilogue and larger tiles win,
// except for few tokens, where a tile is short (24576 x 4096: W8A8 at 128 tokens 25.0 against 25.4 us,
// W8A16 at 24 tokens 45.1 against 49.6, at 64 already 52.5 against 51.1).
bool umma_mid_applicable(int M, int N, int K, bool a16) {
  if (debug_knob(B200Q_KNOB_NO_MID, 0) != 0) return false;
  if ((K % 16) != 0 || (N % 8) != 0 || M < 1) return false;
  const long long tiles = static_cast<long long>((M + kMidTok - 1) / kMidTok) * ((N + 127) / 128);
  if (tiles > sm_count() && M > (a16 ? 32 : 128)) return false;
  if (debug_knob(B200Q_KNOB_BN, 0) == 0 && debug_knob(B200Q_KNOB_CLUSTER, 0) == 0) return true;
  MidPlan pl;   // a forced tile or cluster may not fit
  return mid_plan(M, N, K, a16, &pl);
}

int launch_umma_mid(const GemmArgs& a, bool a16) {
  MidPlan pl;
  if (!mid_plan(a.M, a.N, a.K, a16, &pl)) return B200Q_ERR_UNSUPPORTED_SHAPE;
  CUtensorMap tx, tw;
  const uint64_t x_row = static_cast<uint64_t>(a.K) * (a16 ? 2 : 1);
  const uint32_t w_box = a16 ? kRow8 : 128;
  if (!make_tensor_map(a.x, a.M, x_row, static_cast<uint32_t>(pl.x_rows), 128, &tx) ||
      !get_tensor_map(a.w, a.N, a.K, static_cast<uint32_t>(pl.bn), w_box, &tw))
    return B200Q_ERR_LAUNCH;
  // K a multiple of a block: everything comes through the 3-D maps (blocks beyond K read as zeros);
  // otherwise the chunk with the partial block, and what follows it, goes block by block
  const int whole = a.K / (a16 ? kBlockK : 128);
  const bool even = a.K % (a16 ? kBlockK : 128) == 0;
  const int chunks_3d = even ? pl.chunks : whole / pl.kc;
  CUtensorMap tx3 = tx, tw3 = tw;
  if (chunks_3d > 0 &&
      (!make_tensor_map(a.x, a.M, x_row, static_cast<uint32_t>(pl.x_rows), 128, &tx3, pl.kc) ||
       !get_tensor_map(a.w, a.N, a.K, static_cast<uint32_t>(pl.bn), w_box, &tw3, pl.kc)))
    return B200Q_ERR_LAUNCH;
  MidParams mp{};
  mp.M = a.M;
  mp.N = a.N;
  mp.bn = pl.bn;
  mp.x_rows = pl.x_rows;
  mp.tiles_m = pl.tiles_m;
  mp.kc = pl.kc;
  mp.chunks = pl.chunks;
  mp.chunks_per_split = pl.chunks_per_split;
  mp.chunks_3d = chunks_3d;
  mp.splits = pl.splits;
  mp.stages = pl.stages;
  mp.stage_bytes = pl.stage_bytes;
  mp.raw_bytes = pl.raw_bytes;
  mp.tmem_cols = pl.bn;
  mp.is_bf16 = a.dtype == B200Q_DTYPE_BF16 ? 1 : 0;
  mp.a_scales = a.a_scales;
  mp.w_scales = a.w_scales;
  mp.bias = a.bias;
  mp.out = a.acc_out != nullptr ? static_cast<void*>(a.acc_out) : a.y;
  mp.status = a.status;
  cudaError_t e;
  if (a16)
    e = mp.is_bf16 ? launch_mid_kernel<umma_mid_kernel<MID_F16, __nv_bfloat16>>(tx, tw, tx3, tw3, mp, pl, a.stream)
                   : launch_mid_kernel<umma_mid_kernel<MID_F16, __half>>(tx, tw, tx3, tw3, mp, pl, a.stream);
  else if (a.acc_out != nullptr)
    e = launch_mid_kernel<umma_mid_kernel<MID_I8_RAW, __nv_bfloat16>>(tx, tw, tx3, tw3, mp, pl, a.stream);
  else
    e = mp.is_bf16 ? launch_mid_kernel<umma_mid_kernel<MID_I8, __nv_bfloat16>>(tx, tw, tx3, tw3, mp, pl, a.stream)
                   : launch_mid_kernel<umma_mid_kernel<MID_I8, __half>>(tx, tw, tx3, tw3, mp, pl, a.stream);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return B200Q_ERR_LAUNCH;
  }
  count_launch();
  return B200Q_OK;
}

}  // namespace b200q
