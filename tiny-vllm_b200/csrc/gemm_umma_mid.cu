// W8A8 at tens to hundreds of tokens on tcgen05: int8 x int8 -> int32 (kind::i8), then
// (float(acc) * a_s[m]) * w_s[n] + b[n]  (nanovllm/quantization/csrc/w8a8_gemm.cu:165-183, 387-390).
//
// What bounds these sizes is not a rate but a chain: start-up, first weights from HBM, first
// activations from L2, MMAs, epilogue, and then the next launch.  Hence:
//   * the NEXT kernel of the stream is resident while this one runs: on the same SMs (two CTAs of at
//     most 112 KB) or, with a deeper ring, on the SMs that a grid of 64-128 CTAs leaves free.
//     Weights are constants: a CTA sets up and asks for its first weight tiles before it waits
//     for the kernel that produces its activations (griddepcontrol.wait), and lets its own successor start at once.
//   * one output tile per CTA, 128 tokens x 32 to 256 channels, and K split over a cluster
//     of up to 8 CTAs, so that narrow layers fill the GPU too.  Every CTA of a cluster owns
//     128 / S of the token rows (row % S): the others write their partial sums for these rows
//     into its shared memory, and it adds them in rank order, scales, rounds and stores.
//     (A single leader would need S - 1 whole tiles of shared memory and do all of the work.)
//
// What a chain of such launches takes per launch (64 tokens, us; before: the persistent kernels, whose
// start-up and first loads do not overlap anything): W8A8 4096 x 1024 3.8 (5.9), 1024 x 3072 4.2
// (10.7), 768 x 4096 4.3 (8.5).  Of the 3.8 us, 0.9 pass between the
// predecessor's end and the release of the wait, 0.4 until the activations land, 1.5 in the
// MMAs (some 45 cycles each at 32-64 channels, and 400 per chunk of waits and set-up) and 0.6 in the epilogue.
//
// Warp roles (352 threads): warp 0 TMA of the activations, warp 1 UMMA, warps 2-9 epilogue,
// warp 10 TMA of the weights.
// Every mbarrier wait is bounded; the cluster barrier is reached by every thread on every path, and no CTA of a
// cluster waits for tensor memory (the residency rule of umma_mid_common.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.h"
#include "ptx_sm100.cuh"
#include "umma_mid_common.cuh"
#include "w8a16_device.cuh"

namespace b200q {
namespace {

constexpr int kMidTok = 128;                     // UMMA M: token rows of a tile
constexpr int kMidXTile = kMidTok * 128;         // bytes the UMMA reads per K block of activations
// One CTA per SM, and room beside it for those of the quantiser that runs between two such kernels (1 KB each): with all
// of the shared memory taken, a CTA waits for the quantiser to leave its SM.  Plans that use it have fewer CTAs with wider
// tiles, too, so the limit pays where no quantiser runs (layers of the 0.6B model at 129 to 512 tokens, 226 / 218 KB:
// 1.018-1.025 with a quantiser, 1.005-1.047 on codes).
constexpr int kMidSmemQuant = 218 * 1024;
// But long rows of more than one token tile go round a ring of two or three chunks many times, and a chunk more is worth
// more than the early start: at 129 to 256 tokens layers with down projections of K = 12288, 9728, 9472 and 6144 take
// 0.960-0.985 of their time with 226 KB (0.936-0.975 on codes).  Up to one token tile, or K = 4096, it is either way.
bool mid_wants_deep_ring(int M, int K) { return M > kMidTok && K > 4096; }

struct MidParams {
  int M, N;
  int bn;                  // channels per tile
  int x_rows;              // token rows loaded per K block: 128, or M rounded up to 8
  int tiles_m;
  int kc;                  // K blocks of 128 per chunk
  int chunks, chunks_per_split;
  int chunks_3d;           // chunks below this one come through the 3-D maps: one TMA instruction
  int splits;              // cluster size
  int stages, stage_bytes; // ring of chunks: activations and weights
  int ring_bytes;          // the ring, or the output tile that lies over it at the end
  int out_pitch;           // bytes of a token's row of that tile, 0: not through shared memory
  int tmem_cols;
  const float* a_scales;   // per token
  const float* w_scales;   // per channel
  const void* bias;        // per channel or nullptr
  void* out;
  int* status;
};

// Eight sums of one token row -> eight outputs.  Packed products round each half like the scalar instruction; the sums
// with the bias are scalar, so that they are not contracted with them.
template <typename T>
__device__ __forceinline__ uint4 scale8(const uint32_t (&w)[8], float a_s, const float* s_ws, const T* bias, int col) {
  const float4 c0 = *reinterpret_cast<const float4*>(s_ws), c1 = *reinterpret_cast<const float4*>(s_ws + 4);
  const float2 c[4] = {{c0.x, c0.y}, {c0.z, c0.w}, {c1.x, c1.y}, {c1.z, c1.w}}, a2 = make_float2(a_s, a_s);
  float2 v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    v[j] = __fmul2_rn(__fmul2_rn(make_float2(static_cast<float>(static_cast<int>(w[2 * j])),
                                             static_cast<float>(static_cast<int>(w[2 * j + 1]))), a2), c[j]);
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = make_float2(__fadd_rn(v[j].x, to_float<T>(bias[col + 2 * j])), __fadd_rn(v[j].y, to_float<T>(bias[col + 2 * j + 1])));
  }
  return make_uint4(pack2_rn<T>(v[0]), pack2_rn<T>(v[1]), pack2_rn<T>(v[2]), pack2_rn<T>(v[3]));
}

// Eight raw sums of a row.
__device__ __forceinline__ void store8_raw(const MidParams& p, const uint32_t (&w)[8], int row, int col) {
  uint4* dst = reinterpret_cast<uint4*>(static_cast<int32_t*>(p.out) + static_cast<size_t>(row) * p.N + col);
  dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
  dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

template <bool RAW, typename T>
__global__ void __launch_bounds__(kMidThreads, 2)
w8a8_mid_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                const __grid_constant__ CUtensorMap tmap_x3, const __grid_constant__ CUtensorMap tmap_w3,
                const MidParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* red = smem + p.ring_bytes;                 // [S][rows_own][bn] 32-bit sums (S > 1)
  const int rows_own = (min(kMidTok, p.x_rows) + p.splits - 1) / p.splits;   // token rows a CTA owns
  const int x_blk = p.x_rows * 128;                            // bytes of one K block of activations
  float* s_ws = reinterpret_cast<float*>(red + (p.splits > 1 ? p.splits * rows_own * p.bn * 4 : 0));
  float* s_as = s_ws + p.bn;                                   // scales of the 128 token rows
  uint8_t* ctrl = reinterpret_cast<uint8_t*>(s_as + kMidTok);
  uint64_t* xfull = reinterpret_cast<uint64_t*>(ctrl);         // activations of a stage have landed
  uint64_t* wfull = xfull + kMidMaxStages;                     // weights of a stage have landed
  uint64_t* empty = wfull + kMidMaxStages;                     // the MMAs that read a stage are done
  uint64_t* tfull = empty + kMidMaxStages;                    // accumulator complete
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
      ptx::mbar_init(ptx::smem_u32(empty + s), 1);
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
      const bool weights = warp != 0;
      const MidStream s{weights ? &tmap_w : &tmap_x, weights ? &tmap_w3 : &tmap_x3,
                        weights ? tile_n * p.bn : tile_m * kMidTok, 128, weights ? w_blk : x_blk, p.kc,
                        smem_base + (weights ? w_off : 0u), static_cast<uint32_t>(p.stage_bytes), p.stages,
                        weights ? wfull : xfull, empty, c0, n_ch, p.chunks_3d};
      if (weights) {
        if (ptx::elect_one())
          for (int i = p.stages; i < n_ch && i < p.stages + 8 && c0 + i < p.chunks_3d; ++i)
            ptx::tma_prefetch_l2_3d(s.map3, 0, s.row0, (c0 + i) * p.kc);
      } else {
        ptx::grid_dependency_wait();
      }
      mid_produce(s, abort_flag);
    }
  } else if (warp == 1) {
    if (run) {
      // ----------------------------------------------------------------- UMMA issuer
      // An iteration costs some 400 cycles of waits, fences and descriptor set-up whatever it issues,
      // more than the MMAs of one K block take: hence chunks of several blocks.
      const uint32_t idesc = ptx::umma_idesc(2u, 1u, kMidTok, static_cast<uint32_t>(p.bn));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < n_ch; ++i) {
        if (!ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(wfull + stage), phase, abort_flag) &&
                           ptx::mbar_wait(ptx::smem_u32(xfull + stage), phase, abort_flag))) {
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
              ptx::umma_i8_ss(tmem_base, a_desc + 2u * k, b_desc + 2u * k, idesc, acc);
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
    if (!RAW && tid < p.bn) {
      const int col = tile_n * p.bn + tid;
      s_ws[tid] = col < p.N ? __ldg(p.w_scales + col) : 0.f;
    }
    ptx::grid_dependency_wait();         // a_scales come from the previous kernel, y may be in use by it
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                       // token row of the tile = TMEM lane
    const int grow = tile_m * kMidTok + row;
    const bool live = grow < p.M;
    float a_s = 1.f;
    if (!RAW) {
      a_s = live ? p.a_scales[grow] : 0.f;   // while the main loop runs (not __ldg: it must stay behind the wait)
      if (cw < 4) s_as[row] = a_s;
    }
    const T* bias = reinterpret_cast<const T*>(p.bias);
    // ------------------------------------------------ partial sums -> the rows' owners
    if (p.splits > 1) cluster_wait();    // every CTA of the cluster runs: its memory may be written
    else ptx::named_bar_sync(1, 256);             // s_ws complete
    const bool done = run && ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(tfull), 0u, abort_flag));
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
        // no split.  Wide tiles go through shared memory (over the ring, which is done with: the MMAs that read the
        // last of it have completed); of a narrow one, and of raw sums, a thread stores its pieces of a row itself
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          const int col = tile_n * p.bn + c * 32 + j;
          if (col >= p.N) break;         // N % 8 == 0
          const uint32_t w[8] = {v[j], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7]};
          if (RAW) {
            store8_raw(p, w, grow, col);
          } else {
            const uint4 o = scale8<T>(w, a_s, s_ws + c * 32 + j, bias, col);
            if (p.out_pitch > 0)
              *reinterpret_cast<uint4*>(smem + row * p.out_pitch + (c * 32 + j) * 2) = o;
            else
              *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + static_cast<size_t>(grow) * p.N + col) = o;
          }
        }
      }
    }
    if (!RAW && p.out_pitch > 0) {
      // out in whole rows, 16 bytes a thread
      ptx::named_bar_sync(1, 256);
      const int shift = __ffs(p.bn) - 4, pieces = 1 << shift;     // 16-byte pieces of a row
      const int sub = tid & (pieces - 1), n0 = tile_n * p.bn + sub * 8, step = 256 >> shift;
      const int rows = min(kMidTok, p.M - tile_m * kMidTok);
      if (done && n0 < p.N) {
        T* out = static_cast<T*>(p.out) + static_cast<size_t>(tile_m * kMidTok) * p.N + n0;
        for (int r0 = tid >> shift; r0 < rows; r0 += 4 * step) {
          uint4 v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (r0 + j * step < rows) v[j] = *reinterpret_cast<const uint4*>(smem + (r0 + j * step) * p.out_pitch + sub * 16);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (r0 + j * step < rows) *reinterpret_cast<uint4*>(out + static_cast<size_t>(r0 + j * step) * p.N) = v[j];
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
          w[j] += in[j];
      }
      if (RAW)
        store8_raw(p, w, grow, col);
      else
        *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + static_cast<size_t>(grow) * p.N + col) =
            scale8<T>(w, s_as[row], s_ws + cg * 8, bias, col);
    }
  }
  if (threadIdx.x == 0 && *abort_flag != 0)
    atomicCAS(p.status, 0, 0xA00 | (*abort_flag << 4) | (static_cast<int>(blockIdx.x) << 12));
}

}  // namespace

// ------------------------------------------------------------------------------ host
namespace {

struct MidPlan {
  int bn, x_rows, splits, kc, chunks, chunks_per_split, tiles_m, tiles_n, stages, stage_bytes, ring_bytes, out_pitch;
  size_t smem;
};

bool mid_plan_for(int M, int N, int k_blocks, int bn, int splits, int kc,
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
  const int rows_own = (pl->x_rows + splits - 1) / splits;
  int fixed = (splits > 1 ? splits * rows_own * bn * 4 : 0) + bn * 4 + kMidTok * 4 + kMidCtrlBytes;
  // the UMMA reads 128 rows of activations whatever x_rows is: the last block's excess must still
  // lie inside the CTA's shared memory (what it holds only reaches accumulator rows nobody reads)
  fixed = std::max(fixed, (kc - 1) * pl->x_rows * 128 + kMidXTile - pl->stage_bytes);
  pl->stages = std::min({(smem_cap - fixed) / pl->stage_bytes, kMidMaxStages, pl->chunks_per_split});
  if (pl->stages < 1 || (pl->stages < 2 && pl->chunks_per_split > 1)) return false;
  // A thread's pieces of a row fill whole lines where the tile is narrow, and few rows are soon stored (64 tokens, 4096 x
  // 1024 in tiles of 32 channels 3.7 us, 4.0 through shared memory); larger tiles are stored by rows (256 tokens, 6144 x
  // 1024 in tiles of 128 5.9 -> 5.4 us, 128 tokens, 24576 x 4096 25.2 -> 23.8, one eighth of the 8B model at 256 tokens, in tiles of
  // 64, 37.5 -> 36.8 a layer)
  const bool by_rows = splits == 1 && (bn >= 128 || (bn == 64 && 4 * M >= 3 * kMidTok));
  pl->out_pitch = by_rows ? bn * 2 + 16 : 0;   // + 16: rows on different banks
  pl->ring_bytes = std::max(pl->stages * pl->stage_bytes, pl->x_rows * pl->out_pitch);
  pl->smem = static_cast<size_t>(pl->ring_bytes) + fixed;
  if (splits > 1) pl->smem = std::max<size_t>(pl->smem, kClusterSmemMin);
  return pl->smem <= static_cast<size_t>(smem_cap);
}

// Predicted time of one call in a stream of such calls, in microseconds.  The form follows what the
// kernel does (MMAs, the issue loop's overhead per K block and the loads overlap, hence the root of cubes); the
// coefficients are fitted to 2,000 measured configurations (18 shapes from 2 to 100 MB of weights, 24 to 2000 tokens) so that
// the one with the smallest prediction is close to the best: on average 1.6 %, at worst 17 % slower than it (4.3
// and 34 % for a model that counted two CTAs of an SM as twice the work).
double mid_cost(const MidPlan& pl, int M) {
  const double clk = 1850.0;   // cycles per microsecond
  const int ctas = pl.tiles_m * pl.tiles_n * pl.splits;
  const int per_sm = pl.smem <= kMidSmemTwo ? 2 : 1;
  // clusters of 4 and 8 do not fill every SM (a cluster lives inside one group of SMs)
  const int sms = sm_count() - (pl.splits == 8 ? 28 : pl.splits == 4 ? 12 : 0);
  const int passes = (ctas + sms - 1) / sms, waves = (ctas + sms * per_sm - 1) / (sms * per_sm);
  // two CTAs on an SM share its load bandwidth, but wait on different things most of the time
  const double work = per_sm == 1 ? passes : waves;
  const double kb = pl.chunks_per_split * pl.kc;
  const double mma = kb * 4 * 0.637 * pl.bn * work, issue = 211.0 * kb * work;
  const double load = kb * 128 * (pl.x_rows + pl.bn) * passes / 296.0;
  double us = 1.93 + std::cbrt(mma * mma * mma + issue * issue * issue + load * load * load) / clk;
  // a ring shorter than the K loop goes round at the latency of a load
  us += 1.08 * waves * std::max(0, pl.chunks_per_split - pl.stages) / pl.stages;
  us += 0.0757 * waves * pl.chunks_per_split;
  const double values = std::min(M, kMidTok) * pl.bn / 64.0;
  us += pl.splits > 1 ? 0.00746 * values * passes + 0.746 * std::log2(pl.splits) : 0.00185 * values * work;
  // start-up (1 us, and the first weights from HBM) hides under the previous kernel only as far as
  // both fit the GPU
  const double slots = static_cast<double>(sm_count()) * per_sm;
  us += 1.4 * std::min(1.0, std::max(0.0, (2.0 * ctas - slots) / slots));
  us += (per_sm == 1 ? 2.6 : 2.15) * (waves - 1);
  // Clusters that need several SMs at once, two CTAs on each, start late: behind a quantiser that still has CTAs of its own
  // (layers of hidden 4096 and 2560 at 20 and 32 tokens without / with the factor 1.03-1.05) and behind another GEMM (1.02-1.045
  // on codes).  Against it: layers of hidden 1024 on codes at 20 and 32 tokens, 0.987-0.992; elsewhere no difference.
  return pl.splits > 1 && ctas > sm_count() ? 1.15 * us : us;
}

bool search_plan(int M, int N, int K, MidPlan* best) {
  const int k_blocks = (K + 127) / 128;
  const int want_bn = debug_knob(B200Q_KNOB_BN, 0), want_s = debug_knob(B200Q_KNOB_CLUSTER, 0);
  double best_cost = 1e30;
  for (int bn : {128, 64, 32, 256}) {
    if (want_bn != 0 && bn != want_bn) continue;
    for (int s : {1, 2, 4, 8}) {
      if (want_s != 0 && s != want_s) continue;
      for (int kc : {4, 2, 1}) {
        for (int cap : {mid_wants_deep_ring(M, K) ? kMidSmemOne : kMidSmemQuant, kMidSmemTwo}) {
          MidPlan pl;
          if (!mid_plan_for(M, N, k_blocks, bn, s, kc, cap, &pl)) continue;
          const double cost = mid_cost(pl, M);
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

}  // namespace

// Up to 148 tiles of 128 x 128 outputs (one wave), where this kernel beats the persistent ones by
// 1.1 to 2.7 times at every measured shape (4096 x 1024 at 256 tokens 4.8 against 6.2 us; 1024 x 3072 at 64
// 4.1 against 8.0; 768 x 4096 at 64 4.2 against 8.5).  Beyond one wave their overlapped epilogue and
// larger tiles win, except for few tokens, where a tile is short (24576 x 4096 at 128 tokens 25.0 against 25.4 us).
bool umma_mid_applicable(int M, int N, int K) {
  if (debug_knob(B200Q_KNOB_NO_MID, 0) != 0) return false;
  if ((K % 16) != 0 || (N % 8) != 0 || M < 1) return false;
  const long long tiles = static_cast<long long>((M + kMidTok - 1) / kMidTok) * ((N + 127) / 128);
  if (tiles > sm_count() && M > 128) return false;
  if (debug_knob(B200Q_KNOB_BN, 0) == 0 && debug_knob(B200Q_KNOB_CLUSTER, 0) == 0) return true;
  MidPlan pl;   // a forced tile or cluster may not fit
  return mid_plan<MidPlan, search_plan>(M, N, K, &pl);
}

bool umma_mid_shape(int M, int N, int K, MidShape* s) {
  MidPlan pl;
  if (!umma_mid_applicable(M, N, K) || !mid_plan<MidPlan, search_plan>(M, N, K, &pl)) return false;
  *s = MidShape{kMidTok, pl.bn, pl.splits, pl.bn, static_cast<int>(pl.smem), pl.tiles_m * pl.tiles_n * pl.splits};
  return true;
}

int launch_umma_mid(const GemmArgs& a) {
  MidPlan pl;
  if (!mid_plan<MidPlan, search_plan>(a.M, a.N, a.K, &pl)) return B200Q_ERR_UNSUPPORTED_SHAPE;
  MidMaps maps;
  if (!maps.make({a.x, static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.K), static_cast<uint32_t>(pl.x_rows), 128},
                 {a.w, static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.K), static_cast<uint32_t>(pl.bn), 128},
                 a.K, 128, pl.kc, pl.chunks))
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
  mp.chunks_3d = maps.chunks_3d;
  mp.splits = pl.splits;
  mp.stages = pl.stages;
  mp.stage_bytes = pl.stage_bytes;
  mp.ring_bytes = pl.ring_bytes;
  mp.out_pitch = pl.out_pitch;
  mp.tmem_cols = pl.bn;
  mp.a_scales = a.a_scales;
  mp.w_scales = a.w_scales;
  mp.bias = a.bias;
  mp.out = a.acc_out != nullptr ? static_cast<void*>(a.acc_out) : a.y;
  mp.status = a.status;
  cudaError_t e;
  const int ctas = pl.tiles_m * pl.tiles_n * pl.splits;
  if (a.acc_out != nullptr)
    e = launch_mid_kernel<w8a8_mid_kernel<true, __nv_bfloat16>>(ctas, pl.splits, pl.smem, a.stream, maps, mp);
  else
    e = a.dtype == B200Q_DTYPE_BF16
            ? launch_mid_kernel<w8a8_mid_kernel<false, __nv_bfloat16>>(ctas, pl.splits, pl.smem, a.stream, maps, mp)
            : launch_mid_kernel<w8a8_mid_kernel<false, __half>>(ctas, pl.splits, pl.smem, a.stream, maps, mp);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return B200Q_ERR_LAUNCH;
  }
  count_launch();
  return B200Q_OK;
}

}  // namespace b200q
