// W8A16 at tens to hundreds of tokens on tcgen05: weights expanded int8 -> 16 bit on the way (exact) into
// TENSOR memory, kind::f16, fp32 sums, then acc * s[n] + b[n]
// (nanovllm/quantization/csrc/int8_weight_only_gemm.cu:258-292, 397-412).
//
// The W8A16 counterpart of gemm_umma_mid.cu, whose reasons hold here too: the next kernel of the stream is resident
// while this one runs, weights are loaded AND expanded before the wait for the activations, several K
// blocks per TMA instruction and turn of the issue loop, K split over a cluster whose CTAs share the
// reduction.  What differs is where the expanded weights go.  In shared memory (as operand B beside the
// activations) they took a third of the ring, and their write, proxy fence and second read made the
// expansion the slowest stage.  Here
//   * the channels are the 128 rows of the UMMA tile and the tokens its columns (16 to 256): a converter thread
//     reads one row of int8 from shared memory and writes it expanded to its TMEM lane (tcgen05.st);
//     the MMA takes its A operand from there;
//   * a tile may have fewer than 128 channels: as many as give every CTA that the GPU holds one tile
//     (24576 x 4096 at 64 tokens: 280 tiles of 88 channels 26.3 us, 192 of 128 30.4);
//   * an MMA of 64 columns takes 51 cycles and one of 128 68, whatever part of the 128 rows is used, so
//     it is the tokens, the operand with fewer rows, that are cut finely.
// The output tile leaves through shared memory, two tokens to a word as the accumulators lie in a thread, then whole
// rows, 16 bytes a thread.  (4-byte stores from the registers, which neighbouring lanes had paired, took 2.2 us of a 128 x 128
// tile, this 1.2.)  With K split the owner's sums, scales and conversions work on vectors: 1.0 -> 0.7 us.
// Chains of launches, us per linear (without the two; expanded weights in shared memory; persistent kernels before
// that): 4096 x 1024 at 512 tokens 7.7 (8.6; 11.6; 13.7), 6144 x 1024 at 512 10.0 (10.7), 4096 x 1024 at 77 4.2 (4.7), 4096 x
// 512 at 64 3.3 (3.7), 4096 x 1536 at 64 4.8 (5.1), 768 x 4096 at 64 4.4 (4.4; 5.9; 16.0), 6144 x 4096 at 256 18.3 (19.3; 35.4; 39.6).
//
// Warp roles (352 threads): warp 0 TMA of the activations, warp 1 UMMA, warps 2-9 expansion (two groups of
// four that take the chunks in turn: a warp reaches one TMEM lane quarter), then epilogue, warp 10
// TMA of the weights.
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

constexpr int kMidCh = 128;                      // UMMA M: channels of a tile
constexpr int kMidWeightWarp = kMidThreads / 32 - 1;
constexpr int kMidACols = 32;                    // TMEM columns of one K block of expanded weights
constexpr int kOutPitch = kMidCh * 4;            // bytes of two tokens' rows of the output tile in shared memory

struct MidParams {
  int M, N;
  int bt;                  // tokens per tile (UMMA N)
  int rows;                // channels per tile: 128, or fewer where that spreads the matrix better
  int tiles_t;
  int kc;                  // K blocks (64 elements) per chunk
  int chunks, chunks_per_split;
  int chunks_3d;           // chunks below this one come through the 3-D maps: one TMA instruction
  int splits;              // cluster size
  int stages;              // ring of chunks of activations and of int8 weights: an even number, or one in all
  int stage_bytes, raw_bytes;
  int ring_bytes;          // both rings, or the output tile that lies over them at the end
  int a_stages;            // ring of chunks of expanded weights in TMEM (likewise)
  int a_col0;              // its first TMEM column
  int tmem_cols;
  int is_bf16;
  const float* w_scales;   // per channel
  const void* bias;        // per channel or nullptr
  void* out;
  int* status;
};

template <typename T>
__global__ void __launch_bounds__(kMidThreads, 2)
w8a16_mid_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_x3, const __grid_constant__ CUtensorMap tmap_w3,
                 const MidParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int rows_own = (p.bt + p.splits - 1) / p.splits;       // tokens a CTA owns
  const uint32_t raw_base = static_cast<uint32_t>(p.stages * p.stage_bytes);
  uint8_t* red = smem + p.ring_bytes;                          // [S][rows_own][128] 32-bit sums (S > 1)
  float* s_ws = reinterpret_cast<float*>(red + (p.splits > 1 ? p.splits * rows_own * kMidCh * 4 : 0));   // [128]
  uint8_t* ctrl = reinterpret_cast<uint8_t*>(s_ws + kMidCh);
  uint64_t* xfull = reinterpret_cast<uint64_t*>(ctrl);         // activations of a stage have landed
  uint64_t* empty = xfull + kMidMaxStages;                     // the MMAs that read a stage are done
  uint64_t* wfull = empty + kMidMaxStages;                     // int8 weights have landed
  uint64_t* rempty = wfull + kMidMaxStages;                    // ... and are read
  uint64_t* cfull = rempty + kMidMaxStages;                    // [4] expanded weights are in TMEM
  uint64_t* aempty = cfull + 4;                                // [4] the MMAs that read them are done
  uint64_t* tfull = aempty + 4;                                // accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(p.splits > 1 ? ptx::cluster_ctarank() : 0);
  const int tile = static_cast<int>(blockIdx.x) / p.splits;
  const int tile_t = tile % p.tiles_t, tile_c = tile / p.tiles_t;  // neighbours share the weights
  const int c0 = rank * p.chunks_per_split;
  const int n_ch = min(p.chunks, c0 + p.chunks_per_split) - c0;    // >= 1 by construction
  const uint32_t smem_base = ptx::smem_u32(smem);
  const bool aligned = (smem_base & 1023u) == 0u;
  const int x_blk = p.bt * 128;                                // one K block of activations

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(ptx::smem_u32(xfull + s), 1);
      ptx::mbar_init(ptx::smem_u32(empty + s), 1);
      ptx::mbar_init(ptx::smem_u32(wfull + s), 1);
      ptx::mbar_init(ptx::smem_u32(rempty + s), 4);
    }
    for (int s = 0; s < 4; ++s) {
      ptx::mbar_init(ptx::smem_u32(cfull + s), 4);
      ptx::mbar_init(ptx::smem_u32(aempty + s), 1);
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

  if (warp == 0 || warp == kMidWeightWarp) {
    if (run) {
      // -------------------------------------------------------------- TMA producers
      const bool weights = warp != 0;
      const MidStream s{weights ? &tmap_w : &tmap_x, weights ? &tmap_w3 : &tmap_x3,
                        weights ? tile_c * p.rows : tile_t * p.bt, weights ? kRow8 : 128,
                        weights ? p.rows * kRow8 : x_blk, p.kc, smem_base + (weights ? raw_base : 0u),
                        static_cast<uint32_t>(weights ? p.raw_bytes : p.stage_bytes), p.stages,
                        weights ? wfull : xfull, weights ? rempty : empty, c0, n_ch, p.chunks_3d};
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
      const uint32_t idesc = ptx::umma_idesc(1u, p.is_bf16 ? 1u : 0u, kMidCh, static_cast<uint32_t>(p.bt));
      int stage = 0, as = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      for (int i = 0; i < n_ch; ++i) {
        if (!ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(cfull + as), aphase, abort_flag) &&
                           ptx::mbar_wait(ptx::smem_u32(xfull + stage), phase, abort_flag))) {
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          uint64_t b_desc = ptx::umma_desc_k_sw128(smem_base + stage * p.stage_bytes);
          uint32_t a_tmem = tmem_base + static_cast<uint32_t>(p.a_col0 + as * p.kc * kMidACols);
          for (int b = 0; b < p.kc; ++b) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {   // 32 bytes of K per instruction
              const uint32_t acc = (i > 0 || b > 0 || k > 0) ? 1u : 0u;
              ptx::umma_f16_ts(tmem_base, a_tmem + 8u * k, b_desc + 2u * k, idesc, acc);
            }
            b_desc += static_cast<uint32_t>(x_blk >> 4);
            a_tmem += kMidACols;
          }
          ptx::umma_commit(ptx::smem_u32(empty + stage));
          ptx::umma_commit(ptx::smem_u32(aempty + as));
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++as == p.a_stages) {
          as = 0;
          aphase ^= 1u;
        }
      }
      if (ok && ptx::elect_one()) ptx::umma_commit(ptx::smem_u32(tfull));
    }
  } else {
    const int cw = warp - 2, tid = threadIdx.x - 64;
    const int quarter = warp & 3;                              // the TMEM lanes this warp may access
    const int ch = quarter * 32 + lane;                        // channel of the tile = TMEM lane
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    // channel scales: constants, fetched ahead of the wait
    if (tid < kMidCh) {
      const int col = tile_c * p.rows + tid;
      s_ws[tid] = tid < p.rows && col < p.N ? __ldg(p.w_scales + col) * kCodeUnit<T> : 0.f;
    }
    if (run) {
      // -------------------------------------------------------------- expansion
      // Both rings have an even number of slots, so a slot always belongs to the same group: a group that has not
      // seen the previous use of a slot complete could not tell its barrier's phases apart.
      const int group = cw >> 2;
      const int sw8 = (min(ch, p.rows - 1) >> 1) & 3;          // rows % 8 == 0: the same in every block
      int rs = group, as = group;
      uint32_t rphase = 0, aphase = 1;
      bool ok = true;
      for (int i = group; i < n_ch; i += 2) {
        if (!ptx::mbar_wait(ptx::smem_u32(wfull + rs), rphase, abort_flag)) ok = false;
        if (i >= p.a_stages && !ptx::mbar_wait(ptx::smem_u32(aempty + as), aphase, abort_flag)) ok = false;
        ptx::tc_fence_after_sync();
        // rows beyond the tile's last: what they hold only reaches accumulator lanes nobody reads
        const uint8_t* src = smem + raw_base + rs * p.raw_bytes + min(ch, p.rows - 1) * kRow8;
        for (int b = quarter * 32 < p.rows ? 0 : p.kc; b < p.kc; ++b, src += p.rows * kRow8) {
          uint32_t v[32];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 w = *reinterpret_cast<const uint4*>(src + ((c ^ sw8) << 4));
            const uint2 e0 = expand4_scaled<T>(w.x), e1 = expand4_scaled<T>(w.y), e2 = expand4_scaled<T>(w.z), e3 = expand4_scaled<T>(w.w);
            v[8 * c + 0] = e0.x;
            v[8 * c + 1] = e0.y;
            v[8 * c + 2] = e1.x;
            v[8 * c + 3] = e1.y;
            v[8 * c + 4] = e2.x;
            v[8 * c + 5] = e2.y;
            v[8 * c + 6] = e3.x;
            v[8 * c + 7] = e3.y;
          }
          ptx::tmem_st_32x32b_x32(lanes + static_cast<uint32_t>(p.a_col0 + (as * p.kc + b) * kMidACols), v);
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0 && ok) {
          ptx::mbar_arrive(ptx::smem_u32(cfull + as));
          ptx::mbar_arrive(ptx::smem_u32(rempty + rs));
        }
        if ((rs += 2) >= p.stages) {
          rs = group;
          rphase ^= 1u;
        }
        if ((as += 2) >= p.a_stages) {
          as = group;
          aphase ^= 1u;
        }
      }
    }
    __syncwarp();
    ptx::grid_dependency_wait();         // y may be in use by the previous kernel
    // every CTA of the cluster runs: its memory may be written / scales of this CTA complete
    if (p.splits > 1) cluster_wait();
    else ptx::named_bar_sync(1, 256);
    const bool done = run && ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(tfull), 0u, abort_flag));
    if (done) {
      ptx::tc_fence_after_sync();
      const T* bias = reinterpret_cast<const T*>(p.bias);
      const int n = tile_c * p.rows + ch;
      const bool mine_n = ch < p.rows && n < p.N;
      const int shift = __ffs(p.splits) - 1;
      const uint32_t mine = ptx::smem_u32(red) + static_cast<uint32_t>(rank * rows_own * kMidCh + ch) * 4u;
      const int live = min(p.bt, p.M - tile_t * p.bt);         // tokens of this tile
      for (int c = (cw >> 2) * 32; c < live; c += 64) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(lanes + static_cast<uint32_t>(c), v);
        ptx::tmem_ld_wait();
        if (p.splits > 1) {
          // ------------------------------------------ partial sums -> the tokens' owners
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int tok = c + j;
            if (tok < live && ch < p.rows)
              ptx::st_shared_cluster_u32(
                  ptx::map_to_cta(mine + static_cast<uint32_t>((tok >> shift) * kMidCh) * 4u,
                                  static_cast<uint32_t>(tok & (p.splits - 1))),
                  v[j]);
          }
        } else {
          // no split: scaled, rounded and two tokens to a word into shared memory as [token / 2][channel] (the rings
          // are done with: the MMAs that read the last of them have completed)
          uint32_t* slab = reinterpret_cast<uint32_t*>(smem + (c >> 1) * kOutPitch) + ch;
          const float w_s = s_ws[ch];
          const float b = bias != nullptr && mine_n ? to_float<T>(bias[n]) : 0.f;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float2 o = make_float2(__fmul_rn(__uint_as_float(v[j]), w_s), __fmul_rn(__uint_as_float(v[j + 1]), w_s));
            if (bias != nullptr) o = make_float2(__fadd_rn(o.x, b), __fadd_rn(o.y, b));
            slab[(j >> 1) * (kOutPitch / 4)] = pack2_rn<T>(o);
          }
        }
      }
    }
    if (p.splits == 1) {
      // whole rows of the tile, 16 bytes a thread (N % 8 == 0, rows % 8 == 0: a piece is inside or outside)
      ptx::named_bar_sync(1, 256);
      const int sub = tid & 15, n0 = tile_c * p.rows + sub * 8;
      if (done && sub < (p.rows >> 3) && n0 < p.N) {
        const int live = min(p.bt, p.M - tile_t * p.bt);
        T* out = static_cast<T*>(p.out) + static_cast<size_t>(tile_t * p.bt) * p.N + n0;
        for (int t0 = (tid >> 4) * 2; t0 < live; t0 += 64) {
          uint4 v[4];     // of token pairs t0 and t0 + 32: channels 0-3 and 4-7 of the piece
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (t0 + 32 * (j >> 1) < live)
              v[j] = *reinterpret_cast<const uint4*>(smem + (t0 / 2 + 16 * (j >> 1)) * kOutPitch + sub * 32 + 16 * (j & 1));
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int t = t0 + 32 * j;
            const uint4 a = v[2 * j], b = v[2 * j + 1];
            if (t < live)
              *reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * p.N) =
                  make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410), __byte_perm(b.x, b.y, 0x5410),
                             __byte_perm(b.z, b.w, 0x5410));
            if (t + 1 < live)
              *reinterpret_cast<uint4*>(out + static_cast<size_t>(t + 1) * p.N) =
                  make_uint4(__byte_perm(a.x, a.y, 0x7632), __byte_perm(a.z, a.w, 0x7632), __byte_perm(b.x, b.y, 0x7632),
                             __byte_perm(b.z, b.w, 0x7632));
          }
        }
      }
    }
  }
  if (p.splits > 1 && (warp < 2 || warp == kMidWeightWarp)) {
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

  // ------------------------------------------------------ own tokens: add, scale, round, store
  if (p.splits > 1) {
    const T* bias = reinterpret_cast<const T*>(p.bias);
    for (int u = threadIdx.x; u < rows_own * (kMidCh / 8); u += kMidThreads) {
      const int tl = u / (kMidCh / 8), cg = u % (kMidCh / 8);  // 8 channels: one 16-byte store
      const int tok = tl * p.splits + rank;
      const int row = tile_t * p.bt + tok, col = tile_c * p.rows + cg * 8;
      if (tok >= p.bt || cg * 8 >= p.rows || row >= p.M || col >= p.N) continue;   // N % 8 == 0
      float2 w[4];
      for (int s = 0; s < p.splits; ++s) {       // rank order: results do not depend on the run
        const float4* src = reinterpret_cast<const float4*>(red) + ((s * rows_own + tl) * kMidCh + cg * 8) / 4;
        const float4 a = src[0], b = src[1];
        const float2 in[4] = {{a.x, a.y}, {a.z, a.w}, {b.x, b.y}, {b.z, b.w}};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          w[j] = s == 0 ? in[j] : make_float2(__fadd_rn(w[j].x, in[j].x), __fadd_rn(w[j].y, in[j].y));
      }
      const float4 s0 = *reinterpret_cast<const float4*>(s_ws + cg * 8), s1 = *reinterpret_cast<const float4*>(s_ws + cg * 8 + 4);
      const float2 sc[4] = {{s0.x, s0.y}, {s0.z, s0.w}, {s1.x, s1.y}, {s1.z, s1.w}};
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = make_float2(__fmul_rn(w[j].x, sc[j].x), __fmul_rn(w[j].y, sc[j].y));
      if (bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          w[j] = make_float2(__fadd_rn(w[j].x, to_float<T>(bias[col + 2 * j])), __fadd_rn(w[j].y, to_float<T>(bias[col + 2 * j + 1])));
      }
      uint32_t packed[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) packed[j] = pack2_rn<T>(w[j]);
      *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + static_cast<size_t>(row) * p.N + col) =
          make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
  }
  if (threadIdx.x == 0 && *abort_flag != 0)
    atomicCAS(p.status, 0, 0xB00 | (*abort_flag << 4) | (static_cast<int>(blockIdx.x) << 12));
}

}  // namespace

// ------------------------------------------------------------------------------ host
namespace {

struct MidPlan {
  int bt, rows, splits, kc, chunks, chunks_per_split, tiles_t, tiles_c;
  int stages, stage_bytes, raw_bytes, ring_bytes, a_stages, a_col0, tmem_cols;
  size_t smem;
};

bool mid_plan_for(int M, int N, int k_blocks, int bt, int rows, int splits, int kc, int smem_cap, MidPlan* pl) {
  pl->bt = bt;
  pl->rows = rows;
  pl->kc = kc;
  pl->splits = splits;
  pl->chunks = (k_blocks + kc - 1) / kc;
  pl->chunks_per_split = (pl->chunks + splits - 1) / splits;
  if (pl->chunks_per_split * (splits - 1) >= pl->chunks) return false;   // a CTA without work
  pl->tiles_t = (M + bt - 1) / bt;
  pl->tiles_c = (N + rows - 1) / rows;
  pl->stage_bytes = kc * bt * 128;
  pl->raw_bytes = (kc * rows * kRow8 + 1023) / 1024 * 1024;
  const int rows_own = (bt + splits - 1) / splits;
  const int fixed = (splits > 1 ? splits * rows_own * kMidCh * 4 : 0) + kMidCh * 4 + kMidCtrlBytes;
  const int ring_bytes = pl->stage_bytes + pl->raw_bytes;
  int stages = std::min({(smem_cap - fixed) / ring_bytes, kMidMaxStages, pl->chunks_per_split});
  if (stages < 1 || (stages < 2 && pl->chunks_per_split > 1)) return false;
  // the converter groups take the chunks in turn: an even number of slots, or a single chunk
  if (pl->chunks_per_split > 1) stages &= ~1;
  int cols = (bt + 31) / 32 * 32;
  pl->a_col0 = cols;
  // at most 256 columns leave room for the next CTA; a wide tile takes them all
  const int chunk_cols = kc * kMidACols, room = (cols + 2 * chunk_cols <= 256 ? 256 : 512) - cols;
  pl->a_stages = std::min({room / chunk_cols, 4, pl->chunks_per_split});
  if (pl->chunks_per_split > 1) pl->a_stages &= ~1;
  if (pl->a_stages < 1) return false;
  cols += pl->a_stages * chunk_cols;
  pl->stages = stages;
  pl->tmem_cols = 32;
  while (pl->tmem_cols < cols) pl->tmem_cols *= 2;
  pl->ring_bytes = stages * ring_bytes;
  if (splits == 1) pl->ring_bytes = std::max(pl->ring_bytes, (bt + 31) / 32 * 16 * kOutPitch);
  pl->smem = static_cast<size_t>(pl->ring_bytes) + fixed;
  if (pl->smem > static_cast<size_t>(smem_cap)) return false;
  // no other CTA of a cluster fits beside it (see the residency rule in umma_mid_common.cuh)
  if (splits > 1) pl->smem = pl->tmem_cols > 256 ? kMidSmemOne : std::max<size_t>(pl->smem, kClusterSmemMin);
  return true;
}

// Predicted time of one call in a stream of such calls, in microseconds.  The form follows what the
// kernel does; the coefficients are fitted to 3,700 measured configurations (17 shapes from 2 to 100 MB of weights, 16
// to 1500 tokens) so that the one with the smallest prediction is close to the best: on average 1.5 %, at worst
// 12 % slower than it (a model with the expansion and HBM as further pipes: 3.6 and 30 %).
double mid_cost(const MidPlan& pl, int M) {
  const int ctas = pl.tiles_t * pl.tiles_c * pl.splits;
  const int per_sm = pl.smem <= kMidSmemTwo && pl.tmem_cols <= 256 ? 2 : 1;
  // clusters of 4 and 8 do not fill every SM (a cluster lives inside one group of SMs)
  const int sms = sm_count() - (pl.splits == 8 ? 28 : pl.splits == 4 ? 12 : 0);
  const int passes = (ctas + sms - 1) / sms, waves = (ctas + sms * per_sm - 1) / (sms * per_sm);
  // two CTAs on an SM wait on different things most of the time: the second costs 18 % of the first
  const double work = per_sm == 1 ? passes : waves * (1 + 0.182 * ((passes + waves - 1) / waves - 1));
  const double live = std::min(M, pl.bt);
  double us = 0.804 + pl.chunks_per_split * pl.kc * 4 * (39.1 + 0.0706 * pl.bt) * work / 1850.0;   // MMAs, at 1850 MHz
  // a ring shorter than the K loop goes round at the latency of a load
  us += 0.294 * waves * std::max(0, pl.chunks_per_split - pl.stages) / pl.stages;
  us += 0.319 * waves * pl.chunks_per_split;
  us += pl.splits > 1 ? 0.0165 * live * passes + 0.882 * std::log2(pl.splits) : 0.0144 * live * work;
  // start-up (1 us, and the first weights from HBM) hides under the previous kernel only as far as
  // both fit the GPU; alone on its SM a tile's start and end hide under nothing.  The neighbours in a layer
  // have other shapes: they are taken to hold 128 SMs at least (64 tokens through one eighth of the 8B model 21.5 us a
  // layer; planned for neighbours like itself 25.0)
  const double slots = static_cast<double>(sm_count()) * per_sm;
  us += (per_sm == 1 ? 2.38 : 2.8) * std::min(1.0, std::max(0.0, (ctas + std::max<double>(ctas, 128.0 * per_sm) - slots) / slots));
  if (per_sm == 1) us += 2.42 * (waves - 1);
  return us;
}

bool search_plan(int M, int N, int K, MidPlan* best) {
  const int k_blocks = (K + kBlockK - 1) / kBlockK;
  const int want_bt = debug_knob(B200Q_KNOB_BN, 0), want_s = debug_knob(B200Q_KNOB_CLUSTER, 0);
  double best_cost = 1e30;
  for (int bt : {16, 32, 48, 64, 96, 128, 192, 256}) {
    if (want_bt != 0 ? bt != want_bt : bt >= M + 32 && bt > 32) continue;
    const int tiles_t = (M + bt - 1) / bt;
    for (int s : {1, 2, 4, 8}) {
      if (want_s != 0 && s != want_s) continue;
      // channels per tile: all 128, or as many as make one tile for every CTA that the GPU holds
      for (int ctas : {0, 1, 2}) {
        int rows = kMidCh;
        if (ctas > 0) {
          const int tiles_c = ctas * sm_count() / (s * tiles_t);
          if (tiles_c < 1) continue;
          rows = ((N + tiles_c - 1) / tiles_c + 7) / 8 * 8;
          if (rows < 64 || rows >= kMidCh) continue;
        }
        for (int kc : {4, 2, 1}) {
          for (int cap : {kMidSmemOne, kMidSmemTwo}) {
            MidPlan pl;
            if (!mid_plan_for(M, N, k_blocks, bt, rows, s, kc, cap, &pl)) continue;
            if (s > 1 && pl.tiles_t * pl.tiles_c * s > 2 * sm_count()) continue;   // beyond what was measured
            const double cost = mid_cost(pl, M);
            if (cost < best_cost) {
              best_cost = cost;
              *best = pl;
            }
          }
        }
      }
    }
  }
  return best_cost < 1e30;
}

}  // namespace

// Up to 2.6 waves of 128 x 128 outputs.  There this kernel beats the persistent ones (gemm_umma_w8a16_ts.cu,
// and from 1024 tokens gemm_umma_pair.cu on weights expanded beforehand) at every measured shape: 24576 x 4096 at 24 tokens 28 against 49 us, at 256 61 against 106; 4096 x 4096 at 1200
// tokens 42 against 59; 6144 x 1024 at 800 15.0 against 24.4; 1024 x 2048 at 1500 12.7 against
// 21.6.  Beyond, an overlapped epilogue and an expansion done once win (6144 x 1024 at 1200 tokens, 3.2 waves:
// 23.1 against 22.1; 4096 x 1024 at 2000, 3.5 waves: 23.9 against 20.5), and above 2048 tokens little is left
// to gain on few tiles either (1024 x 2048 at 3000: 16.6 against 18.2).
bool umma16_mid_applicable(int M, int N, int K) {
  if (debug_knob(B200Q_KNOB_NO_MID, 0) != 0) return false;
  if ((K % 16) != 0 || (N % 8) != 0 || M < 1) return false;
  const long long tiles = static_cast<long long>((M + 127) / 128) * ((N + 127) / 128);
  if (M > 2048 || 5 * tiles > 13 * sm_count()) return false;
  if (debug_knob(B200Q_KNOB_BN, 0) == 0 && debug_knob(B200Q_KNOB_CLUSTER, 0) == 0) return true;
  MidPlan pl;   // a forced tile or cluster may not fit
  return mid_plan<MidPlan, search_plan>(M, N, K, &pl);
}

bool umma16_mid_shape(int M, int N, int K, MidShape* s) {
  MidPlan pl;
  if (!umma16_mid_applicable(M, N, K) || !mid_plan<MidPlan, search_plan>(M, N, K, &pl)) return false;
  *s = MidShape{pl.bt, pl.rows, pl.splits, pl.tmem_cols, static_cast<int>(pl.smem), pl.tiles_t * pl.tiles_c * pl.splits};
  return true;
}

int launch_umma16_mid(const GemmArgs& a) {
  MidPlan pl;
  if (!mid_plan<MidPlan, search_plan>(a.M, a.N, a.K, &pl)) return B200Q_ERR_UNSUPPORTED_SHAPE;
  MidMaps maps;
  if (!maps.make({a.x, static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.K) * 2, static_cast<uint32_t>(pl.bt), 128},
                 {a.w, static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.K), static_cast<uint32_t>(pl.rows), kRow8},
                 a.K, kBlockK, pl.kc, pl.chunks))
    return B200Q_ERR_LAUNCH;
  MidParams mp{};
  mp.M = a.M;
  mp.N = a.N;
  mp.bt = pl.bt;
  mp.rows = pl.rows;
  mp.tiles_t = pl.tiles_t;
  mp.kc = pl.kc;
  mp.chunks = pl.chunks;
  mp.chunks_per_split = pl.chunks_per_split;
  mp.chunks_3d = maps.chunks_3d;
  mp.splits = pl.splits;
  mp.stages = pl.stages;
  mp.stage_bytes = pl.stage_bytes;
  mp.raw_bytes = pl.raw_bytes;
  mp.ring_bytes = pl.ring_bytes;
  mp.a_stages = pl.a_stages;
  mp.a_col0 = pl.a_col0;
  mp.tmem_cols = pl.tmem_cols;
  mp.is_bf16 = a.dtype == B200Q_DTYPE_BF16 ? 1 : 0;
  mp.w_scales = a.w_scales;
  mp.bias = a.bias;
  mp.out = a.y;
  mp.status = a.status;
  const int ctas = pl.tiles_t * pl.tiles_c * pl.splits;
  const cudaError_t e =
      mp.is_bf16 ? launch_mid_kernel<w8a16_mid_kernel<__nv_bfloat16>>(ctas, pl.splits, pl.smem, a.stream, maps, mp)
                 : launch_mid_kernel<w8a16_mid_kernel<__half>>(ctas, pl.splits, pl.smem, a.stream, maps, mp);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return B200Q_ERR_LAUNCH;
  }
  count_launch();
  return B200Q_OK;
}

}  // namespace b200q
