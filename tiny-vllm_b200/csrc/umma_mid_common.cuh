// What the two kernels for tens to hundreds of tokens (gemm_umma_mid.cu, gemm_umma_mid_w8a16.cu) share:
// cluster operations, the TMA producer warps, the table of plans and the launch.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "common.h"
#include "ptx_sm100.cuh"

namespace b200q {

// Residency rule.  tcgen05.alloc waits, without a limit, until the SM has that many free columns, and a CTA of a
// cluster keeps its columns until every CTA of the cluster has arrived at the cluster barrier.  Two CTAs of one cluster
// on one SM, or two clusters that each hold the columns the other one waits for, would therefore never end.  So the
// CTAs of clusters that can share an SM must not need more than its 512 columns together:
//   * at most two CTAs of these kernels fit an SM: more would exceed its registers (launch_mid_kernel checks it);
//   * a CTA of a cluster has at most 256 columns, or it takes the shared memory of a whole SM (kMidSmemOne: beside it there
//     is room for no kernel with dynamic shared memory).
// A CTA without a cluster may wait for columns: who holds them ends without it.  The other kernels that allocate
// tensor memory for clusters are alone on their SM: umma_pair_kernel by its shared memory (kPairSmem and kClusterSmemMin
// in common.h), the clustered w8a8_umma_kernel by its registers and its shared memory.
constexpr int kMidThreads = 352;
constexpr int kMidMaxStages = 12;
constexpr int kMidCtrlBytes = 768;
constexpr int kMidSmemTwo = 112 * 1024;          // two CTAs per SM
constexpr int kMidSmemOne = 226 * 1024;          // one, with a deep ring

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

// One operand's way through its ring of chunks of K blocks.
struct MidStream {
  const CUtensorMap* map;      // a block at a time: the end of K
  const CUtensorMap* map3;     // whole chunks of whole blocks: one instruction
  int row0, k_step;            // first row of the tile; bytes of a row per block
  int blk, kc;                 // bytes of a block's tile; blocks per chunk
  uint32_t dst, dst_step;      // shared address of the first slot, distance to the next
  int ring;                    // slots
  uint64_t *full, *free_bar;
  int c0, chunks, chunks_3d;   // first chunk, how many; chunks below chunks_3d come through map3
};

// One warp per operand: the weights run ahead as far as their ring allows, first of all ahead of
// the kernel that produces the activations.
__device__ __forceinline__ void mid_produce(const MidStream& s, volatile int* abort_flag) {
  int stage = 0;
  uint32_t phase = 1;                                      // the first round waits for nobody
  bool ok = true;
  for (int issued = 0; issued < s.chunks; ++issued) {
    if (ok && issued >= s.ring) ok = ptx::mbar_wait(ptx::smem_u32(s.free_bar + stage), phase, abort_flag);
    if (ptx::elect_one() && ok) {
      const uint32_t bar = ptx::smem_u32(s.full + stage), dst = s.dst + stage * s.dst_step;
      const int c = (s.c0 + issued) * s.kc;
      ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(s.kc * s.blk));
      if (s.c0 + issued < s.chunks_3d) {
        ptx::tma_load_3d(dst, s.map3, bar, 0, s.row0, c);
      } else {
        for (int b = 0; b < s.kc; ++b) ptx::tma_load_2d(dst + b * s.blk, s.map, bar, (c + b) * s.k_step, s.row0);
      }
    }
    __syncwarp();
    if (ok && ++stage == s.ring) {
      stage = 0;
      phase ^= 1u;
    }
  }
  if (ptx::elect_one() && *abort_flag != 0) ptx::drain_ring(s.full, s.ring, stage, phase ^ 1u);
}

// The search for a plan costs some 10 us of host time, more than the launch: its results are kept per
// thread, in a table of fixed size where a new shape replaces the one in its slot.
template <typename Plan, bool (*search)(int, int, int, Plan*)>
bool mid_plan(int M, int N, int K, Plan* best) {
  if (debug_knob(B200Q_KNOB_BN, 0) != 0 || debug_knob(B200Q_KNOB_CLUSTER, 0) != 0) return search(M, N, K, best);
  struct Entry {
    int M, N, K;   // M = 0: empty
    Plan plan;
  };
  constexpr unsigned kSlots = 1024;
  thread_local Entry table[kSlots];
  const unsigned h = static_cast<unsigned>(M) * 0x9E3779B1u ^ static_cast<unsigned>(N) * 0x85EBCA77u ^
                     static_cast<unsigned>(K) * 0xC2B2AE3Du;
  Entry& e = table[(h >> 16) % kSlots];
  if (e.M != M || e.N != N || e.K != K) {
    Entry fresh{M, N, K, {}};
    if (!search(M, N, K, &fresh.plan)) return false;
    e = fresh;
  }
  *best = e.plan;
  return true;
}

// Descriptors of a call's two operands.  Chunks of whole K blocks come through the 3-D maps, one instruction each; the
// chunk with a partial block, and what follows it, goes block by block through the 2-D ones (blocks beyond K
// read as zeros either way).  Only those that the kernel reads are made: an encoding costs a microsecond of
// host time, and the weights' are all made again on the first pass over a model and over a new box.
struct MidMaps {
  struct Matrix {
    const void* base;
    uint64_t rows, row_bytes;
    uint32_t box_rows, box_bytes;
  };
  CUtensorMap x, w, x3, w3;
  int chunks_3d;   // chunks below this one come through the 3-D maps
  bool make(const Matrix& mx, const Matrix& mw, int K, int block, int kc, int chunks) {
    chunks_3d = K % block == 0 ? chunks : K / block / kc;
    const uint32_t box = static_cast<uint32_t>(kc);
    if (chunks_3d < chunks && (!make_tensor_map(mx.base, mx.rows, mx.row_bytes, mx.box_rows, mx.box_bytes, &x) ||
                               !get_tensor_map(mw.base, mw.rows, mw.row_bytes, mw.box_rows, mw.box_bytes, &w)))
      return false;
    if (chunks_3d > 0 && (!make_tensor_map(mx.base, mx.rows, mx.row_bytes, mx.box_rows, mx.box_bytes, &x3, box) ||
                          !get_tensor_map(mw.base, mw.rows, mw.row_bytes, mw.box_rows, mw.box_bytes, &w3, box)))
      return false;
    if (chunks_3d == chunks) x = x3, w = w3;   // never read
    if (chunks_3d == 0) x3 = x, w3 = w;
    return true;
  }
};

template <auto kernel, typename Params>
cudaError_t launch_mid_kernel(int ctas, int splits, size_t smem, cudaStream_t stream, const MidMaps& maps,
                              const Params& mp) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmemOne);
    if (e != cudaSuccess) return e;
    int per_sm = 0;   // by registers and threads alone: the residency rule
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kMidThreads, 0);
    if (e != cudaSuccess) return e;
    if (per_sm > 2) return cudaErrorInvalidConfiguration;
    if (dev < 64) attr_set[dev] = true;
  }
  // Up to 32 tokens the neighbours may be kernels that live on L1 (reg_decode_preferred), and these leave an SM's memory
  // divided as it is: layers of 17 to 32 tokens with MAX_SHARED / without, W8A16 of hidden 1792 and 2048 1.03-1.045, W8A8 on codes of the 0.6B
  // model and of an eighth of the 8B one 1.05-1.09, with a quantiser 1.00-1.025, elsewhere 0.985-1.01.
  return launch_clustered(mp.M > 32 ? MAX_SHARED : DEFAULT_SPLIT, splits, true, kernel, dim3(ctas), dim3(kMidThreads), smem,
                          stream, maps.x, maps.w, maps.x3, maps.w3, mp);
}

}  // namespace b200q
