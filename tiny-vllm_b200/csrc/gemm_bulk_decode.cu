// Weight-streaming decode kernels for decode-sized batches (M <= 32 tokens) over LARGE weight
// matrices: a persistent grid of one CTA per SM, each CTA owning an equal share of the output
// channels.  Eight lanes of a producer warp each feed one consumer warp through a private ring of
// shared-memory slots filled by TMA (cp.async.bulk.tensor, 128-byte swizzle, completion counted
// on mbarriers); the consumer warps run the same warp-level MMAs as the register-streaming
// kernels of gemm_mma_decode.cu.
//
// Why a second kernel.  The register-streaming kernel gives every 8 output channels a CTA of
// its own; each CTA re-reads the whole activation matrix from L2 (M x K bytes against 8 x K
// bytes of weights: twice the weight stream at M = 16) and has bytes in flight only between
// its start-up and its reduction, so on the 8B model's matrices (25-100 MB) it reaches
// 0.5-0.6 of the copy rate.  Here
//   * an SM asks for its weights through rings that always hold 100-190 KB of requests, none
//     of which occupy registers while they travel, and the first ring-full of weight tiles
//     is requested before the kernel waits for the producer of its activations;
//   * a unit of work is up to 48 channels, so the activations cross L2 -> SM once per 48
//     channels instead of once per 8;
//   * the channels are cut into one equal share per CTA (no 8-row rounding), so every SM
//     streams the same number of bytes and the grid has no tail;
//   * a tile is one TMA instruction per 48 rows x 128 bytes.  (Untiled cp.async.bulk row copies
//     of 0.5-1 KB were tried first: they retire at about one copy per 80 cycles per SM whatever
//     their size, 6-12 bytes per cycle, half of what the register kernel reaches.)
//
// Work split: K is cut into segments of 128 elements; segment s belongs to ring s % 8, which
// one consumer warp reads (or two, each taking half of the tile's rows).  Within a segment lane (g = lane / 4, t = lane % 4) owns elements [32 t, 32 t + 32) of
// weight rows g, g + 8, ..., g + 40 of the unit and of token rows g, g + 8 of every 16-token
// tile.  Which physical k sits in which MMA slot does not matter as long as both operands agree:
// 16-byte piece q of row r lies at r * 128 + ((q ^ (r & 7)) << 4) under the swizzle, and with
// pieces 2 t and 2 t + 1 per lane a quarter warp (two rows, four t) touches all eight 16-byte
// bank groups once.  The eight partial tiles are summed through shared memory in warp order,
// so results do not depend on the launch.
//   W8A8  m16n8k32 s8, exact int32 sums, then (float(acc) * a_s[m]) * w_s[n] + bias[n]
//         (nanovllm/quantization/csrc/w8a8_gemm.cu:165-183, 387-390)
//   W8A16 m16n8k16 f16/bf16 after an exact in-register expansion of the codes, fp32 sums of
//         x * float(q), then acc * s[n] + bias[n]
//         (nanovllm/quantization/csrc/int8_weight_only_gemm.cu:258-292)
// At most 8 tokens have a kernel of their own (stream_decode_m8_kernel).
// Rows and columns outside the matrices are zero-filled by TMA, so ragged K needs no masks.
// Every mbarrier wait is bounded; a wait that runs out stops the CTA's loops (the consumer
// warps still meet at their barriers), is reported through the status word, and the producer
// lanes wait, again bounded, for the tiles they still have in flight.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "common.h"
#include "expand_device.cuh"
#include "mma_device.cuh"
#include "ptx_sm100.cuh"

namespace b200q {
namespace {

constexpr int kPipes = 8;                        // rings per CTA = producer lanes
// A kernel has kPipes * WPP consumer warps (WPP = warps per ring: 1, or 2 sharing every tile,
// each taking half of its rows) and one producer warp.
constexpr int kSeg = 128;                        // K elements of one segment (one slot)
constexpr int kUnitRows = 48;                    // channels per unit of work (6 MMA n-tiles)
constexpr int kNT = kUnitRows / 8;
constexpr int kMaxSlots = 8;                     // ring depth per consumer warp
constexpr int kMaxMT = 2;  // token tiles: more would not fit the register file beside the prefetch
constexpr int kBarBytes = 2 * kPipes * kMaxSlots * 8;
constexpr int kSmemLimit = 227 * 1024;

// Host-made description of the rings and of the CTAs' shares of the channels.  Shared memory of a CTA (1 KB
// aligned): [8 rings x slots x weight tile][partial tiles of the consumer warps][activations, where they are kept
// here][full barriers][empty barriers][abort flag].
struct StreamPlan {
  int slots;       // ring depth per consumer warp
  int segs;        // segments of K: ceil(K / 128)
  int unit_rows;   // rows of the weight tile, <= 48
  int units;       // per CTA
  int share, rest; // channels per CTA; the first `rest` CTAs have one more
  int slot_bytes;  // bytes of a weight tile in shared memory (unit_rows x 128, 1 KB multiple)
  int tx_bytes;    // bytes TMA reports per tile
  int red_bytes;   // partial tiles of the consumer warps
  int x_pitch;     // bytes of a token row kept in shared memory, 0: activations are read from L2
  int x_bytes;
};

// The CTA's share of the channels, [lo, hi), cut into p.units pieces of at most p.unit_rows rows.
struct Share {
  int lo, hi;
};
__device__ __forceinline__ Share share_of(const StreamPlan& p, int cta) {
  Share s;
  s.lo = p.share * cta + min(cta, p.rest);
  s.hi = s.lo + p.share + (cta < p.rest ? 1 : 0);
  return s;
}
__device__ __forceinline__ void unit_range(const StreamPlan& p, const Share& s, int u, int& ulo, int& rows) {
  ulo = s.lo + u * p.unit_rows;
  rows = min(p.unit_rows, s.hi - ulo);   // shares differ by one channel: of the last unit that one may be all
}

template <int THREADS>
__device__ __forceinline__ void consumer_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}

// Producer lane `pipe` (0-7) feeds consumer warp `pipe`: segments pipe, pipe + 8, ... of every
// unit, in order, through that warp's ring.  Weights are constants, so nothing here waits for
// the previous kernel in the stream: the rings fill while that kernel is still finishing.
__device__ __forceinline__ void produce(const CUtensorMap* tm_w, const StreamPlan& p, const Share& sh,
                                        int pipe, uint32_t ring, uint64_t* full, uint64_t* empty,
                                        volatile int* abort_flag) {
  const int my_segs = (p.segs - pipe + kPipes - 1) / kPipes;
  int it = 0, slot = 0;
  uint32_t phase = 1;             // of the empty barriers; the first turn of the ring does not wait
  bool ok = true;
  for (int u = 0; ok && u < p.units; ++u) {
    int ulo, rows;
    unit_range(p, sh, u, ulo, rows);
    for (int c = 0; c < my_segs; ++c, ++it) {
      if (it >= p.slots && !ptx::mbar_wait(ptx::smem_u32(empty + slot), phase, abort_flag)) {
        ok = false;
        break;
      }
      const uint32_t bar = ptx::smem_u32(full + slot);
      ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(p.tx_bytes));
      ptx::tma_load_2d(ring + slot * p.slot_bytes, tm_w, bar, (pipe + kPipes * c) * kSeg, ulo);
      if (++slot == p.slots) {
        slot = 0;
        phase ^= 1u;
      }
    }
  }
  if (*abort_flag != 0) ptx::drain_ring(full, p.slots, slot, phase ^ 1u);   // a wait ran out somewhere in the CTA
}

struct CtaSmem {
  uint8_t* base;     // 1 KB aligned
  uint8_t* red;
  uint8_t* x;
  uint64_t* full;    // [8][kMaxSlots]
  uint64_t* empty;   // [8][kMaxSlots]
  volatile int* abort_flag;
};
__device__ __forceinline__ CtaSmem carve(uint8_t* raw, const StreamPlan& p) {
  CtaSmem c;
  const uint32_t a = ptx::smem_u32(raw);
  c.base = raw + ((1024u - (a & 1023u)) & 1023u);
  c.red = c.base + kPipes * p.slots * p.slot_bytes;
  c.x = c.red + p.red_bytes;
  c.full = reinterpret_cast<uint64_t*>(c.x + p.x_bytes);
  c.empty = c.full + kPipes * kMaxSlots;
  c.abort_flag = reinterpret_cast<volatile int*>(c.empty + kPipes * kMaxSlots);
  return c;
}
__device__ __forceinline__ void init_barriers(const CtaSmem& c, const StreamPlan& p, int wpp) {
  if (threadIdx.x < 2 * kPipes * kMaxSlots) {  // full and empty barriers are adjacent
    // a tile is filled by one TMA load and released by the wpp warps that read it
    ptx::mbar_init(ptx::smem_u32(c.full + threadIdx.x), threadIdx.x < kPipes * kMaxSlots ? 1 : wpp);
    if (threadIdx.x == 0) *c.abort_flag = 0;
    ptx::fence_mbar_init();
  }
  __syncthreads();
}

// ------------------------------------------------------------------------- W8A8
// 16 bytes of activations: a plain load (the read-only path may move it above the wait for the kernel that
// writes them).
__device__ __forceinline__ uint4 ld_act(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ float ld_scale(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Activations come straight from global memory (they are small and stay in L2): the lane's
// 32 bytes of token rows g and g + 8 of the NEXT segment are requested before the wait for
// the current weight tile, so their latency is covered by a whole segment of work.  (Keeping a
// lane's activations of all its segments in registers for the whole CTA, possible for
// K <= 4096, measured 1-2 us SLOWER: every CTA then asks for the same few lines at once.)
template <typename OutT, int MT, bool RAW_I32, int WPP>
__global__ void __launch_bounds__(kPipes * WPP * 32 + 32, 1)
w8a8_stream_decode_kernel(const __grid_constant__ CUtensorMap tm_w, const int8_t* xq,
                          const float* a_s, const float* __restrict__ w_s,
                          const OutT* __restrict__ bias, void* __restrict__ out, int M, int N, int K,
                          const StreamPlan p, int* status) {
  constexpr int kCW = kPipes * WPP, kCT = kCW * 32;  // consumer warps / threads
  constexpr int NTW = kNT / WPP;                     // 8-row MMA tiles per consumer warp
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const CtaSmem sm = carve(smem_raw, p);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Share sh = share_of(p, blockIdx.x);
  if (threadIdx.x == kCT) ptx::tma_prefetch_desc(&tm_w);
  init_barriers(sm, p, WPP);
  ptx::grid_launch_dependents();
  if (warp == kCW) {
    if (lane < kPipes)
      produce(&tm_w, p, sh, lane, ptx::smem_u32(sm.base) + lane * p.slots * p.slot_bytes,
              sm.full + lane * kMaxSlots, sm.empty + lane * kMaxSlots, sm.abort_flag);
    return;
  }
  ptx::grid_dependency_wait();  // activations and their scales come from the previous kernel

  const int g = lane >> 2, t = lane & 3;
  const int pipe = warp % kPipes, part = warp / kPipes;  // part: which NTW tiles of the unit
  const uint8_t* ring = sm.base + pipe * p.slots * p.slot_bytes;
  uint64_t* full = sm.full + pipe * kMaxSlots;
  uint64_t* empty = sm.empty + pipe * kMaxSlots;
  int* red = reinterpret_cast<int*>(sm.red);
  // swizzled positions of this lane's two 16-byte pieces in a 128-byte row whose index is g mod 8
  const int o0 = g * 128 + (((2 * t) ^ g) << 4), o1 = g * 128 + (((2 * t + 1) ^ g) << 4);
  const int my_segs = (p.segs - pipe + kPipes - 1) / kPipes;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

  // x[m][0..1] = pieces of token row m*16+g, x[m][2..3] = of token row m*16+g+8
  auto load_x = [&](int c, uint4 (&x)[MT][4]) {
    const int k = (pipe + kPipes * c) * kSeg + 32 * t;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int r0 = m * 16 + g, r1 = r0 + 8;
      const int8_t* p0 = xq + static_cast<size_t>(r0) * K + k;
      const int8_t* p1 = xq + static_cast<size_t>(r1) * K + k;
      x[m][0] = (r0 < M && k < K) ? ld_act(p0) : zero;
      x[m][1] = (r0 < M && k + 16 < K) ? ld_act(p0 + 16) : zero;
      x[m][2] = (r1 < M && k < K) ? ld_act(p1) : zero;
      x[m][3] = (r1 < M && k + 16 < K) ? ld_act(p1 + 16) : zero;
    }
  };

  uint4 xc[MT][4], xn[MT][4];
  if (p.units > 0 && my_segs > 0) load_x(0, xc);
  bool alive = true;
  int it = 0;
  for (int u = 0; u < p.units; ++u) {
    int ulo, rows;
    unit_range(p, sh, u, ulo, rows);
    int acc[MT][NTW][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < NTW; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][j][i] = 0;

    auto segment = [&](const uint4 (&xv)[MT][4]) {
      const int slot = it % p.slots;
      if (alive)
        alive = ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(full + slot), static_cast<uint32_t>((it / p.slots) & 1),
                                             sm.abort_flag));
      if (alive) {
        const uint8_t* ws = ring + slot * p.slot_bytes;
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
          const int jj = part * NTW + j;  // tile of the unit
          if (jj * 8 < rows) {
            const uint4 w0 = *reinterpret_cast<const uint4*>(ws + jj * 1024 + o0);
            const uint4 w1 = *reinterpret_cast<const uint4*>(ws + jj * 1024 + o1);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              // each pair of words is one k32 step: slots 4t..4t+3 and 16+4t..16+4t+3
              mma_s8(acc[m][j], xv[m][0].x, xv[m][2].x, xv[m][0].y, xv[m][2].y, w0.x, w0.y);
              mma_s8(acc[m][j], xv[m][0].z, xv[m][2].z, xv[m][0].w, xv[m][2].w, w0.z, w0.w);
              mma_s8(acc[m][j], xv[m][1].x, xv[m][3].x, xv[m][1].y, xv[m][3].y, w1.x, w1.y);
              mma_s8(acc[m][j], xv[m][1].z, xv[m][3].z, xv[m][1].w, xv[m][3].w, w1.z, w1.w);
            }
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(empty + slot));
      }
      ++it;
    };
    for (int c = 0; c < my_segs; ++c) {
      if (c + 1 < my_segs || u + 1 < p.units) load_x(c + 1 < my_segs ? c + 1 : 0, xn);
      segment(xc);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) xc[m][i] = xn[m][i];
    }

    // C fragment: acc[m][j][0..1] = (token m*16+g, channels 8j+2t, +1), [2..3] = token + 8
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      int* r = red + pipe * (16 * kUnitRows) + part * NTW * 8;
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        r[g * kUnitRows + j * 8 + 2 * t] = acc[m][j][0];
        r[g * kUnitRows + j * 8 + 2 * t + 1] = acc[m][j][1];
        r[(g + 8) * kUnitRows + j * 8 + 2 * t] = acc[m][j][2];
        r[(g + 8) * kUnitRows + j * 8 + 2 * t + 1] = acc[m][j][3];
      }
      consumer_barrier<kCT>();
      for (int o = threadIdx.x; o < 16 * kUnitRows; o += kCT) {
        const int tok = m * 16 + o / kUnitRows, ch = o % kUnitRows;
        if (tok >= M || ch >= rows) continue;
        int sum = 0;
#pragma unroll
        for (int wi = 0; wi < kPipes; ++wi) sum += red[wi * (16 * kUnitRows) + o];
        const int n = ulo + ch;
        const size_t idx = static_cast<size_t>(tok) * N + n;
        if (RAW_I32) {
          reinterpret_cast<int32_t*>(out)[idx] = sum;
        } else {
          const float b = bias != nullptr ? to_float<OutT>(bias[n]) : 0.f;
          const float v =
              __fadd_rn(__fmul_rn(__fmul_rn(static_cast<float>(sum), a_s[tok]), w_s[n]), b);
          reinterpret_cast<OutT*>(out)[idx] = from_float<OutT>(v);
        }
      }
      consumer_barrier<kCT>();
    }
  }
  if (threadIdx.x == 0 && *sm.abort_flag != 0)
    atomicCAS(status, 0, 0x900 | (static_cast<int>(blockIdx.x) << 12));
}

// ------------------------------------------------------------------------ W8A16
// The lane's 32 activations of a segment are 64 contiguous bytes per token row.  Weight word i
// of the lane (4 codes) meets activation words 2 i and 2 i + 1 (2 values each) in one k16 step.
template <typename T, int MT, int WPP>
__global__ void __launch_bounds__(kPipes * WPP * 32 + 32, 1)
w8a16_stream_decode_kernel(const __grid_constant__ CUtensorMap tm_w, const T* x,
                           const float* __restrict__ sc, const T* __restrict__ bias,
                           T* __restrict__ y, int M, int N, int K, const StreamPlan p, int* status) {
  constexpr int kCW = kPipes * WPP, kCT = kCW * 32;  // consumer warps / threads
  constexpr int NTW = kNT / WPP;                     // 8-row MMA tiles per consumer warp
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const CtaSmem sm = carve(smem_raw, p);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Share sh = share_of(p, blockIdx.x);
  if (threadIdx.x == kCT) ptx::tma_prefetch_desc(&tm_w);
  init_barriers(sm, p, WPP);
  ptx::grid_launch_dependents();
  if (warp == kCW) {
    if (lane < kPipes)
      produce(&tm_w, p, sh, lane, ptx::smem_u32(sm.base) + lane * p.slots * p.slot_bytes,
              sm.full + lane * kMaxSlots, sm.empty + lane * kMaxSlots, sm.abort_flag);
    return;
  }
  ptx::grid_dependency_wait();  // activations come from the previous kernel in the stream

  const int g = lane >> 2, t = lane & 3;
  const int pipe = warp % kPipes, part = warp / kPipes;  // part: which NTW tiles of the unit
  const uint8_t* ring = sm.base + pipe * p.slots * p.slot_bytes;
  uint64_t* full = sm.full + pipe * kMaxSlots;
  uint64_t* empty = sm.empty + pipe * kMaxSlots;
  float* red = reinterpret_cast<float*>(sm.red);
  const int o0 = g * 128 + (((2 * t) ^ g) << 4), o1 = g * 128 + (((2 * t + 1) ^ g) << 4);
  const int my_segs = (p.segs - pipe + kPipes - 1) / kPipes;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

  // xa[m][0..3] = the 32 values of token row m*16+g, xb[m][0..3] = of token row m*16+g+8
  auto load_x = [&](int c, uint4 (&xa)[MT][4], uint4 (&xb)[MT][4]) {
    const int k = (pipe + kPipes * c) * kSeg + 32 * t;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int r0 = m * 16 + g, r1 = r0 + 8;
      const T* p0 = x + static_cast<size_t>(r0) * K + k;
      const T* p1 = x + static_cast<size_t>(r1) * K + k;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool k_ok = k + 8 * j < K;  // K is a multiple of 16: a piece is inside or outside
        xa[m][j] = (r0 < M && k_ok) ? ld_act(p0 + 8 * j) : zero;
        xb[m][j] = (r1 < M && k_ok) ? ld_act(p1 + 8 * j) : zero;
      }
    }
  };

  uint4 ca[MT][4], cb[MT][4], na[MT][4], nb[MT][4];
  if (p.units > 0 && my_segs > 0) load_x(0, ca, cb);
  bool alive = true;
  int it = 0;
  for (int u = 0; u < p.units; ++u) {
    int ulo, rows;
    unit_range(p, sh, u, ulo, rows);
    float acc[MT][NTW][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < NTW; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][j][i] = 0.f;

    for (int c = 0; c < my_segs; ++c, ++it) {
      if (c + 1 < my_segs || u + 1 < p.units) load_x(c + 1 < my_segs ? c + 1 : 0, na, nb);
      const int slot = it % p.slots;
      if (alive)
        alive = ptx::warp_all(ptx::mbar_wait(ptx::smem_u32(full + slot), static_cast<uint32_t>((it / p.slots) & 1),
                                             sm.abort_flag));
      if (alive) {
        const uint8_t* ws = ring + slot * p.slot_bytes;
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
          const int jj = part * NTW + j;  // tile of the unit
          if (jj * 8 < rows) {
            const uint4 w0 = *reinterpret_cast<const uint4*>(ws + jj * 1024 + o0);
            const uint4 w1 = *reinterpret_cast<const uint4*>(ws + jj * 1024 + o1);
            const uint2 e0 = expand4_scaled<T>(w0.x), e1 = expand4_scaled<T>(w0.y), e2 = expand4_scaled<T>(w0.z),
                        e3 = expand4_scaled<T>(w0.w), e4 = expand4_scaled<T>(w1.x), e5 = expand4_scaled<T>(w1.y),
                        e6 = expand4_scaled<T>(w1.z), e7 = expand4_scaled<T>(w1.w);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              mma_16<T>(acc[m][j], ca[m][0].x, cb[m][0].x, ca[m][0].y, cb[m][0].y, e0.x, e0.y);
              mma_16<T>(acc[m][j], ca[m][0].z, cb[m][0].z, ca[m][0].w, cb[m][0].w, e1.x, e1.y);
              mma_16<T>(acc[m][j], ca[m][1].x, cb[m][1].x, ca[m][1].y, cb[m][1].y, e2.x, e2.y);
              mma_16<T>(acc[m][j], ca[m][1].z, cb[m][1].z, ca[m][1].w, cb[m][1].w, e3.x, e3.y);
              mma_16<T>(acc[m][j], ca[m][2].x, cb[m][2].x, ca[m][2].y, cb[m][2].y, e4.x, e4.y);
              mma_16<T>(acc[m][j], ca[m][2].z, cb[m][2].z, ca[m][2].w, cb[m][2].w, e5.x, e5.y);
              mma_16<T>(acc[m][j], ca[m][3].x, cb[m][3].x, ca[m][3].y, cb[m][3].y, e6.x, e6.y);
              mma_16<T>(acc[m][j], ca[m][3].z, cb[m][3].z, ca[m][3].w, cb[m][3].w, e7.x, e7.y);
            }
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(empty + slot));
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ca[m][i] = na[m][i];
          cb[m][i] = nb[m][i];
        }
    }

#pragma unroll
    for (int m = 0; m < MT; ++m) {
      float* r = red + pipe * (16 * kUnitRows) + part * NTW * 8;
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        r[g * kUnitRows + j * 8 + 2 * t] = acc[m][j][0];
        r[g * kUnitRows + j * 8 + 2 * t + 1] = acc[m][j][1];
        r[(g + 8) * kUnitRows + j * 8 + 2 * t] = acc[m][j][2];
        r[(g + 8) * kUnitRows + j * 8 + 2 * t + 1] = acc[m][j][3];
      }
      consumer_barrier<kCT>();
      for (int o = threadIdx.x; o < 16 * kUnitRows; o += kCT) {
        const int tok = m * 16 + o / kUnitRows, ch = o % kUnitRows;
        if (tok >= M || ch >= rows) continue;
        float sum = 0.f;
#pragma unroll
        for (int wi = 0; wi < kPipes; ++wi)
          sum = __fadd_rn(sum, red[wi * (16 * kUnitRows) + o]);  // fixed order
        const int n = ulo + ch;
        const float b = bias != nullptr ? to_float<T>(bias[n]) : 0.f;
        y[static_cast<size_t>(tok) * N + n] = from_float<T>(__fadd_rn(__fmul_rn(sum, sc[n] * kCodeUnit<T>), b));
      }
      consumer_barrier<kCT>();
    }
  }
  if (threadIdx.x == 0 && *sm.abort_flag != 0)
    atomicCAS(status, 0, 0x900 | (static_cast<int>(blockIdx.x) << 12));
}

// ------------------------------------------------- at most 8 tokens, either scheme
// With 8 tokens or fewer the CHANNELS go on the 16-row side of the MMA and the tokens on its 8-column side: one
// instruction covers 16 channels (rows g and g + 8 of a pair of 8-row tiles), half of what the kernels above issue.
// Two consumer warps share a ring, each with one of a lane's two 16-byte pieces of a row.
//
// What bounds a streaming kernel here is how fast a tile is consumed, not HBM: with the loads alone a chain of
// launches moves 6.7 TB/s, whatever the shape of the TMA boxes, and a round (a tile of every ring) takes 1800 cycles
// to arrive; expansions, MMAs and shared-memory reads of a round take 940 (W8A8 510) when nothing else is in
// the way.  Hence
//   * the number of 16-row tiles of a unit, NQ, is a template argument: a branch around a tile keeps the compiler
//     from overlapping the tiles' expansions and MMAs (24576 x 4096 from L2, 10.9 -> 9.3 us per 50 MB);
//   * a lane's weights of a segment go into registers at once and the slot back to the producer before the first MMA;
//   * the activations wait in shared memory where that pays (make_plan_m8): a load from L2 per segment costs more
//     than its MMAs;
//   * channel scales, which come from HBM, are asked for a unit ahead of their use.
// 1 token, us per launch in a chain, before / now: W8A16 24576 x 4096 24.0 / 18.1, 4096 x 12288 12.6 / 10.0, 6144 x 4096
// 7.2 / 6.5, 4096 x 4096 5.5 / 4.8; W8A8 (which had the 16-token kernel) 20.5 / 17.0, 11.1 / 9.4, 6.5 / 5.6, 5.3 / 4.1.
// Of what is left 2.5 us are the release by the previous kernel (0.8), the first activations from a busy L2 (1.2) and
// the last reduction.  Measured and not taken: two CTAs per SM, so that the next kernel fills its rings under this
// one (rings of half the depth cost more: 20.3-22.7 us, and CTAs of a grid meet on one SM when a small kernel stands
// between); weights prefetched into L2 beyond the ring (24-30 us); consumer warps that refill their rings themselves.
// X = int8_t: W8A8, exact int32 sums; else W8A16 with X = T, the type of the activations.
template <typename X, typename T, int NQ, bool X_SMEM>
__global__ void __launch_bounds__(kPipes * 2 * 32 + 32, 1)
stream_decode_m8_kernel(const __grid_constant__ CUtensorMap tm_w, const X* x, const float* a_s,
                        const float* __restrict__ sc, const T* __restrict__ bias, T* __restrict__ y, int M, int N,
                        int K, const StreamPlan p, int* status) {
  constexpr bool kA8 = sizeof(X) == 1;
  constexpr int kCW = kPipes * 2, kCT = kCW * 32;
  constexpr int kXP = kA8 ? 1 : 2;             // 16-byte pieces of activations that meet a piece of weights
  constexpr int kRows = NQ * 16;
  using Acc = typename std::conditional<kA8, int, float>::type;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const CtaSmem sm = carve(smem_raw, p);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Share sh = share_of(p, blockIdx.x);
  if (threadIdx.x == kCT) ptx::tma_prefetch_desc(&tm_w);
  init_barriers(sm, p, 2);
  ptx::grid_launch_dependents();
  if (warp == kCW) {
    if (lane < kPipes)
      produce(&tm_w, p, sh, lane, ptx::smem_u32(sm.base) + lane * p.slots * p.slot_bytes,
              sm.full + lane * kMaxSlots, sm.empty + lane * kMaxSlots, sm.abort_flag);
    return;
  }
  const int g = lane >> 2, t = lane & 3;
  const int pipe = warp % kPipes, part = warp / kPipes;  // part: which 16-byte piece of a lane's 32 bytes
  const uint8_t* ring = sm.base + pipe * p.slots * p.slot_bytes + g * 128 + (((2 * t + part) ^ g) << 4);
  const uint32_t full = ptx::smem_u32(sm.full + pipe * kMaxSlots), empty = ptx::smem_u32(sm.empty + pipe * kMaxSlots);
  Acc* red = reinterpret_cast<Acc*>(sm.red);
  const int my_segs = (p.segs - pipe + kPipes - 1) / kPipes;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  // this thread's output of a unit
  const int o_tok = static_cast<int>(threadIdx.x) / kRows, o_ch = static_cast<int>(threadIdx.x) % kRows;
  auto load_scale = [&](int u, float& o_sc, float& o_b) {
    int ulo, rows;
    unit_range(p, sh, u, ulo, rows);
    const bool mine = u < p.units && o_tok < M && o_ch < rows;
    o_sc = mine ? __ldg(sc + ulo + o_ch) : 0.f;
    o_b = mine && bias != nullptr ? to_float<T>(bias[ulo + o_ch]) : 0.f;
  };
  float o_sc, o_b;
  load_scale(0, o_sc, o_b);     // constants: ahead of the wait
  ptx::grid_dependency_wait();  // activations and their scales come from the previous kernel
  const float o_as = kA8 && o_tok < M ? ld_scale(a_s + o_tok) : 1.f;
  if (X_SMEM) {
    // token rows -> shared memory, zero beyond K up to the end of the last segment
    const int in16 = K * static_cast<int>(sizeof(X)) / 16, all16 = p.segs * (kSeg * static_cast<int>(sizeof(X)) / 16);
    for (int m = 0; m < M; ++m) {
      const uint8_t* src = reinterpret_cast<const uint8_t*>(x + static_cast<size_t>(m) * K);
      for (int i = threadIdx.x; i < all16; i += 4 * kCT) {
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = i + j * kCT < in16 ? ld_act(src + (i + j * kCT) * 16) : zero;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i + j * kCT < all16) *reinterpret_cast<uint4*>(sm.x + m * p.x_pitch + (i + j * kCT) * 16) = v[j];
      }
    }
    consumer_barrier<kCT>();
  }
  // the sixteen activations of token row g that meet this lane's piece of segment pipe + 8 c
  const int k_lane = pipe * kSeg + 32 * t + 16 * part;
  auto load_x = [&](int c, uint4 (&xv)[kXP]) {
    const int k = k_lane + c * (kPipes * kSeg);
    const bool in = g < M && (X_SMEM || k < K);    // K % 16 == 0: they are in or out together
#pragma unroll
    for (int j = 0; j < kXP; ++j) {
      if (X_SMEM)
        xv[j] = in ? *reinterpret_cast<const uint4*>(sm.x + g * p.x_pitch + k * static_cast<int>(sizeof(X)) + 16 * j) : zero;
      else
        xv[j] = in ? ld_act(reinterpret_cast<const uint8_t*>(x + static_cast<size_t>(g) * K + k) + 16 * j) : zero;
    }
  };
  uint4 xc[kXP], xn[kXP];
  if (!X_SMEM && my_segs > 0) load_x(0, xn);
  bool alive = true;
  int slot = 0;
  uint32_t phase = 0;
  for (int u = 0; u < p.units; ++u) {
    int ulo, rows;
    unit_range(p, sh, u, ulo, rows);
    Acc acc[NQ][4];
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[q][i] = 0;

    for (int c = 0; c < my_segs; ++c) {
      if (!X_SMEM) {
#pragma unroll
        for (int j = 0; j < kXP; ++j) xc[j] = xn[j];
        load_x(c + 1 < my_segs ? c + 1 : 0, xn);
      }
      // as a warp, by a vote where activations come from L2 on the way, else without (us, 1 token, staged: 8B, 16 linears
      // 160.7 with votes, 159.4 without; 7 tokens, not staged, 8 linears 101.7 and 102.8)
      if constexpr (X_SMEM) {
        if (alive) alive = ptx::mbar_wait(full + slot * 8, phase, sm.abort_flag);
      } else {
        if (alive) alive = ptx::warp_all(ptx::mbar_wait(full + slot * 8, phase, sm.abort_flag));
      }
      if (X_SMEM || alive) {
        const uint8_t* ws = ring + slot * p.slot_bytes;
        uint4 a[NQ], b[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          // channel 16 q + g (tile 2 q) and channel 16 q + 8 + g (tile 2 q + 1)
          a[q] = *reinterpret_cast<const uint4*>(ws + (2 * q) * 1024);
          b[q] = *reinterpret_cast<const uint4*>(ws + (2 * q + 1) * 1024);
        }
        if (X_SMEM) load_x(c, xc);
        // The slot may be overwritten once the loads have RETURNED: neither the barrier's release nor __syncwarp waits
        // for a load in flight, and the refill does not come through the pipe of the loads.  So the arrival depends
        // on a word of each of them (which lane arrives does not matter).
        uint32_t seen = 0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) seen |= a[q].x | b[q].x;
        const int who = __any_sync(0xFFFFFFFFu, seen == 0u) ? 1 : 0;
        if (lane == who && alive) ptx::mbar_arrive(empty + slot * 8);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          if constexpr (kA8) {
            mma_s8(acc[q], a[q].x, b[q].x, a[q].y, b[q].y, xc[0].x, xc[0].y);
            mma_s8(acc[q], a[q].z, b[q].z, a[q].w, b[q].w, xc[0].z, xc[0].w);
          } else {
            // weight word i of the piece meets activation words 2 i and 2 i + 1
            uint2 ea = expand4_scaled<T>(a[q].x), eb = expand4_scaled<T>(b[q].x);
            mma_16<T>(acc[q], ea.x, eb.x, ea.y, eb.y, xc[0].x, xc[0].y);
            ea = expand4_scaled<T>(a[q].y); eb = expand4_scaled<T>(b[q].y);
            mma_16<T>(acc[q], ea.x, eb.x, ea.y, eb.y, xc[0].z, xc[0].w);
            ea = expand4_scaled<T>(a[q].z); eb = expand4_scaled<T>(b[q].z);
            mma_16<T>(acc[q], ea.x, eb.x, ea.y, eb.y, xc[1].x, xc[1].y);
            ea = expand4_scaled<T>(a[q].w); eb = expand4_scaled<T>(b[q].w);
            mma_16<T>(acc[q], ea.x, eb.x, ea.y, eb.y, xc[1].z, xc[1].w);
          }
        }
      }
      if (++slot == p.slots) {
        slot = 0;
        phase ^= 1u;
      }
    }

    // C fragment: acc[q][0..1] = (channel 16q+g, tokens 2t, 2t+1), [2..3] = channel 16q+8+g.
    // One partial tile [M rounded up to 2][kRows] per consumer warp.
    const int red_tile = ((M + 1) & ~1) * kRows;
    if (2 * t < M) {
      Acc* r = red + warp * red_tile + 2 * t * kRows + g;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        r[16 * q] = acc[q][0];
        r[kRows + 16 * q] = acc[q][1];
        r[16 * q + 8] = acc[q][2];
        r[kRows + 16 * q + 8] = acc[q][3];
      }
    }
    consumer_barrier<kCT>();
    if (o_tok < M && o_ch < rows) {
      Acc sum = 0;
#pragma unroll
      for (int wi = 0; wi < kCW; ++wi) {   // fixed order
        const Acc v = red[wi * red_tile + o_tok * kRows + o_ch];
        if constexpr (kA8) sum += v; else sum = __fadd_rn(sum, v);
      }
      const float v = kA8 ? __fmul_rn(__fmul_rn(static_cast<float>(sum), o_as), o_sc)
                          : __fmul_rn(static_cast<float>(sum), o_sc * kCodeUnit<T>);
      y[static_cast<size_t>(o_tok) * N + ulo + o_ch] = from_float<T>(__fadd_rn(v, o_b));
    }
    load_scale(u + 1, o_sc, o_b);
    consumer_barrier<kCT>();
  }
  if (threadIdx.x == 0 && *sm.abort_flag != 0)
    atomicCAS(status, 0, 0x900 | (static_cast<int>(blockIdx.x) << 12));
}

// ------------------------------------------------------------------------ host
int grid_for(int N) { return N < sm_count() ? N : sm_count(); }

// Units of at most max_rows channels; the few-token kernel reads whole 16-row tiles (m8).
bool fit_plan(int N, int K, int max_rows, bool m8, int red_row_bytes, int x_pitch, int x_bytes, StreamPlan& p) {
  const int grid = grid_for(N);
  p.share = N / grid;
  p.rest = N % grid;
  const int most = p.share + (p.rest > 0 ? 1 : 0);
  p.units = (most + max_rows - 1) / max_rows;
  p.unit_rows = (most + p.units - 1) / p.units;
  const int padded = m8 ? (p.unit_rows + 15) / 16 * 16 : p.unit_rows;
  p.slot_bytes = (padded * 128 + 1023) / 1024 * 1024;
  p.tx_bytes = p.unit_rows * 128;
  p.segs = (K + kSeg - 1) / kSeg;
  p.red_bytes = red_row_bytes * (m8 ? padded : kUnitRows);
  p.x_pitch = x_pitch;
  p.x_bytes = x_bytes;
  const int fixed = p.red_bytes + p.x_bytes + kBarBytes + 16 + 1024;  // + slack for the 1 KB alignment
  if (fixed > kSmemLimit) return false;
  p.slots = (kSmemLimit - fixed) / (kPipes * p.slot_bytes);
  if (p.slots > kMaxSlots) p.slots = kMaxSlots;
  const int want = debug_knob(B200Q_KNOB_BULK_SLOTS, 0);  // tuning: a shallower ring
  if (want >= 2 && want < p.slots) p.slots = want;
  return p.slots >= 2;
}

// More than 8 tokens.
bool make_plan(int N, int K, StreamPlan& p) {
  return fit_plan(N, K, kUnitRows, false, kPipes * 16 * 4, 0, 0, p);
}

// At most 8 tokens.  The activations go to shared memory where the K loop, repeated for every unit, is long
// against copying them (us, 16-bit, staged / from L2: 1 token 6144 x 4096 6.4 / 7.1, 4096 x 12288 9.8 / 11.1; 4 tokens
// 24576 x 4096, 4 units, 19.9 / 21.9, but 6144 x 4096, one unit, 8.4 / 7.4; 8 tokens 24576 x 4096 23.9 / 22.7; int8,
// 2 tokens 6144 x 4096 6.3 / 6.2, 4 tokens 24576 x 4096 18.6 / 18.2).
bool make_plan_m8(int M, int N, int K, int x_size, StreamPlan& p) {
  const int red = kPipes * 2 * ((M + 1) / 2 * 2) * 4;
  if (!fit_plan(N, K, kUnitRows, true, red, 0, 0, p)) return false;
  if (M > p.units) return true;
  const long long row = static_cast<long long>(p.segs) * kSeg * x_size + 16;  // + 16: token rows on different banks
  StreamPlan q;
  if (row * M < kSmemLimit &&
      fit_plan(N, K, kUnitRows, true, red, static_cast<int>(row), static_cast<int>(row) * M, q))
    p = q;
  return true;
}

size_t plan_smem(const StreamPlan& p) {
  return static_cast<size_t>(kPipes) * p.slots * p.slot_bytes + p.red_bytes + p.x_bytes + kBarBytes + 16 + 1024;
}

// The kernel is a template ARGUMENT, so every kernel has a flag of its own (kernels of one
// signature share a function-pointer type).
template <auto kernel, typename... Args>
cudaError_t launch_stream(int grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  static bool raised[64] = {false};  // per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !raised[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return e;
    if (dev < 64) raised[dev] = true;
  }
  return launch_overlapped(MAX_SHARED, kernel, dim3(grid), dim3(threads), smem, stream, args...);
}

// knob BULK_WPP = 1: the 16-token kernels also for M <= 8 (tests compare the two forms)
bool takes_m8(const GemmArgs& a) {
  return a.M <= 8 && a.acc_out == nullptr && debug_knob(B200Q_KNOB_BULK_WPP, 2) != 1;
}

template <typename X, typename T, int NQ>
cudaError_t launch_m8_nq(const GemmArgs& a, const StreamPlan& p) {
  CUtensorMap tm_w;
  if (!get_tensor_map(a.w, a.N, a.K, p.unit_rows, 128, &tm_w)) return cudaErrorInvalidValue;
  const int threads = kPipes * 2 * 32 + 32;
  const X* x = static_cast<const X*>(a.x);
  const T* bias = static_cast<const T*>(a.bias);
  T* y = static_cast<T*>(a.y);
  return p.x_pitch != 0
             ? launch_stream<stream_decode_m8_kernel<X, T, NQ, true>>(grid_for(a.N), threads, plan_smem(p), a.stream, tm_w, x,
                                                                      a.a_scales, a.w_scales, bias, y, a.M, a.N, a.K, p, a.status)
             : launch_stream<stream_decode_m8_kernel<X, T, NQ, false>>(grid_for(a.N), threads, plan_smem(p), a.stream, tm_w, x,
                                                                       a.a_scales, a.w_scales, bias, y, a.M, a.N, a.K, p, a.status);
}
template <typename X, typename T>
cudaError_t launch_m8_typed(const GemmArgs& a) {
  StreamPlan p;
  if (!make_plan_m8(a.M, a.N, a.K, sizeof(X), p)) return cudaErrorInvalidValue;
  const int nq = (p.unit_rows + 15) / 16;
  const cudaError_t e = nq == 1 ? launch_m8_nq<X, T, 1>(a, p) : nq == 2 ? launch_m8_nq<X, T, 2>(a, p) : launch_m8_nq<X, T, 3>(a, p);
  if (e == cudaSuccess) count_launch();
  return e;
}
template <typename X>
cudaError_t launch_m8(const GemmArgs& a) {
  if constexpr (sizeof(X) == 1)
    return a.dtype == B200Q_DTYPE_BF16 ? launch_m8_typed<X, __nv_bfloat16>(a) : launch_m8_typed<X, __half>(a);
  else
    return launch_m8_typed<X, X>(a);
}

}  // namespace

// One token tile over matrices large enough that every SM gets a share worth a ring, unless the whole matrix
// is better held in registers (reg_decode_preferred).  Beyond 16 tokens the tcgen05 kernels are ahead (W8A8 at 32:
// 24576 x 4096 20.4 against 28.5 us).  Knob BULK_DECODE: 1 = never, 2 = wherever the kernel can run.
bool bulk_decode_applicable(int M, int N, int K, bool a16) {
  const int knob = debug_knob(B200Q_KNOB_BULK_DECODE, 0);
  if (knob == 1) return false;
  // 16-bit activations: one token tile (two tiles plus their prefetch exceed the register file)
  if (M < 1 || M > (a16 ? 16 : 16 * kMaxMT) || K < 16 || (K % 16) != 0 || N < 1) return false;
  StreamPlan p;
  if (!make_plan(N, K, p)) return false;
  if (knob == 2) return true;
  return M <= 16 && static_cast<long long>(N) * K >= (8ll << 20) && N >= 8 * sm_count() &&
         !(a16 && bulk_decode_yields(M, N, K)) && !reg_decode_preferred(M, N, K, a16);
}

// W8A16 from 9 tokens on: the 16-token kernel then needs twice the MMAs, and the tcgen05 kernel is ahead (us at 16 tokens, this
// kernel first): 24576 x 4096 34.4 and 22.9, 4096 x 12288 18.6 and 14.3, 9728 x 2560 12.6 and 9.4, 2560 x 9728 13.6
// and 10.1, 4096 x 4096 8.4 and 6.6.  It stays where a CTA's share is one well-filled unit of 40 to 48
// channels and the matrix is not large (6144 x 4096), the case it is laid out for.
bool bulk_decode_yields(int M, int N, int K) {
  const bool one_unit = N >= 40 * sm_count() && N <= kUnitRows * sm_count();
  return M > 8 && (N % 8) == 0 && !(one_unit && static_cast<long long>(N) * K < (32ll << 20));
}

cudaError_t launch_w8a8_bulk_decode(const GemmArgs& a) {
  StreamPlan p;
  if (takes_m8(a)) return launch_m8<int8_t>(a);
  if (!make_plan(a.N, a.K, p)) return cudaErrorInvalidValue;
  CUtensorMap tm_w;
  if (!get_tensor_map(a.w, a.N, a.K, p.unit_rows, 128, &tm_w)) return cudaErrorInvalidValue;
  const int8_t* xq = reinterpret_cast<const int8_t*>(a.x);
  const int grid = grid_for(a.N);
  const size_t smem = plan_smem(p);
  cudaError_t e = cudaSuccess;
#define B200Q_STREAM_A8(MT, WPP)                                                                   \
  if (a.acc_out != nullptr)                                                                        \
    e = launch_stream<w8a8_stream_decode_kernel<__nv_bfloat16, MT, true, WPP>>(                     \
        grid, kPipes * WPP * 32 + 32, smem, a.stream, tm_w, xq, a.a_scales, a.w_scales,             \
        static_cast<const __nv_bfloat16*>(nullptr), static_cast<void*>(a.acc_out), a.M, a.N, a.K,   \
        p, a.status);                                                                               \
  else if (a.dtype == B200Q_DTYPE_BF16)                                                            \
    e = launch_stream<w8a8_stream_decode_kernel<__nv_bfloat16, MT, false, WPP>>(                    \
        grid, kPipes * WPP * 32 + 32, smem, a.stream, tm_w, xq, a.a_scales, a.w_scales,             \
        static_cast<const __nv_bfloat16*>(a.bias), a.y, a.M, a.N, a.K, p, a.status);                \
  else                                                                                             \
    e = launch_stream<w8a8_stream_decode_kernel<__half, MT, false, WPP>>(                           \
        grid, kPipes * WPP * 32 + 32, smem, a.stream, tm_w, xq, a.a_scales, a.w_scales,             \
        static_cast<const __half*>(a.bias), a.y, a.M, a.N, a.K, p, a.status)
  // One token tile: two consumer warps per ring (more warps to cover the latencies of the
  // ring waits and the activation loads: 3-9 % on the 8B projections).  Two token tiles do not
  // fit the register file of 17 warps without spilling (M = 32: 28 against 17.6 us).
  if (a.M <= 16 && debug_knob(B200Q_KNOB_BULK_WPP, 2) == 2) {
    B200Q_STREAM_A8(1, 2);
  } else if (a.M <= 16) {
    B200Q_STREAM_A8(1, 1);
  } else {
    B200Q_STREAM_A8(2, 1);
  }
#undef B200Q_STREAM_A8
  if (e == cudaSuccess) count_launch();
  return e;
}

cudaError_t launch_w8a16_bulk_decode(const GemmArgs& a) {
  StreamPlan p;
  if (takes_m8(a)) return a.dtype == B200Q_DTYPE_BF16 ? launch_m8<__nv_bfloat16>(a) : launch_m8<__half>(a);
  if (!make_plan(a.N, a.K, p)) return cudaErrorInvalidValue;
  CUtensorMap tm_w;
  if (!get_tensor_map(a.w, a.N, a.K, p.unit_rows, 128, &tm_w)) return cudaErrorInvalidValue;
  const int grid = grid_for(a.N);
  const size_t smem = plan_smem(p);
  cudaError_t e = cudaSuccess;
#define B200Q_STREAM_A16(MT, WPP)                                                                  \
  if (a.dtype == B200Q_DTYPE_BF16)                                                                 \
    e = launch_stream<w8a16_stream_decode_kernel<__nv_bfloat16, MT, WPP>>(                          \
        grid, kPipes * WPP * 32 + 32, smem, a.stream, tm_w, static_cast<const __nv_bfloat16*>(a.x), \
        a.w_scales, static_cast<const __nv_bfloat16*>(a.bias), static_cast<__nv_bfloat16*>(a.y),    \
        a.M, a.N, a.K, p, a.status);                                                                \
  else                                                                                             \
    e = launch_stream<w8a16_stream_decode_kernel<__half, MT, WPP>>(                                 \
        grid, kPipes * WPP * 32 + 32, smem, a.stream, tm_w, static_cast<const __half*>(a.x),        \
        a.w_scales, static_cast<const __half*>(a.bias), static_cast<__half*>(a.y), a.M, a.N, a.K,   \
        p, a.status)
  // one consumer warp per ring: with two, each pair loads the activations twice and the 16-bit
  // fragments spill (gate_up at M = 1: 37.5 against 34.2 us)
  B200Q_STREAM_A16(1, 1);
#undef B200Q_STREAM_A16
  if (e == cudaSuccess) count_launch();
  return e;
}

}  // namespace b200q
