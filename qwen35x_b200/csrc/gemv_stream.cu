// Streaming W4A16 decode projection for sm_100a: one persistent launch walks a
// work list of (projection, 128-row block) tiles; M = 1..8 tokens.
//
// Replaces the per-phase matvec loops of the reference's persistent decode
// kernel (src/kernels/cuda/decode_kernel.cuh:58-84 calling nvfp4_row_dot,
// src/kernels/cuda/decode_layers.cuh:200-261) for the projections of a step.
//
// Data movement (what bounds the kernel): per 256-column K step a tile moves
//   16 KB of codes   128 rows x 128 B, cp.async.bulk.tensor.2d, 128B swizzle,
//                    straight from the checkpoint-order [rows, K/2] matrix
//    2 KB of scales  four 512-byte 128x4 tiles, cp.async.bulk
// into a shared-memory ring (mbarrier full/empty pairs), so each CTA keeps
// (stages x 18 KB) in flight regardless of how its consumer warps are doing.
//
// Arithmetic (kept off the critical path): one consumer warp per 16 rows of the tile.  Two shapes of CTA: eight
// consumer warps and half of an SM's shared memory, two CTAs per SM, so that one CTA's stalls (change of
// projection, tile hand-over, epilogue) run under the other's arithmetic; or, when the activations need more room,
// sixteen consumer warps in one CTA per SM, two per row group splitting every K step (their partial sums
// meet in shared memory at the end of the tile).  ldmatrix pulls 8 E2M1 codes per lane per register,
// cvt.rn.f16x2.e2m1x2 (the sm_100a FP4 converter) turns every byte into two
// exact fp16 values, and mma.sync m16n8k16 forms the 16-element block dot
// products against fp16 activations; the eight MMA columns are (half h of the
// 32-code chunk, token m<4), so one MMA pair yields, in each lane, the dot
// product of exactly the block that lane loaded: no cross-lane data movement.
// The E4M3 block scale multiplies that block dot in fp32 and accumulates.
// Five to eight tokens use a dense mapping instead: the eight MMA columns are the tokens, every k-slot is used,
// and the block scales are folded exactly into the fp16 weight operand, so the MMAs accumulate straight over K.
// Activations are converted BF16 -> fp16 per token with an exact power-of-two scale taken from the token's amax:
// a dedicated warp bulk-copies the raw rows of the next projection into one of two buffers (under the tiles of the
// projection before), and the consumer warps convert them in place when they get there, each a slice of
// one token, meeting twice on bounded mbarriers (amax known, conversion done).
//
// All waits are bounded; on expiry a code is written to the batch's status word.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <vector>

#include "engine.h"
#include "nvfp4_codec.cuh"

namespace q35b {
namespace {

constexpr int kTileRows = 128;
constexpr int kStepBytes = 128;                 // 256 codes per row per K step
constexpr int kCodesBytes = kTileRows * kStepBytes;
constexpr int kScaleBytes = 4 * 512;
constexpr int kStageBytes = kCodesBytes + kScaleBytes;
constexpr int kRowGroups = 8;                   // 16-row groups per tile
// Two shapes of CTA.  KS = 1: eight consumer warps, one per 16-row group, each taking the whole K step; 112 KB of
// shared memory, so that two CTAs share an SM and each one's stalls (change of projection, tile hand-over, epilogue)
// run under the other's arithmetic.  KS = 2: sixteen consumer warps, two per row group splitting every K step (their
// partial sums meet in shared memory at the end of a tile); one CTA per SM with all of its shared memory, for
// activations too large for the first shape.
__host__ __device__ constexpr int consumer_warps(int ks) { return kRowGroups * ks; }
__host__ __device__ constexpr int cta_threads(int ks) { return (2 + consumer_warps(ks)) * 32; }  // warp 0 producer, warp 1 activation copies
__host__ __device__ constexpr int ctas_per_sm(int ks) { return ks == 1 ? 2 : 1; }
__host__ __device__ constexpr int smem_budget(int ks) { return ks == 1 ? 112 * 1024 : 227 * 1024; }
// floats of the buffer in which the two warps of a row group meet (none when a warp takes the whole K step)
__host__ __device__ constexpr int red_floats(int ks, int mt) { return ks == 2 ? 2 * kRowGroups * 32 * 4 * mt : 0; }
constexpr int kMaxTilesInSmem = 64;             // tile descriptors staged per CTA
constexpr int kMaxStages = 8;
constexpr int kZeroHalfs = 320;                 // covers the 8 chunk offsets (32 halfs apart) of a K step + a bank shift
constexpr uint32_t kWaitLimit = 1u << 22;
// fp16 elements of padding between tokens.  Up to four tokens: consecutive tokens sit 32 bytes apart modulo the
// 128-byte bank window; five to eight tokens (the dense mapping below): 64 bytes apart, because there the eight lanes
// served together by a 128-bit load read 64 contiguous bytes of each of two tokens.
constexpr int kDenseFrom = 5;  // token count from which the dense MMA mapping (template MT = 2) is used; measured: with
                               // two to four tokens the (block, token) mapping is 4-7 % faster
__host__ __device__ constexpr int x_pad(int m_tokens) { return m_tokens >= kDenseFrom ? 32 : 16; }

enum StatusCode : unsigned { kProducerWait = 11, kPrepWait = 12, kConsumerWait = 13, kConsumerXWait = 14, kDependencyWait = 15 };

struct alignas(128) GemvItem {
  CUtensorMap tmap;              // codes [rows, K/2], box 128 rows x 128 bytes, 128B swizzle
  const uint8_t * scales_tiled;
  const __nv_bfloat16 * x;       // [m, K]
  __nv_bfloat16 * y;             // [m, rows]
  int rows;
  int k;
  int k_steps;                   // K / 256
  float s2;
};

// Everything a CTA needs to know about one tile, or about its part of a tile whose K steps are shared by several CTAs,
// staged in shared memory at kernel start so that no role chases pointers through global memory at a tile boundary.
// The order matters: with the fields that only shared tiles need in front of those every tile reads, a 4B-class step of
// four tokens took 345 us instead of 341.
struct alignas(16) GemvTile {
  int item;
  int row_block;
  int k;                           // columns of the projection
  int k_steps;                     // K steps of this part, from k_step0 on
  int rows;
  float s2;
  const uint8_t * scales;          // tiled scales of this row block, from its first K step on
  const __nv_bfloat16 * x;
  __nv_bfloat16 * y;
  const __nv_bfloat16 * residual;  // NULL or [m, rows]: added before the BF16 rounding
  float s2_up;                     // gate/up weight: weight_scale_2 of the up rows
  int flags;                       // kFlagGateUp | kFlagSignal
  int k_step0;
  int x0, x_len;                   // columns of the activations this CTA needs for this item (all its parts of it)
  int wait_item;                   // -1, or the item whose output this item's activations are
  unsigned int wait_count;         // completions that item reports per run (its tiles x 8 storing warps)
  int split;                       // arrival counters of a shared tile
  int slot0;                       // first of its slots of partial sums
  unsigned short part, parts;      // this part, and how many the tile has (1: not shared)
};
static_assert(sizeof(GemvTile) == 96, "tile descriptors are copied as 16-byte words and planned for in shared memory");
constexpr int kFlagGateUp = 1;   // rows alternate 8 gate / 8 up
constexpr int kFlagSignal = 2;   // another item waits for this one: count every stored tile part

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap * map, uint32_t bar, int x, int y) {
  asm volatile(
    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
    "l"(map), "r"(bar), "r"(x), "r"(y)
    : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void * src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t & r0, uint32_t & r1, uint32_t & r2, uint32_t & r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}

// Four bytes of E2M1 pairs -> four fp16x2 registers (low nibble in the low half): exact.
__device__ __forceinline__ void e2m1x8_to_f16(uint32_t w, uint32_t (&h)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
}

// d = a * b (+ c): fp16 operands, fp32 accumulate.
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm volatile(
    "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
    : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void mma_f16_acc(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
  asm volatile(
    "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
    : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Product of two fp16x2 registers.
__device__ __forceinline__ uint32_t hmul2_bits(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Unsigned E4M3 byte (bit 7 clear) -> fp32 (0x7f = 480, subnormals exact): the byte placed at bit 20 is the
// value scaled by 2^-120.  The shift is written as a multiply so that it issues on the FMA pipe.
__device__ __forceinline__ float ue4m3_to_f32(uint32_t byte) {
  return __uint_as_float(byte * 0x100000u) * 0x1p120f;
}

// A tile whose K steps several CTAs share: every storing warp leaves its scaled sums (each part has its own fp16 scales;
// `slots` is the first part's 512 bytes of this warp's row group, the next part's follow eight row groups on) and the
// last one of its row group to arrive adds them all in part order and gets true.  Nobody waits.  Out of line: it runs
// a few times per CTA, and inline it made every other tile slower (2-3 % of a step at four and eight tokens).
// The counter's low half counts the parts, its high half those whose warp gave up on an expired wait (give_up_parts):
// then nobody stores.  Either way the last part leaves it at zero for the next run.
constexpr unsigned int kPartCount = 0xffffu, kGaveUp = 0x10000u;
__device__ __noinline__ bool meet_parts(float4 & sum, float * slots, unsigned int * arrival, int part, int parts, int lane) {
  float4 * mine = reinterpret_cast<float4 *>(slots) + lane;
  constexpr int kNext = kRowGroups * 32;  // float4s between parts
  mine[part * kNext] = sum;
  __threadfence();
  __syncwarp();
  unsigned int before = 0;
  if (lane == 0) before = atomicAdd(arrival, 1u);
  before = __shfl_sync(0xffffffffu, before, 0);
  if ((before & kPartCount) != static_cast<unsigned int>(parts - 1)) return false;
  __threadfence();
  if (lane == 0) *arrival = 0u;
  if (before >= kGaveUp) return false;
  sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
  for (int p = 0; p < parts; ++p) {
    const float4 o = __ldcg(mine + p * kNext);
    sum.x += o.x;
    sum.y += o.y;
    sum.z += o.z;
    sum.w += o.w;
  }
  return true;
}

// A storing warp that gave up counts itself for its tiles from `tile` to `end` all the same (one thread per warp).
__device__ __noinline__ void give_up_parts(const GemvTile * tile, const GemvTile * end, unsigned int * arrivals, int rg) {
  for (; tile < end; ++tile) {
    if (tile->parts < 2) continue;
    unsigned int * arrival = arrivals + tile->split * kRowGroups + rg;
    if ((atomicAdd(arrival, 1u + kGaveUp) & kPartCount) == static_cast<unsigned int>(tile->parts - 1)) *arrival = 0u;
  }
}

// MT = number of 4-token groups (1 for M <= 4, 2 for M <= 8).  SHARED: some tiles of the list are shared by several CTAs
// (compiled in everywhere, that part of the epilogue made a step whose tiles are whole 1-2 % slower).
template <int MT, int KS, bool SHARED>
__global__ void __launch_bounds__(cta_threads(KS), ctas_per_sm(KS))
gemv_w4a16_stream_kernel(const GemvItem * __restrict__ items, const GemvTile * __restrict__ tiles,
                         const int * __restrict__ cta_begin, int m_tokens, const __nv_bfloat16 * x_override,
                         __nv_bfloat16 * y_override, int stages, int x_buf_halfs, int xs_buf_floats,
                         int x_bufs, unsigned long long * item_done,
                         int counted_items, float * partials, unsigned int * arrivals, unsigned int * status, uint32_t wait_limit, unsigned int wait_extra) {
  constexpr bool kDense = (MT == 2);  // five to eight tokens: dense MMA mapping
  constexpr int kConsumerWarps = consumer_warps(KS);
  constexpr int kConsumerShift = KS == 2 ? 4 : 3;  // log2(kConsumerWarps)
  constexpr int kThreads = cta_threads(KS);
  constexpr int kKSplit = KS;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment for the swizzled code tiles; pointer arithmetic on the __shared__ array (rather than an
  // integer round trip) keeps every later access a shared-memory access for the compiler.
  uint8_t * ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __half * xbuf = reinterpret_cast<__half *>(ring + stages * kStageBytes);        // x_bufs (1 or 2) buffers of x_buf_halfs
  __half * zeros = xbuf + x_bufs * x_buf_halfs;                                   // kZeroHalfs of 0.0, 128-byte aligned
  float * xsbuf = reinterpret_cast<float *>(zeros + kZeroHalfs);                   // 2 buffers of xs_buf_floats (1/scale)
  float * red = xsbuf + 2 * xs_buf_floats;                                         // 2 x [8 row groups][32 lanes][4*MT]
  GemvTile * stile = reinterpret_cast<GemvTile *>(red + red_floats(KS, MT));
  uint64_t * bars = reinterpret_cast<uint64_t *>(stile + kMaxTilesInSmem);
  // bars: full[kMaxStages], empty[kMaxStages], xfull[2], xempty[2], red_full[2], red_free[2], conv[2]
  uint64_t * full = bars;
  uint64_t * empty = bars + kMaxStages;
  uint64_t * xfull = bars + 2 * kMaxStages;
  uint64_t * xempty = xfull + 2;
  uint64_t * red_full = xempty + 2;
  uint64_t * red_free = red_full + 2;
  uint64_t * conv = red_free + 2;                                                  // consumers: amax known, conversion done
  uint32_t * amax_s = reinterpret_cast<uint32_t *>(conv + 2);                      // [2][8] per-token amax bits, by item parity

  // Programmatic dependent launch: the next kernel of the stream may start on an SM as soon as this kernel's CTA has
  // left it, and this kernel may start under the tail of the previous one.  Weights, tile descriptors and tensor
  // maps are constant for the life of the work list, so the producer streams them at once; whatever an earlier
  // kernel may have written (activations, residuals, completion counts) and every output store comes after
  // griddepcontrol.wait, which returns when all earlier work of the stream is complete and visible.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tile_begin = cta_begin[blockIdx.x];
  const int n_tiles = cta_begin[blockIdx.x + 1] - tile_begin;

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(smem_u32(full + i), 1);
      mbar_init(smem_u32(empty + i), kConsumerWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(xfull + i), 1);
      mbar_init(smem_u32(xempty + i), kConsumerWarps);
      mbar_init(smem_u32(red_full + i), kRowGroups);
      mbar_init(smem_u32(red_free + i), kRowGroups);
    }
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(conv + i), kConsumerWarps);
    for (int i = 0; i < 16; ++i) amax_s[i] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // stage this CTA's tile descriptors; clear the zero region
  for (int i = threadIdx.x; i < kZeroHalfs / 2; i += kThreads) reinterpret_cast<uint32_t *>(zeros)[i] = 0u;
  {
    const int n_stage = min(n_tiles, kMaxTilesInSmem);
    constexpr int kWords = sizeof(GemvTile) / 16;
    const uint4 * src = reinterpret_cast<const uint4 *>(tiles + tile_begin);
    uint4 * dst = reinterpret_cast<uint4 *>(stile);
    for (int i = threadIdx.x; i < n_stage * kWords; i += kThreads) dst[i] = __ldg(src + i);
  }
  __syncthreads();
  auto tile_at = [&](int i) -> const GemvTile * { return i < kMaxTilesInSmem ? stile + i : tiles + tile_begin + i; };

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int ti = 0; ti < n_tiles && ok; ++ti) {
        const GemvTile * tile = tile_at(ti);
        const CUtensorMap * tmap = &items[tile->item].tmap;
        const int k_steps = tile->k_steps;
        const uint8_t * sc = tile->scales;
        const int row0 = tile->row_block * kTileRows, byte0 = SHARED ? tile->k_step0 * kStepBytes : 0;
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!mbar_wait(smem_u32(empty + stage), phase ^ 1, wait_limit)) {
            atomicCAS(status, 0u, kProducerWait);
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(full + stage);
          uint8_t * dst = ring + stage * kStageBytes;
          mbar_expect_tx(bar, kStageBytes);
          tma_load_2d(smem_u32(dst), tmap, bar, byte0 + ks * kStepBytes, row0);
          bulk_load(smem_u32(dst + kCodesBytes), sc + static_cast<size_t>(ks) * kScaleBytes, kScaleBytes, bar);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ activation copies
    // Bulk-copies the raw BF16 activations of the next projection into one of the (one or two) activation buffers,
    // token rows padded apart; the consumers convert them to scaled fp16 in place.
    auto next_run = [&](int ti, int prev) {  // first tile index >= ti whose projection differs from `prev`
      while (ti < n_tiles && tile_at(ti)->item == prev) ++ti;
      return ti;
    };
    // An item that runs after another one may read its activations only when every storing warp of every tile of
    // that item has counted itself in item_done (stores fenced before the count).
    auto dependency_met = [&](const GemvTile * tl, bool block) -> bool {
      if (tl->wait_item < 0) return true;
      int met = 0;
      if (lane == 0) {
        const volatile unsigned long long * cnt = item_done + tl->wait_item;
        // a sixteenth of the budget of the barrier waits: when a dependency cannot be met this poll gives up first and
        // its code (the first one recorded stays) names the cause; the roles waiting on this warp follow
        for (uint32_t i = 0; i < max(wait_limit >> 4, 1u); ++i) {
          if (*cnt >= tl->wait_count + ((blockIdx.x & 1) == 0 ? wait_extra : 0u)) {
            met = 1;
            break;
          }
          if (!block) break;
          __nanosleep(32);
        }
      }
      met = __shfl_sync(0xffffffffu, met, 0);
      if (met) {
        __threadfence();
        asm volatile("fence.proxy.async;" ::: "memory");  // the bulk copy that follows reads what other SMs stored
      }
      return met != 0;
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int proc_ti = next_run(0, -1);
    uint32_t xi = 0;
    while (proc_ti < n_tiles) {
      // The raw BF16 rows of the next projection go straight into the (padded) buffer the consumers will read; the
      // sixteen consumer warps convert them in place when they reach the item.  (One warp converting eight tokens
      // takes several microseconds per item, and a CTA changes item at almost every tile of a 4B-class step.)
      // With two buffers the copy runs under the tiles of the item before.
      const GemvTile * tile = tile_at(proc_ti);
      if (!dependency_met(tile, true)) {
        if (lane == 0) atomicCAS(status, 0u, kDependencyWait);
        break;
      }
      const int buf = (x_bufs == 2) ? (xi & 1) : 0;
      const uint32_t xphase = (x_bufs == 2) ? ((xi >> 1) & 1) : (xi & 1);
      if (!mbar_wait(smem_u32(xempty + buf), xphase ^ 1, wait_limit)) {
        if (lane == 0) atomicCAS(status, 0u, kPrepWait);
        break;
      }
      if (lane == 0) {
        const int k = tile->k, len = SHARED ? tile->x_len : k;
        const uint32_t bar = smem_u32(xfull + buf);
        const __nv_bfloat16 * x = (x_override != nullptr ? x_override : tile->x) + (SHARED ? tile->x0 : 0);
        __half * xb = xbuf + buf * x_buf_halfs;
        mbar_expect_tx(bar, static_cast<uint32_t>(m_tokens) * len * 2u);
        for (int token = 0; token < m_tokens; ++token) {
          bulk_load(smem_u32(xb + static_cast<size_t>(token) * (len + x_pad(m_tokens))), x + static_cast<size_t>(token) * k,
                    static_cast<uint32_t>(len) * 2u, bar);
        }
      }
      ++xi;
      proc_ti = next_run(proc_ti + 1, tile->item);
    }
  } else {
    // ------------------------------------------------------------ consumers
    const int cw = warp - 2;           // 0..15
    const int rg = cw & 7;             // row group: tile rows 16*rg .. 16*rg+15
    const int kh = cw >> 3;            // which half of every K step (chunk pairs 2*kh, 2*kh+1)
    const int g = lane >> 2;
    const int t = lane & 3;
    // B-operand role of this lane: MMA column g = (half hB, token mB); it feeds k-slots owned by quad thread t.
    const int hB = g >> 2;
    const int mB = g & 3;
    const bool b_owner = (t >> 1) == hB;
    // D role: this lane receives block half hD = t >> 1, tokens 2*(t&1), 2*(t&1)+1 for rows g and g+8.
    const int hD = t >> 1;
    // Dense mapping (five to eight tokens): byte selectors that pull the scale of this lane's block (block
    // 2*cq + hD of a 4-block scale word) into both halves of a register.
    const uint32_t dense_sel[2] = {0x4040u | (static_cast<uint32_t>(hD) * 0x0101u),
                                   0x4040u | (static_cast<uint32_t>(2 + hD) * 0x0101u)};
    // ldmatrix row address of this lane: matrix mi = lane >> 3 -> rows 8*(mi&1).., chunk offset mi >> 1
    const int lm_row = 16 * rg + 8 * ((lane >> 3) & 1) + (lane & 7);
    const int lm_chunk = lane >> 4;
    const uint32_t lm_row_off = lm_row * kStepBytes;
    const int lm_xor = lm_row & 7;
    // scale word address pieces: row r -> (r % 32) * 16 + (r / 32) * 4 inside a 512-byte tile
    const int r0 = 16 * rg + g;
    const int sc_off0 = (r0 & 31) * 16 + (r0 >> 5) * 4;
    const int x_lane_off = 16 * hB + 8 * (t & 1);
    // The eight lanes served together by a 128-bit load hold two tokens of one block half: their activations fill a
    // 64-byte window of the 128-byte bank span (buffers are 128-byte aligned, tokens 32 bytes apart modulo 128).
    // Lanes that must feed zeros read them from the other 64 bytes of the span.
    const __half * zsrc = zeros + (m_tokens == 1 ? 48 : ((64 * (mB >> 1) + 32 * hB + 64) & 127) >> 1);

    int stage = 0;
    uint32_t phase = 0;
    uint32_t xi = 0;
    int prev_item = -1;
    int buf = 0;
    bool ok = true;
    int ti = 0;
    for (; ti < n_tiles && ok; ++ti) {
      const GemvTile * tile = tile_at(ti);
      if (tile->item != prev_item) {
        if (prev_item >= 0) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // a bulk copy overwrites what this warp converted
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(xempty + buf));
        }
        prev_item = tile->item;
        buf = (x_bufs == 2) ? (xi & 1) : 0;
        if (!mbar_wait(smem_u32(xfull + buf), (x_bufs == 2) ? ((xi >> 1) & 1) : (xi & 1), wait_limit)) {
          if (lane == 0) atomicCAS(status, 0u, kConsumerXWait);
          ok = false;
          break;
        }
        if (xi == 0) asm volatile("griddepcontrol.wait;" ::: "memory");  // returns at once: the activation warp has waited
        {
          // The raw BF16 rows of this item have landed in the buffer: the sixteen consumer warps turn them into
          // scaled fp16 in place.  With T = 1, 2, 4 or 8 token slots (the power of two that holds the tokens), warp
          // cw takes token cw % T and slice cw / T of its columns; the warps of a token agree on its amax through
          // shared memory.  Both meeting points are bounded mbarrier waits.
          const int tshift = m_tokens > 4 ? 3 : (m_tokens > 2 ? 2 : (m_tokens > 1 ? 1 : 0));
          const int ctoken = cw & ((1 << tshift) - 1);
          const int x_len = SHARED ? tile->x_len : tile->k;
          const int khalf = x_len >> (kConsumerShift - tshift);  // columns per slice
          const bool live = ctoken < m_tokens;
          __half * crow = xbuf + buf * x_buf_halfs + static_cast<size_t>(ctoken) * (x_len + x_pad(m_tokens)) + (cw >> tshift) * khalf;
          const uint32_t par = xi & 1;
          uint32_t amax_bits = 0;
          if (live) {
            for (int i = lane * 8; i < khalf; i += 256) {
              const uint4 q = *reinterpret_cast<const uint4 *>(crow + i);
              const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                amax_bits = max(amax_bits, (r[j] << 16) & 0x7fffffffu);
                amax_bits = max(amax_bits, r[j] & 0x7fff0000u);
              }
            }
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) amax_bits = max(amax_bits, __shfl_xor_sync(0xffffffffu, amax_bits, off));
          if (lane == 0) {
            if (live) atomicMax(amax_s + par * 8 + ctoken, amax_bits);
            mbar_arrive(smem_u32(conv + 0));
          }
          if (!mbar_wait(smem_u32(conv + 0), par, wait_limit)) {
            if (lane == 0) atomicCAS(status, 0u, kConsumerXWait);
            ok = false;
            break;
          }
          if (live) {
            // exact power-of-two scale putting the token's amax in [2^14, 2^15) (exponent field clamped to stay normal):
            // fp16 then holds every BF16 significand exactly down to 2^-28 of the amax
            int e = static_cast<int>(amax_s[par * 8 + ctoken] >> 23);
            e = min(max(e, 16), 254);
            const float scale = __uint_as_float(static_cast<uint32_t>(268 - e) << 23);
            for (int i = lane * 8; i < khalf; i += 256) {
              const uint4 q = *reinterpret_cast<const uint4 *>(crow + i);
              const uint32_t r[4] = {q.x, q.y, q.z, q.w};
              uint32_t out[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const __half2 h = __floats2half2_rn(__uint_as_float(r[j] << 16) * scale, __uint_as_float(r[j] & 0xffff0000u) * scale);
                out[j] = *reinterpret_cast<const uint32_t *>(&h);
              }
              *reinterpret_cast<uint4 *>(crow + i) = make_uint4(out[0], out[1], out[2], out[3]);
            }
            if ((cw >> tshift) == 0 && lane == 0) (xsbuf + buf * xs_buf_floats)[ctoken] = __uint_as_float(static_cast<uint32_t>(e - 14) << 23);
          }
          // the words of the other parity serve the next item: nobody reads them any more, nobody adds to them yet
          if (cw == 0 && lane < 8) amax_s[(par ^ 1) * 8 + lane] = 0u;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(conv + 1));
          if (!mbar_wait(smem_u32(conv + 1), par, wait_limit)) {
            if (lane == 0) atomicCAS(status, 0u, kConsumerXWait);
            ok = false;
            break;
          }
        }
        ++xi;
      }
      const int k_steps = tile->k_steps;
      const int xstride = (SHARED ? tile->x_len : tile->k) + x_pad(m_tokens);
      const __half * xb = xbuf + buf * x_buf_halfs + (SHARED ? tile->k_step0 * 256 - tile->x0 : 0);
      const float * xs = xsbuf + buf * xs_buf_floats;

      float acc[MT][4];
#pragma unroll
      for (int ts = 0; ts < MT; ++ts)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[ts][i] = 0.0f;

      // B-fragment source of this lane per token group: its slice of the fp16 activations if it owns k-slots of
      // that MMA column, else a zeroed region (same offsets work in both, so the inner loop has no predicates).
      const __half * bsrc[MT];
      int bstep[MT];
      if constexpr (kDense) {
        // dense mapping: MMA column g is token g; this lane feeds the k-slots of its own eight codes of a chunk
        const bool owner = g < m_tokens;
        bsrc[0] = owner ? xb + static_cast<size_t>(g) * xstride + 8 * t : zeros;
        bstep[0] = owner ? 256 : 0;
        bsrc[1] = bsrc[0];
        bstep[1] = 0;
      } else {
#pragma unroll
        for (int ts = 0; ts < MT; ++ts) {
          const int token = 4 * ts + mB;
          const bool owner = b_owner && token < m_tokens;
          bsrc[ts] = owner ? xb + static_cast<size_t>(token) * xstride + x_lane_off : zsrc;
          bstep[ts] = owner ? 256 : 0;
        }
      }
      for (int ks = 0; ks < k_steps; ++ks) {
        if (!mbar_wait(smem_u32(full + stage), phase, wait_limit)) {
          if (lane == 0) atomicCAS(status, 0u, kConsumerWait);
          ok = false;
          break;
        }
        const uint8_t * codes = ring + stage * kStageBytes;
        const uint8_t * sc = codes + kCodesBytes;
        const uint32_t codes_addr = smem_u32(codes) + lm_row_off;

#pragma unroll
        for (int pp = 0; pp < 4 / kKSplit; ++pp) {
          const int pair = (4 / kKSplit) * kh + pp;
          uint32_t r[4];
          ldmatrix_x4(codes_addr + (((2 * pair + lm_chunk) ^ lm_xor) << 4), r[0], r[1], r[2], r[3]);
          if constexpr (kDense) {
            // Five to eight tokens: the eight MMA columns are the tokens, every k-slot is used, and the chunk's two
            // blocks (quad threads 0,1 and 2,3) share one MMA.  Their block scales therefore go into the A operand:
            // E2M1 x E4M3 is exact in fp16 (the scale byte at bit 7 of an fp16 is the scale times 2^-8, 0x7f = 480
            // included; products down to 2^-18 are fp16 subnormals, which multiply and MMA handle exactly), and
            // the MMAs accumulate straight over K in fp32.  The 2^8 is undone in the epilogue.
            const uint32_t sw0 = *reinterpret_cast<const uint32_t *>(sc + pair * 512 + sc_off0);        // row r0, 4 blocks
            const uint32_t sw1 = *reinterpret_cast<const uint32_t *>(sc + pair * 512 + sc_off0 + 128);  // row r0 + 8
#pragma unroll
            for (int cq = 0; cq < 2; ++cq) {
              const int q = 2 * pair + cq;
              uint32_t a_lo[4], a_hi[4];
              e2m1x8_to_f16(r[2 * cq], a_lo);
              e2m1x8_to_f16(r[2 * cq + 1], a_hi);
              const uint32_t s0 = __byte_perm(sw0, 0u, dense_sel[cq]) << 7;  // (scale, scale) as fp16x2, times 2^-8
              const uint32_t s1 = __byte_perm(sw1, 0u, dense_sel[cq]) << 7;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                a_lo[i] = hmul2_bits(a_lo[i], s0);
                a_hi[i] = hmul2_bits(a_hi[i], s1);
              }
              const uint4 b = *reinterpret_cast<const uint4 *>(bsrc[0] + 32 * q);
              mma_f16_acc(acc[cq], a_lo[0], a_hi[0], a_lo[1], a_hi[1], b.x, b.y);
              mma_f16_acc(acc[cq], a_lo[2], a_hi[2], a_lo[3], a_hi[3], b.z, b.w);
            }
          } else {
          // scale bytes of this pair's 4-block tile (blocks 4*pair .. 4*pair+3 of rows r0 and r0+8): plain byte
          // loads keep the integer pipe free for the FP4 conversions
          const uint8_t * sc0 = sc + pair * 512 + sc_off0 + hD;
#pragma unroll
          for (int cq = 0; cq < 2; ++cq) {
            const int q = 2 * pair + cq;  // 32-code chunk index inside the K step
            uint32_t a_lo[4], a_hi[4];
            e2m1x8_to_f16(r[2 * cq], a_lo);      // rows 0..7 of the warp's 16
            e2m1x8_to_f16(r[2 * cq + 1], a_hi);  // rows 8..15
            // block 2*cq + hD of the 4-block tile; rows r0 and r0 + 8 (128 bytes further)
            const float s0 = ue4m3_to_f32(sc0[2 * cq]);
            const float s1 = ue4m3_to_f32(sc0[2 * cq + 128]);
#pragma unroll
            for (int ts = 0; ts < MT; ++ts) {
              const uint4 b = *reinterpret_cast<const uint4 *>(bsrc[ts] + 32 * q);
              float c[4];
              mma_f16_zero(c, a_lo[0], a_hi[0], a_lo[1], a_hi[1], b.x, b.y);
              mma_f16_acc(c, a_lo[2], a_hi[2], a_lo[3], a_hi[3], b.z, b.w);
              acc[ts][0] = fmaf(c[0], s0, acc[ts][0]);
              acc[ts][1] = fmaf(c[1], s0, acc[ts][1]);
              acc[ts][2] = fmaf(c[2], s1, acc[ts][2]);
              acc[ts][3] = fmaf(c[3], s1, acc[ts][3]);
            }
          }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(empty + stage));
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
#pragma unroll
        for (int ts = 0; ts < MT; ++ts) bsrc[ts] += bstep[ts];
      }
      if (!ok) break;
      if constexpr (kDense) {
        // the two MMA chains (even and odd chunks) hold partial sums of the same outputs
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][i] += acc[1][i];
      }
      constexpr int kGroups = kDense ? 1 : MT;  // float4 groups of sums a lane carries into the epilogue
      static_assert(kGroups == 1, "the epilogue handles four sums per lane");

      // Meet the partner warp's half-K sums in shared memory (double-buffered by tile parity): the kh = 1 warp
      // writes, the kh = 0 warp adds, combines the two block halves (lanes t and t^2) and stores.
      const int rb = ti & 1;
      const uint32_t rphase = (ti >> 1) & 1;
      float * slot = red + ((rb * kRowGroups + rg) * 32 + lane) * 4 * MT;
      if (kKSplit == 2 && kh == 1) {
        if (!mbar_wait(smem_u32(red_free + rb), rphase ^ 1, wait_limit)) {
          if (lane == 0) atomicCAS(status, 0u, kConsumerWait);
          ok = false;
          break;
        }
#pragma unroll
        for (int ts = 0; ts < kGroups; ++ts)
          *reinterpret_cast<float4 *>(slot + 4 * ts) = make_float4(acc[ts][0], acc[ts][1], acc[ts][2], acc[ts][3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(red_full + rb));
      } else {
        if constexpr (kKSplit == 2) {
          if (!mbar_wait(smem_u32(red_full + rb), rphase, wait_limit)) {
            if (lane == 0) atomicCAS(status, 0u, kConsumerWait);
            ok = false;
            break;
          }
#pragma unroll
          for (int ts = 0; ts < kGroups; ++ts) {
            const float4 o = *reinterpret_cast<const float4 *>(slot + 4 * ts);
            acc[ts][0] += o.x;
            acc[ts][1] += o.y;
            acc[ts][2] += o.z;
            acc[ts][3] += o.w;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(red_free + rb));
        }
        __nv_bfloat16 * y = y_override != nullptr ? y_override : tile->y;
        const int rows = tile->rows;
        const bool gate_up = (tile->flags & kFlagGateUp) != 0;
        const float s2 = tile->s2, s2_up = gate_up ? tile->s2_up : s2;  // of rows r0 and r0 + 8
        const int row_a = tile->row_block * kTileRows + r0;
        const __nv_bfloat16 * residual = tile->residual;
        const int parts = SHARED ? tile->parts : 1;
        if constexpr (!kDense) {
          // the two block halves of a chunk sit in lanes t and t ^ 2
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[0][i] += __shfl_xor_sync(0xffffffffu, acc[0][i], 2);
        }
        if (parts > 1) {
          const int tok = 2 * (kDense ? t : t & 1);
          const float u0 = xs[tok] * (kDense ? 256.0f : 1.0f), u1 = xs[tok + 1] * (kDense ? 256.0f : 1.0f);
          float4 sum = make_float4(acc[0][0] * (u0 * s2), acc[0][1] * (u1 * s2), acc[0][2] * (u0 * s2_up), acc[0][3] * (u1 * s2_up));
          if (!meet_parts(sum, partials + (static_cast<size_t>(tile->slot0) * kRowGroups + rg) * 128,
                          arrivals + tile->split * kRowGroups + rg, tile->part, parts, lane)) continue;
          acc[0][0] = sum.x;
          acc[0][1] = sum.y;
          acc[0][2] = sum.z;
          acc[0][3] = sum.w;
        }
        // dense: this lane holds tokens 2t, 2t+1 of rows r0 and r0 + 8, with the block scales' 2^-8 still in
        if (kDense || t < 2) {
          const int tok0 = 2 * t;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (tok0 + e < m_tokens) {
              const float unscale = xs[tok0 + e] * (kDense ? 256.0f : 1.0f);  // undoes the token's fp16 scaling
              if (gate_up) {
                // rows alternate 8 gate / 8 up: this lane's row r0 is gate row j, its row r0 + 8 the matching up row
                const int j = (row_a >> 4) * 8 + (row_a & 7);
                if (row_a + 8 < rows) {
                  const float gate = acc[0][e] * (parts > 1 ? 1.0f : unscale * s2);
                  const float up = acc[0][2 + e] * (parts > 1 ? 1.0f : unscale * s2_up);
                  y[static_cast<size_t>(tok0 + e) * (rows >> 1) + j] = __float2bfloat16_rn(gate / (1.0f + expf(-gate)) * up);
                }
              } else {
                const float f = parts > 1 ? 1.0f : unscale * s2;
                if (row_a < rows) {
                  const size_t o = static_cast<size_t>(tok0 + e) * rows + row_a;
                  const float r = residual != nullptr ? __bfloat162float(residual[o]) : 0.0f;
                  y[o] = __float2bfloat16_rn(acc[0][e] * f + r);
                }
                if (row_a + 8 < rows) {
                  const size_t o = static_cast<size_t>(tok0 + e) * rows + row_a + 8;
                  const float r = residual != nullptr ? __bfloat162float(residual[o]) : 0.0f;
                  y[o] = __float2bfloat16_rn(acc[0][2 + e] * f + r);
                }
              }
            }
          }
        }
        if ((tile->flags & kFlagSignal) != 0) {
          // another item of this run reads these outputs: make the stores visible, then count this warp's part
          __threadfence();
          __syncwarp();
          if (lane == 0) atomicAdd(item_done + tile->item, 1ULL);
        }
      }
    }
    if constexpr (SHARED) {
      // the parts from the tile it gave up in on; a warp leaves that loop only before its tile's parts meet.  One that ran
      // out of polls on its first activations may still be under the run before, whose parts use the same counters.
      if (!ok && kh == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0) give_up_parts(tiles + tile_begin + ti, tiles + tile_begin + n_tiles, arrivals, rg);
      }
    }
    if (ok && prev_item >= 0) {
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(xempty + buf));
    }
  }
  if (counted_items > 0) {
    // A run with dependencies leaves its completion counts at zero for the next one: the last CTA to get here clears
    // them (every wait of the run has ended by then, since every CTA is past its last tile).
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned int * ctas_done = reinterpret_cast<unsigned int *>(item_done + counted_items);
      __threadfence();
      if (atomicAdd(ctas_done, 1u) == gridDim.x - 1) {
        for (int i = 0; i < counted_items; ++i) item_done[i] = 0ULL;
        *ctas_done = 0u;
      }
    }
  }
}

constexpr int kBarrierBytes = (2 * kMaxStages + 8 + 2) * 8 + 2 * 8 * 4;

struct Plan {
  int stages = 0;
  int x_buf_halfs = 0;
  int xs_buf_floats = 0;
  int x_bufs = 0;
  int smem_bytes = 0;
  int ksplit = 2;  // shape of the CTA (template KS)
};

// Shared-memory plan for a batch with at most max_k columns: activation buffers (raw BF16 rows land in them and are
// converted in place, so there is no separate raw ring), then as many ring stages as fit.  Two buffers (the next
// item's copy runs under the current item's tiles) when at least five stages remain, else one.
bool make_plan(int m, int max_k, Plan * p, int min_ks = 1) {
  const int mt = m < kDenseFrom ? 1 : 2;
  const int x_halfs = ((m * (max_k + x_pad(m)) + 63) / 64) * 64;  // whole 128-byte bank spans
  const int xs_floats = 8;
  // The two-CTAs-per-SM shape first (measured: 0.8B-class step at one token 51 -> 45 us); it needs four ring stages
  // per CTA beside two activation buffers, or three beside one.  Else the one-CTA shape with all of the SM's memory.
  for (int ks = min_ks; ks <= 2; ++ks) {
    const int base = 1024 + 2 * xs_floats * 4 + red_floats(ks, mt) * 4 + kZeroHalfs * 2 +
                     kMaxTilesInSmem * static_cast<int>(sizeof(GemvTile)) + kBarrierBytes;
    for (int bufs = 2; bufs >= 1; --bufs) {
      const int fixed = base + bufs * x_halfs * 2;
      const int stages = std::min(kMaxStages, (smem_budget(ks) - fixed) / kStageBytes);
      if (stages >= (bufs == 2 ? (ks == 1 ? 4 : 5) : 3)) {
        p->stages = stages;
        p->x_buf_halfs = x_halfs;
        p->xs_buf_floats = xs_floats;
        p->x_bufs = bufs;
        p->smem_bytes = fixed + stages * kStageBytes;
        p->ksplit = ks;
        return true;
      }
    }
  }
  return false;
}

using StreamKernel = void (*)(const GemvItem *, const GemvTile *, const int *, int, const __nv_bfloat16 *, __nv_bfloat16 *,
                              int, int, int, int, unsigned long long *, int, float *, unsigned int *, unsigned int *, uint32_t, unsigned int);

StreamKernel stream_kernel(int m, int ks, bool shared) {
  if (shared) {
    if (m < kDenseFrom) return ks == 1 ? gemv_w4a16_stream_kernel<1, 1, true> : gemv_w4a16_stream_kernel<1, 2, true>;
    return ks == 1 ? gemv_w4a16_stream_kernel<2, 1, true> : gemv_w4a16_stream_kernel<2, 2, true>;
  }
  if (m < kDenseFrom) return ks == 1 ? gemv_w4a16_stream_kernel<1, 1, false> : gemv_w4a16_stream_kernel<1, 2, false>;
  return ks == 1 ? gemv_w4a16_stream_kernel<2, 1, false> : gemv_w4a16_stream_kernel<2, 2, false>;
}

// The plan for a list on the current device: the two-CTAs-per-SM shape only if two of its CTAs really fit on an SM
// (items that wait for other items rely on every CTA of the grid being resident).
cudaError_t plan_for_device(int m, int max_k, bool share_tiles, Plan * p, bool * fits) {
  *fits = make_plan(m, max_k, p);
  if (!*fits) return cudaSuccess;
  for (const bool shared : {false, true}) {
    if (shared && !share_tiles) break;  // a list of whole tiles never runs that kernel
    cudaError_t e = cudaFuncSetAttribute(stream_kernel(m, p->ksplit, shared), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_budget(p->ksplit));
    if (e != cudaSuccess) return e;
    if (p->ksplit == 2) continue;
    int resident = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, stream_kernel(m, 1, shared), cta_threads(1),
                                                      static_cast<size_t>(p->smem_bytes));
    if (e != cudaSuccess) return e;
    if (resident < 2) {
      *fits = make_plan(m, max_k, p, 2);
      if (!*fits) return cudaSuccess;
      for (const bool sh : {false, true}) {
        e = cudaFuncSetAttribute(stream_kernel(m, 2, sh), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_budget(2));
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
  }
  return cudaSuccess;
}

}  // namespace
}  // namespace q35b

using namespace q35b;

struct q35b_gemv_batch {
  int count = 0;
  int m = 0;
  int grid = 0;
  int device = 0;
  Plan plan;
  void * dev_base = nullptr;
  GemvItem * items = nullptr;
  GemvTile * tiles = nullptr;
  int * cta_begin = nullptr;
  unsigned int * status = nullptr;
  unsigned long long * item_done = nullptr;  // per item: storing warps that finished a tile in the current run
  unsigned int * arrivals = nullptr;         // per shared tile and row group: parts that have left their sums
  float * partials = nullptr;                // the parts' sums
  size_t counter_bytes = 0;                  // status, item_done, arrivals and chain_gave, contiguous and zero between runs
  bool has_dependencies = false;
  bool shared = false;                       // some tiles are shared by several CTAs
  size_t bytes_per_run = 0;
  uint32_t wait_limit = kWaitLimit;   // polls every device-side wait of a run may take
  unsigned int wait_extra = 0;        // test hook: completions that every other CTA demands on top of what a dependency delivers
  q35b::WBatch * tensor = nullptr;   // set: the list runs on the tensor path (gemm_wstream.cu), nothing above is used
  std::vector<q35b_gemv_item> chain;  // set: it can run as one launch per item, in this order (gemm_resident.cu)
  bool chained = false;               // it does
  q35b_gemv_batch * one_launch = nullptr;  // test hook: the same list without a chain, for dependencies that cannot be met
  unsigned int * chain_gave = nullptr;  // of a chain, two words per item: whether its launch gave up (gemm_resident.cu)
  int chain_absent = -1;              // test hook: item whose operand is never complete in every other row block
};

namespace q35b {

bool gemv_stream_eligible(const q35b_weight * w, int m) {
  if (w == nullptr || w->rows <= 0 || (w->k % 256) != 0 || w->negative_scales) return false;
  Plan p;
  return make_plan(m, w->k, &p);
}

int gemv_plan_debug(int m, int max_k, int * ctas, int * ring_stages, int * activation_buffers, int * smem_bytes) {
  if (m < 1 || m > 8 || max_k < 256 || (max_k % 256) != 0) return fail(Q35B_ERR_SHAPE, "NVFP4 decode projection supports 1..8 tokens and cols that are a multiple of 256.");
  Plan p;
  if (!make_plan(m, max_k, &p)) return fail(Q35B_ERR_SHAPE, "Activations of the NVFP4 projection work list do not fit in shared memory.");
  if (ctas != nullptr) *ctas = ctas_per_sm(p.ksplit);
  if (ring_stages != nullptr) *ring_stages = p.stages;
  if (activation_buffers != nullptr) *activation_buffers = p.x_bufs;
  if (smem_bytes != nullptr) *smem_bytes = p.smem_bytes;
  return Q35B_OK;
}

namespace {

// What each CTA of a grid of `grid` does: contiguous runs of tiles (projection-major order) of about equal cost, level
// by level (a CTA changes projection, and converts a new activation vector, as rarely as possible, and neighbouring
// CTAs stream neighbouring rows; an item's level is one more than that of the item it runs after, and every level is
// spread over all CTAs by itself, so that the whole grid works on the tiles something is waiting for).
//
// A tile goes to the CTA in whose share of the total its midpoint falls.  With whole tiles the down projection of one
// layer, [2560, 9216], keeps 20 of 296 CTAs busy for 36 K steps each.  So where a level has fewer tiles than the grid has
// CTAs, a CTA's share ends where it ends, inside a tile if need be, and the tile's parts meet in memory at the end (MLP
// block [2560, 9216] at two tokens 40 -> 25 us, [512, 8192] 24 -> 15).  From five tokens on the conversion of the weights
// bounds a CTA rather than the bandwidth all CTAs share, and an even split pays up to four tiles per CTA (a step of 41 us
// at seven tokens 38); with fewer tokens the CTAs that finish early leave their bandwidth to the others, and meeting costs
// more than it saves (steps of 19 us at one and two tokens: 20 and 22).
// A part has at least kMinPart steps (parts of four or more: the blocks above 25 and 15 us, [3584, 3328] 24 instead of 20).
// A level whose tiles are all short stays whole: meeting takes about as long as eight steps of a CTA that has an SM's
// bandwidth to itself ([512, 1280] at four tokens 10.7 us whole, 12.5 shared; [768, 2048] 13.5 and 13.7).
constexpr int kMinPart = 2;
constexpr int kWholeSteps = 8;

struct Assignment {
  std::vector<std::vector<GemvTile>> per_cta;
  int splits = 0, slots = 0;  // shared tiles, and parts of shared tiles
  int max_x = 0;              // most activation columns any CTA needs of an item
};

Assignment assign_tiles(const std::vector<GemvTile> & all, const std::vector<int> & level, int max_level, int grid, int m, bool share_tiles) {
  Assignment out;
  out.per_cta.resize(grid);
  for (int lv = 0; lv <= max_level; ++lv) {
    long total = 0;
    int tiles = 0, longest = 0;
    for (const GemvTile & tl : all) {
      if (level[tl.item] != lv) continue;
      total += tl.k_steps + 1;
      ++tiles;
      longest = std::max(longest, tl.k_steps);
    }
    const bool share = share_tiles && longest > kWholeSteps && (tiles < grid || (m >= kDenseFrom && tiles < 4 * grid));
    long done = 0;
    int c = 0;
    for (const GemvTile & tl : all) {
      if (level[tl.item] != lv) continue;
      const int cost = tl.k_steps + 1;
      if (!share) {
        while (c + 1 < grid && (done + cost / 2) * grid >= static_cast<long>(c + 1) * total) ++c;
        out.per_cta[c].push_back(tl);
        done += cost;
        continue;
      }
      while (c + 1 < grid && (static_cast<long>(c + 1) * total + grid / 2) / grid <= done) ++c;  // shares that are full
      std::vector<std::pair<int, int>> cuts;  // (CTA, end step) of the parts so far
      int begin = 0;
      while (begin < tl.k_steps) {
        // where CTA c's share ends, in steps of this tile
        const long end_cost = (static_cast<long>(c + 1) * total + grid / 2) / grid - done;
        int end = c + 1 < grid ? static_cast<int>(std::min<long>(std::max<long>(end_cost, 0), tl.k_steps)) : tl.k_steps;
        if (tl.k_steps - end < kMinPart) end = tl.k_steps;
        if (end - begin >= kMinPart || (end == tl.k_steps && begin == 0)) {
          cuts.emplace_back(c, end);
          begin = end;
        } else if (end == tl.k_steps && !cuts.empty()) {
          cuts.back().second = end;  // too short a rest for the next CTA
          begin = end;
        }
        if (begin < tl.k_steps || end_cost <= cost) c = std::min(c + 1, grid - 1);
      }
      done += cost;
      if (cuts.size() > 1) ++out.splits;
      int step = 0;
      for (size_t i = 0; i < cuts.size(); ++i) {
        GemvTile part = tl;
        part.k_step0 = step;
        part.k_steps = cuts[i].second - step;
        part.scales = tl.scales + static_cast<size_t>(step) * kScaleBytes;
        part.part = static_cast<unsigned short>(i);
        part.parts = static_cast<unsigned short>(cuts.size());
        part.split = out.splits - 1;
        part.slot0 = out.slots;
        step = cuts[i].second;
        out.per_cta[cuts[i].first].push_back(part);
      }
      if (cuts.size() > 1) out.slots += static_cast<int>(cuts.size());
    }
  }
  for (auto & tiles : out.per_cta) {
    std::stable_sort(tiles.begin(), tiles.end(), [&](const GemvTile & a, const GemvTile & d) {
      if (level[a.item] != level[d.item]) return level[a.item] < level[d.item];
      return a.item != d.item ? a.item < d.item : a.row_block < d.row_block;
    });
    // the columns of an item's activations that any of the CTA's parts of it reads
    for (size_t i = 0; i < tiles.size();) {
      size_t j = i;
      int lo = tiles[i].k_step0, hi = lo;
      for (; j < tiles.size() && tiles[j].item == tiles[i].item; ++j) {
        lo = std::min(lo, tiles[j].k_step0);
        hi = std::max(hi, tiles[j].k_step0 + tiles[j].k_steps);
      }
      for (; i < j; ++i) {
        tiles[i].x0 = lo * 256;
        tiles[i].x_len = (hi - lo) * 256;
      }
      out.max_x = std::max(out.max_x, (hi - lo) * 256);
    }
  }
  return out;
}

// Whether a list runs on the tensor cores (gemm_wstream.cu): independent items, block scales the tensor cores read as this
// kernel does, enough weights, and whole tiles that come out even.  That path puts one more launch in front of every run (5 us
// for one token, 9 for eight, under which the next weights fill the rings), issues a fifth of the instructions and, in runs
// long enough to meet the power cap, keeps its clock; it deals its tiles out longest first, where this kernel's contiguous runs
// (a change of projection costs it a conversion) leave some CTA with up to twice an even share; and it never splits a tile.
// From 128 MiB on it takes whatever it can deal out to 1.45 of an even share: us, this kernel / tensor cores in runs of 0.2 s,
// 223 MiB of 1024-column projections one token 49 / 42, eight 61 / 55, 1.8 GiB one token 358 / 292, four 405 / 317; a list with a longest share of 1.55
// to 2.3 of an even one took 1.1 to 1.4 times as long there.  Below, lists of tiles of four and more K steps on average,
// with 250 and more rows per token (the digits are made once per column, whatever the rows), that it deals out better than this
// kernel by as much as the constants say.  One, four and eight tokens, by the ratio of the shares:
//   1.42 to 2: 26 MiB 12.7 / 8.5, 13.5 / 9.4, 14.3 / 10.4; 28 MiB 12.8 / 9.1, 13.6 / 10.3, 14.2 / 12.1; 37 MiB 13.2 / 12.0, 14.1 / 12.7,
//              15.7 / 16.3; 47 MiB 15.5 / 14.2, 17.2 / 15.4, 18.5 / 16.2; 71 MiB 20.9 / 17.7, 22.7 / 19.1, 23.8 / 19.9; 74 MiB 21.1 / 17.5, 22.0 / 20.2,
//              25.0 / 24.0
//   1.32 to 1.42: 51 MiB 14.5 / 14.6, 15.2 / 15.7, 19.3 / 18.5; 93 MiB 23.5 / 20.7, 24.9 / 23.9, 29.0 / 26.7; 115 MiB 29.7 / 24.7, 34.9 / 26.2, 34.7 / 29.6
//   1.2 to 1.3: 84 MiB four tokens 21.6 / 22.6; 102 MiB 22.2 / 22.0, 23.6 / 24.8, 28.1 / 27.0
//   tiles of 2.3 steps on average: 25 MiB 9.7 / 9.7, 10.3 / 12.8, 11.4 / 16.5; 160 rows per token: 47 MiB seven tokens 16.8 / 20.0
constexpr int kTensorDigits = 8;  // three bits each, and more of them where a value needs them (gemm_wstream.cu)
constexpr size_t kTensorBytes = 128u << 20, kTensorBytesEven = 64u << 20, kTensorBytesLeast = 24u << 20;
constexpr double kTensorLongest = 1.45, kTensorBetterEven = 1.32, kTensorBetterLeast = 1.42;
constexpr int kTensorSteps = 4, kTensorRows = 250;

// The longest CTA's share of a list's K steps over an even one, two CTAs per SM and whole tiles in contiguous runs.
double contiguous_share(const q35b_gemv_item * items, int count) {
  long total = 0, tiles = 0, done = 0, share = 0, longest = 0;
  for (int i = 0; i < count; ++i) tiles += (items[i].weight->rows + kTileRows - 1) / kTileRows;
  for (int i = 0; i < count; ++i) total += static_cast<long>((items[i].weight->rows + kTileRows - 1) / kTileRows) * (items[i].weight->k / 256 + 1);
  const long grid = std::min<long>(2 * sm_count(), tiles);
  long c = 0;
  for (int i = 0; i < count; ++i) {
    const long cost = items[i].weight->k / 256 + 1;
    for (int t = 0; t < (items[i].weight->rows + kTileRows - 1) / kTileRows; ++t) {
      while (c + 1 < grid && (done + cost / 2) * grid >= (c + 1) * total) {
        ++c;
        share = 0;
      }
      longest = std::max(longest, share += cost);
      done += cost;
    }
  }
  return total > 0 ? static_cast<double>(longest) * grid / total : 1.0;
}

bool tensor_list(const q35b_gemv_item * items, int count, int m) {
  size_t bytes = 0;
  long steps = 0, tiles = 0, columns = 0;
  double weights = 0.0;
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    if (items[i].after != 0 || w->rows <= 0 || !w->has_maps || w->nan_scales || items[i].x_bf16 == nullptr || items[i].y_bf16 == nullptr) return false;
    bytes += w->codes_bytes + w->scales_bytes;
    tiles += (w->rows + kTileRows - 1) / kTileRows;
    steps += static_cast<long>((w->rows + kTileRows - 1) / kTileRows) * (w->k / 256);
    columns += w->k;
    weights += static_cast<double>(w->rows) * w->k;
  }
  if (bytes < kTensorBytesLeast) return false;
  const double longest = wbatch_longest_share(items, count);
  if (bytes >= kTensorBytes) return longest <= kTensorLongest;
  return steps >= kTensorSteps * tiles && weights >= static_cast<double>(kTensorRows) * m * columns && contiguous_share(items, count) >= longest * (bytes >= kTensorBytesEven ? kTensorBetterEven : kTensorBetterLeast);
}

// Whether a list runs as one launch per item in which the operand is made in shared memory (gemm_resident.cu): a chain, so
// that the launches follow one another as the items would.  us, one launch / one per item, MLP blocks [hidden, inter], weights from HBM.
//   Up to four tokens, unless all items are shorter than four K steps: the meeting inside one launch costs more than two launches do.
//     [2560, 9216] one token 25.8 / 16.7, four 27.3 / 22.9; [1024, 3584] 15.3 / 10.3, 16.0 / 12.1; [512, 1024] 9.9 / 9.5, 10.5 / 10.2; [1024, 768] 10.2 /
//     9.9, 11.1 / 10.5; not [512, 768] 9.2 / 9.7, 10.1 / 10.0, [256, 512] -, 8.9 / 9.9; and with three and four not what does not fit the GPU at once:
//     [5120, 5120] twice one 21.9 / 14.3, four 22.6 / 26.5; [5136, 8704] and [1024, 5120] two 23.4 / 19.6, four 25.1 / 24.9
//   Five and six: every row block makes the operand anew, so only short shares of it, and not beside short items alone.  [1024, 3584] 16.7 /
//     13.7, 16.9 / 14.5; [4096, 2048] 21.2 / 15.3, 21.6 / 16.0; not [768, 512] 10.5 / 11.5, 10.4 / 11.7, [512, 6400] 15.3 / 16.5, -, [2048, 6144] 22.5 / 20.0,
//     22.6 / 26.4.  From seven on the one launch is ahead: [2560, 9216] 28.9 / 29.2, [512, 1280] 11.5 / 11.7.
// A list of one item has nothing to wait for; what the one launch costs it is that CTAs share a tile of more than eight K steps
// and meet, or walk 1792 columns and more one after the other.  us, weights from HBM, [rows, K]:
//   one and two tokens: [300, 4096] 6.9 / 4.6, 7.1 / 4.6; [2560, 9216] 9.9 / 6.9, 10.1 / 7.4; [18432, 2560] 12.3 / 8.7, 12.4 / 9.3; not [9328, 8448] 15.9 / 17.9, -,
//     whose clusters do not fit the GPU at once
//   three and four: [2560, 4096] 8.2 / 6.1, 8.2 / 6.3; [2168, 5888] 8.9 / 6.7, -; not [3488, 6400] -, 9.6 / 10.6, [9432, 2816] -, 8.8 / 12.6
//   five and six: [1024, 3584] 7.6 / 6.6, 7.7 / 6.2; [2560, 2560] 7.3 / 7.3, 7.3 / 7.1; not [2224, 5120] 8.6 / 8.9, 8.6 / 9.2
//   up to eight K steps: [2048, 2048] one token 6.1 / 5.1, four 6.5 / 5.7; [4096, 2048] 6.0 / 5.0, 6.5 / 6.2; not [9000, 1792] two 6.1 / 6.4, [6144, 2048] four 6.6 /
//     7.2; never below 1792 columns: [3584, 1024] 4.3 / 4.8, 4.6 / 5.5, [7200, 1536] 5.3 / 5.5, 5.6 / 6.3
constexpr int kResidentTokens = 6, kResidentFewTokens = 4;
constexpr int kChainColumns = 1024, kChainColumnsMany = 2048;
constexpr double kChainMany = 2000.0;  // estimate (ns) up to which an item of a chain may make its operand for five and six tokens
constexpr int kSingleColumns = 1792, kSingleOutputs = 8192;
constexpr double kSingleFew = 1700.0, kSingleMany = 1300.0;

// can: it could, whatever is faster.
bool resident_chain(const q35b_gemv_item * items, const std::vector<int> & level, int m, bool * can) {
  *can = false;
  if (m > kResidentTokens) return false;
  int longest = 0;
  double most = 0.0;
  bool at_once = true;
  for (size_t i = 0; i < level.size(); ++i) {
    const q35b_weight * w = items[i].weight;
    bool held = false;
    const double ns = level[i] == static_cast<int>(i) && items[i].x_bf16 != nullptr && items[i].y_bf16 != nullptr ? decode_resident_chain_ns(w, m, &held) : 0.0;
    if (ns == 0.0) return false;
    longest = std::max(longest, w->k);
    most = std::max(most, ns);
    at_once = at_once && held;
  }
  *can = true;
  if (level.size() > 1) {
    if (m <= kResidentFewTokens) return longest >= kChainColumns && (at_once || m <= 2);
    return longest >= kChainColumnsMany && most <= kChainMany;
  }
  if (longest <= kWholeSteps * 256) return longest >= kSingleColumns && static_cast<long>(items[0].weight->rows) * m <= kSingleOutputs;
  return m <= 2 ? at_once : most <= (m <= kResidentFewTokens ? kSingleFew : kSingleMany);
}

}  // namespace

namespace {

// A list that runs as one launch per item owns a status word and the items' words.
int build_chain(const q35b_gemv_item * items, int count, int m, q35b_gemv_batch ** out) {
  auto * b = new q35b_gemv_batch();
  b->count = count;
  b->m = m;
  b->chain.assign(items, items + count);
  b->chained = true;
  for (int i = 0; i < count; ++i) b->bytes_per_run += items[i].weight->codes_bytes + items[i].weight->scales_bytes;
  b->counter_bytes = sizeof(unsigned int) * (4 + 2 * static_cast<size_t>(count));
  cudaError_t e = cudaMalloc(&b->dev_base, b->counter_bytes);
  if (e == cudaSuccess) e = cudaMemset(b->dev_base, 0, b->counter_bytes);
  if (e != cudaSuccess) {
    cudaFree(b->dev_base);
    delete b;
    return fail_cuda(e, "cudaMalloc(projection work list)");
  }
  b->status = static_cast<unsigned int *>(b->dev_base);
  b->chain_gave = b->status + 4;
  *out = b;
  return Q35B_OK;
}

// share_tiles: a caller's list, tiles of which several CTAs may share; chains: which may run as one launch per item.
int build_list(const q35b_gemv_item * items, int count, int m, bool share_tiles, bool chains, q35b_gemv_batch ** out) {
  if (items == nullptr || out == nullptr || count <= 0) return fail(Q35B_ERR_ARGUMENT, "Invalid NVFP4 projection work list.");
  if (m < 1 || m > 8) return fail(Q35B_ERR_SHAPE, "NVFP4 decode projection supports 1..8 tokens.");
  *out = nullptr;
  int max_k = 0;
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    if (w == nullptr) return fail(Q35B_ERR_ARGUMENT, "NVFP4 projection work list holds a null weight.");
    if ((w->k % 256) != 0) return fail(Q35B_ERR_SHAPE, "The streaming NVFP4 projection needs cols to be a multiple of 256.");
    if (w->negative_scales) return fail(Q35B_ERR_FORMAT, "The streaming NVFP4 projection needs unsigned E4M3 block scales.");
    if (w->gate_up && items[i].residual_bf16 != nullptr) {
      return fail(Q35B_ERR_ARGUMENT, "A gate/up projection takes no residual.");
    }
    if ((reinterpret_cast<uintptr_t>(items[i].x_bf16) & 15u) != 0) {
      return fail(Q35B_ERR_ARGUMENT, "Activations of the NVFP4 projection work list must be 16-byte aligned.");
    }
    if (items[i].after < 0 || items[i].after > i) {
      return fail(Q35B_ERR_ARGUMENT, "An NVFP4 projection work list item can only run after an earlier item of the list.");
    }
    max_k = std::max(max_k, w->k);
  }
  // only what the plan below takes too: a list whose activations do not fit it is refused whatever its size
  if (Plan fits_plan; share_tiles && tensor_list(items, count, m) && make_plan(m, max_k, &fits_plan)) {
    WBatch * t = nullptr;
    if (const int st = wbatch_build(items, count, m, kTensorDigits, true, &t)) return st;
    auto * b = new q35b_gemv_batch();
    b->count = count;
    b->m = m;
    b->tensor = t;
    b->bytes_per_run = wbatch_bytes(t);
    *out = b;
    return Q35B_OK;
  }
  std::vector<int> level(count, 0);
  for (int i = 0; i < count; ++i) {
    if (items[i].after > 0) level[i] = level[items[i].after - 1] + 1;
  }
  bool can = false;
  if (Plan fits_plan; share_tiles && resident_chain(items, level, m, &can) && chains && make_plan(m, max_k, &fits_plan)) return build_chain(items, count, m, out);
  auto * b = new q35b_gemv_batch();
  b->count = count;
  b->m = m;
  if (cudaGetDevice(&b->device) != cudaSuccess) {
    delete b;
    return fail_cuda(cudaGetLastError(), "cudaGetDevice");
  }
  bool fits = false;
  if (const cudaError_t pe = plan_for_device(m, max_k, share_tiles, &b->plan, &fits); pe != cudaSuccess) {
    delete b;
    return fail_cuda(pe, "planning the projection work list");
  }
  if (!fits) {
    delete b;
    return fail(Q35B_ERR_SHAPE, "Activations of the NVFP4 projection work list do not fit in shared memory.");
  }

  std::vector<GemvTile> all;
  std::vector<GemvItem> h_items(count);
  long total_steps = 0;
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    GemvItem & it = h_items[i];
    if (const int st = make_code_map(&it.tmap, w->codes, std::max(w->rows, 1), w->k / 2, kTileRows)) {
      delete b;
      return st;
    }
    it.scales_tiled = w->scales_tiled;
    it.x = static_cast<const __nv_bfloat16 *>(items[i].x_bf16);
    it.y = static_cast<__nv_bfloat16 *>(items[i].y_bf16);
    it.rows = w->rows;
    it.k = w->k;
    it.k_steps = w->k / 256;
    it.s2 = w->s2;
    bool signal = false;
    for (int j = i + 1; j < count; ++j) signal = signal || items[j].after - 1 == i;
    for (int rb = 0; rb < (w->rows + kTileRows - 1) / kTileRows; ++rb) {
      GemvTile tl = {};
      tl.item = i;
      tl.row_block = rb;
      tl.k = w->k;
      tl.k_steps = it.k_steps;
      tl.x_len = w->k;
      tl.rows = w->rows;
      tl.s2 = w->s2;
      tl.scales = w->scales_tiled + static_cast<size_t>(rb) * it.k_steps * kScaleBytes;
      tl.x = it.x;
      tl.y = it.y;
      tl.residual = static_cast<const __nv_bfloat16 *>(items[i].residual_bf16);
      tl.s2_up = w->s2_up;
      tl.flags = (w->gate_up ? kFlagGateUp : 0) | (signal ? kFlagSignal : 0);
      tl.wait_item = items[i].after - 1;
      tl.parts = 1;
      if (tl.wait_item >= 0) {
        const q35b_weight * dep = items[tl.wait_item].weight;
        tl.wait_count = static_cast<unsigned int>((dep->rows + kTileRows - 1) / kTileRows) * kRowGroups;
        b->has_dependencies = true;
      }
      all.push_back(tl);
      total_steps += it.k_steps;
    }
    b->bytes_per_run += w->codes_bytes + w->scales_bytes;
  }
  const int max_level = *std::max_element(level.begin(), level.end());
  const int most = share_tiles ? static_cast<int>(std::min<long>(total_steps, 1 << 20)) : static_cast<int>(all.size());
  auto grid_for = [&](int ksplit) { return std::max(1, std::min(sm_count() * ctas_per_sm(ksplit), most)); };
  int grid = grid_for(b->plan.ksplit);
  Assignment todo = assign_tiles(all, level, max_level, grid, m, share_tiles);
  if (share_tiles && todo.splits == 0) {
    // whole tiles only: no CTA without one
    share_tiles = false;
    grid = std::max(1, std::min(grid, static_cast<int>(all.size())));
    todo = assign_tiles(all, level, max_level, grid, m, false);
  }
  if (share_tiles) {
    // Parts of tiles need only their columns of the activations, so a list may fit the two-CTAs-per-SM shape, a second
    // activation buffer or a deeper ring although its longest projection would not.
    for (int ks = 1; ks <= b->plan.ksplit; ++ks) {
      const int g = grid_for(ks);
      Assignment a = ks == b->plan.ksplit ? todo : assign_tiles(all, level, max_level, g, m, true);
      Plan p;
      bool ok = false;
      if (const cudaError_t pe = plan_for_device(m, std::max(a.max_x, 256), true, &p, &ok); pe != cudaSuccess) {
        delete b;
        return fail_cuda(pe, "planning the projection work list");
      }
      if (ok && p.ksplit == ks) {
        b->plan = p;
        grid = g;
        todo = std::move(a);
        break;
      }
    }
  }
  std::vector<GemvTile> h_tiles;
  std::vector<int> h_begin(grid + 1, 0);
  for (int c = 0; c < grid; ++c) {
    h_begin[c] = static_cast<int>(h_tiles.size());
    for (const GemvTile & tl : todo.per_cta[c]) h_tiles.push_back(tl);
  }
  h_begin[grid] = static_cast<int>(h_tiles.size());
  b->grid = grid;
  b->shared = todo.splits > 0;

  const size_t o_tiles = sizeof(GemvItem) * count;
  const size_t o_begin = (o_tiles + sizeof(GemvTile) * h_tiles.size() + 15) / 16 * 16;
  const size_t o_status = (o_begin + sizeof(int) * (grid + 1) + 15) / 16 * 16;
  const size_t o_done = o_status + 16;
  const size_t o_arrivals = o_done + sizeof(unsigned long long) * (count + 1);  // + the finished-CTA count
  const size_t o_gave = o_arrivals + sizeof(unsigned int) * kRowGroups * todo.splits;
  const size_t o_partials = (o_gave + sizeof(unsigned int) * 2 * count + 127) / 128 * 128;
  const size_t part_bytes = sizeof(float) * kRowGroups * 32 * 4;  // four sums per lane, in either MMA mapping
  const size_t total = o_partials + part_bytes * todo.slots;
  cudaError_t e = cudaMalloc(&b->dev_base, total);
  if (e != cudaSuccess) {
    delete b;
    return fail_cuda(e, "cudaMalloc(projection work list)");
  }
  auto * base = static_cast<uint8_t *>(b->dev_base);
  b->items = reinterpret_cast<GemvItem *>(base);
  b->tiles = reinterpret_cast<GemvTile *>(base + o_tiles);
  b->cta_begin = reinterpret_cast<int *>(base + o_begin);
  b->status = reinterpret_cast<unsigned int *>(base + o_status);
  b->item_done = reinterpret_cast<unsigned long long *>(base + o_done);
  b->arrivals = reinterpret_cast<unsigned int *>(base + o_arrivals);
  b->chain_gave = reinterpret_cast<unsigned int *>(base + o_gave);
  b->partials = reinterpret_cast<float *>(base + o_partials);
  b->counter_bytes = o_partials - o_status;
  e = cudaMemcpy(b->items, h_items.data(), sizeof(GemvItem) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->tiles, h_tiles.data(), sizeof(GemvTile) * h_tiles.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->cta_begin, h_begin.data(), sizeof(int) * (grid + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(b->status, 0, b->counter_bytes);
  if (e != cudaSuccess) {
    cudaFree(b->dev_base);
    delete b;
    return fail_cuda(e, "uploading the projection work list");
  }
  if (can) b->chain.assign(items, items + count);
  *out = b;
  return Q35B_OK;
}

}  // namespace

int gemv_batch_build(const q35b_gemv_item * items, int count, int m, bool share_tiles, q35b_gemv_batch ** out) {
  return build_list(items, count, m, share_tiles, true, out);
}

int gemv_batch_build_tensor(const q35b_gemv_item * items, int count, int m, int digits, q35b_gemv_batch ** out) {
  if (out == nullptr) return fail(Q35B_ERR_ARGUMENT, "Invalid NVFP4 projection work list.");
  *out = nullptr;
  WBatch * t = nullptr;
  if (const int st = wbatch_build(items, count, m, digits, false, &t)) return st;
  auto * b = new q35b_gemv_batch();
  b->count = count;
  b->m = m;
  b->tensor = t;
  b->bytes_per_run = wbatch_bytes(t);
  *out = b;
  return Q35B_OK;
}

int gemv_batch_launch(const q35b_gemv_batch * b, const void * x_override, void * y_override, cudaStream_t s) {
  if (b == nullptr) return fail(Q35B_ERR_ARGUMENT, "Null NVFP4 projection work list.");
  if (b->tensor != nullptr) return wbatch_launch(b->tensor, s);
  if (b->one_launch != nullptr && b->wait_extra != 0) return gemv_batch_launch(b->one_launch, x_override, y_override, s);
  if (b->chained) {
    for (size_t i = 0; i < b->chain.size(); ++i) {
      const q35b_gemv_item & it = b->chain[i];
      const ResidentChain neighbours = {i + 1 < b->chain.size() ? b->chain[i + 1].weight : nullptr, b->chain_gave + 2 * i,
                                        i > 0 ? b->chain_gave + 2 * (i - 1) : nullptr, static_cast<int>(i) == b->chain_absent};
      if (const int st = launch_decode_resident(it.weight, it.x_bf16, b->m, it.y_bf16, it.residual_bf16, &neighbours, b->status, b->wait_limit, s)) return st;
    }
    return Q35B_OK;
  }
  const auto * xo = static_cast<const __nv_bfloat16 *>(x_override);
  auto * yo = static_cast<__nv_bfloat16 *>(y_override);
  const int counted = b->has_dependencies ? b->count : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(b->grid));
  cfg.blockDim = dim3(static_cast<unsigned>(cta_threads(b->plan.ksplit)));
  cfg.dynamicSmemBytes = static_cast<size_t>(b->plan.smem_bytes);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const GemvItem * d_items = b->items;
  const GemvTile * d_tiles = b->tiles;
  const int * d_begin = b->cta_begin;
  const Plan & pl = b->plan;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, stream_kernel(b->m, pl.ksplit, b->shared), d_items,
                                            d_tiles, d_begin, b->m, xo, yo, pl.stages, pl.x_buf_halfs, pl.xs_buf_floats,
                                            pl.x_bufs, b->item_done, counted, b->partials, b->arrivals, b->status, b->wait_limit,
                                            b->wait_extra);
  count_launch();
  Q35B_CUDA_TRY(le, "gemv_w4a16_stream_kernel launch");
  return Q35B_OK;
}

void gemv_batch_free(q35b_gemv_batch * b) {
  if (b == nullptr) return;
  wbatch_free(b->tensor);
  gemv_batch_free(b->one_launch);
  if (b->dev_base != nullptr) cudaFree(b->dev_base);
  delete b;
}

int gemv_batch_read_status(const q35b_gemv_batch * b, unsigned int * out) {
  if (b == nullptr || out == nullptr) return fail(Q35B_ERR_ARGUMENT, "Null NVFP4 projection work list.");
  if (b->tensor != nullptr) return wbatch_status(b->tensor, out);
  Q35B_CUDA_TRY(cudaMemcpy(out, b->status, sizeof(unsigned int), cudaMemcpyDeviceToHost), "cudaMemcpy(work list status)");
  if (*out == 0u && b->one_launch != nullptr) return gemv_batch_read_status(b->one_launch, out);
  return Q35B_OK;
}

size_t gemv_batch_bytes(const q35b_gemv_batch * b) { return b ? b->bytes_per_run : 0; }

int gemv_batch_debug_wait(q35b_gemv_batch * b, unsigned int wait_limit, unsigned int extra_completions) {
  if (b == nullptr || wait_limit == 0) return fail(Q35B_ERR_ARGUMENT, "Invalid NVFP4 projection work list.");
  if (b->tensor != nullptr) return wbatch_debug_wait(b->tensor, wait_limit);
  if (b->chained && extra_completions != 0 && b->one_launch == nullptr) {
    if (const int st = build_list(b->chain.data(), b->count, b->m, true, false, &b->one_launch)) return st;
  }
  if (b->one_launch != nullptr) {
    if (const int st = gemv_batch_debug_wait(b->one_launch, wait_limit, extra_completions)) return st;
  }
  b->wait_limit = wait_limit;
  b->wait_extra = extra_completions;
  // only the recorded code: every run leaves its counters at zero, also one that gave up
  Q35B_CUDA_TRY(cudaMemset(b->status, 0, sizeof(unsigned int)), "cudaMemset(work list status)");
  return Q35B_OK;
}

int gemv_batch_debug_absent(q35b_gemv_batch * b, int item) {
  if (b == nullptr || item < -1 || item >= b->count) return fail(Q35B_ERR_ARGUMENT, "Invalid NVFP4 projection work list.");
  if (!b->chained) return fail(Q35B_ERR_SHAPE, "The NVFP4 projection work list is not a chain of launches.");
  b->chain_absent = item;
  return Q35B_OK;
}

int gemv_batch_debug_chain(q35b_gemv_batch * b) {
  if (b == nullptr || b->chain.empty()) return fail(Q35B_ERR_SHAPE, "The NVFP4 projection work list does not fit a chain of launches.");
  b->chained = true;
  return Q35B_OK;
}

}  // namespace q35b
