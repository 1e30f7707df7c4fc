// Weight-streaming block-scaled FP4 projection for few tokens (1..128 operand columns) on sm_100a.
//
// The prefill GEMMs put the tokens on the 128 rows of the tensor-core tile and stream weights as the narrow
// operand; with few tokens that wastes the tile and leaves most SMs without work.  Here the roles are swapped:
//
//   UMMA A (128 rows)  = one 128-row block of the WEIGHT, streamed once from HBM: codes in checkpoint order
//                        through the weight's 128-row TMA map, scale factors as the weight's 512-byte scale tiles;
//   UMMA B (N columns) = the activation operand, N = 16..128 rows of NVFP4 codes (re-read from L2 by every tile);
//   D [128, N] fp32    = in TMEM; a lane is a weight row, a column is an operand row.
//
// One persistent CTA per SM walks a list of (projection, row block) tiles, as the streaming decode kernel does, with
// a TMA-fed shared-memory ring (weights and activations have separate producer threads: weights are constant and
// start streaming before the previous kernel of the stream has finished, activations wait for it), one MMA thread
// issuing tcgen05.mma kind::mxf4nvf4.block_scale per 64 columns of K, two TMEM accumulators so that the epilogue of
// a tile runs under the MMAs of the next, and epilogue warps that turn accumulator lanes into BF16 outputs
// y[token, row].
//
// Decode (W4A16, 1..8 tokens): every token enters as `digits` operand rows, the octal digits of its BF16 activations
// (split_digits_kernel below), and the epilogue adds the digits' accumulator columns.  Eight digits hold all eight bits of a
// value down to about 2^-16 of its block's largest one; smaller values need up to six more, the deep digits.  They are rows
// of a second operand that is loaded and multiplied only in the K steps where some value has them (one in 60,000 normal
// values does), with sums of their own; with one token they fit into the padding of the first.  Replaces nvfp4_row_dot / matvec_nvfp4_bf16
// (src/kernels/cuda/decode_layers.cuh:200-284) with the FP4 decode done by the tensor core instead of by conversion
// instructions: a fifth of gemv_stream.cu's instructions, so a long run of steps does not meet the power cap.
//
// Every wait is bounded; an expired wait records a code in *status and the role stops.  The CTA then waits (again with a
// limit) for the copies and MMAs that it has under way, and frees its TMEM.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "digits.cuh"
#include "engine.h"
#include "nvfp4_codec.cuh"

namespace q35b {
namespace {

constexpr int kRows = 128;               // weight rows per tile (UMMA M)
constexpr int kStepBytes = 128;          // 256 FP4 columns of K per ring stage
constexpr int kMmaPerStage = 4;          // K = 64 per MMA
constexpr int kSfChunk = 512;            // scale factors of 128 rows x 64 columns
constexpr int kABytes = kRows * kStepBytes;          // 16 KB
constexpr int kSfBytes = kMmaPerStage * kSfChunk;    // 2 KB (weights, and activations: at most 128 operand rows)
constexpr int kMaxCols = 128;
constexpr int kMaxStages = 8;
// Warp 0 weight producer, 1 MMA, 2 activation producer, the others epilogue: two per quarter of the TMEM lanes, which take turns
// at the tokens; three from seven tokens on in lists of short tiles, which are over before two have the sums out.  us, two /
// three, lists of 0.3 GB of [4096, K], eight tokens: K = 768 84.0 / 78.8, 1024 70.1 / 67.6, 1536 60.0 / 60.4, 2048 58.4 / 59.0, 2560 58.2 / 58.4
// (seven the same); 0.8B-class step (5.1 K steps per tile) seven tokens 52.1 / 51.3, eight 54.8 / 53.4, six 48.9 / 49.1, one 41.6 / 44.2;
// 4B-class eight 339.7 / 344.9.  Four per quarter: 0.8B-class eight tokens as with three, but no CTA of the digits' kernel fits beside them.
constexpr int kEpilogueWarps = 8, kEpilogueWarpsWide = 12, kWideTokens = 7, kWideSteps = 6;
constexpr int threads_for(int epilogue_warps) { return (3 + epilogue_warps) * 32; }
// Registers: of 112 per thread the wide CTA leaves room for one of split_digits_kernel's.
constexpr int kLaunchBound = 512;
constexpr int kTmemCols = 512;           // two accumulator buffers ...
constexpr int kAccBufCols = 224;         // partial accumulators of the operand rows, then those of the deep digits' rows
constexpr int kSfaCol = 2 * kAccBufCols;   // ... and two sets of scale-factor columns (A 16 + B 16 each), used by stages in turn,
constexpr int kSfbCol = kSfaCol + 16;      // so that the copies of one stage do not wait for the MMAs of the one before
constexpr int kSfSetCols = 32;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr uint32_t kDrainLimit = 1u << 22;  // polls for what is still under way after an expired wait, however short that one's limit was
constexpr int kSmemBudget = 220 * 1024;   // dynamic part; the staged tile descriptors are static shared memory

enum StatusCode : unsigned { kWeightWait = 41, kActWait = 42, kMmaWait = 43, kMmaDrainWait = 44, kEpilogueWait = 45 };
enum Epilogue : int { kEpiPlain = 0, kEpiGateUp = 1 };

// One projection of the list, in device memory; the tensor maps are read by the TMA unit from there.
struct alignas(128) WItem {
  CUtensorMap tmap_w;            // weight codes [rows, K/2], box 128 rows x 128 bytes, 128B swizzle
  const uint8_t * w_scales;      // weight scale tiles
  const uint8_t * x_ops;         // the operand, one run of bytes per K step: codes as they lie in shared memory (n_cols rows of
                                 // 128 bytes, 128B swizzle) and four scale tiles, then the same of the deep digits' rows
  const uint32_t * x_deep;       // NULL (no deep digits), or for every 32 K steps a word per token (eight): the steps where it has them
  const float * x_g;             // the operand's scale, one per token (NaN or infinity: the token has such values, see infinite_dot)
  const uint8_t * w_codes;       // for such tokens: weight codes and the activations themselves
  const __nv_bfloat16 * x;
  __nv_bfloat16 * y;             // [tokens, ldy]
  const __nv_bfloat16 * residual;  // NULL or [tokens, ldr]
  int rows;                      // weight rows
  int k_steps;                   // K / 256
  int n_cols;                    // operand rows padded to a multiple of 16 (UMMA N)
  int deep_cols;                 // the same of the deep digits' rows; 0: there are none, or they are
  int deep_rows;                 // rows of the operand itself, from this one on
  int tokens;
  int digits;                    // operand rows per token
  int ldy, ldr;
  float s2, s2_up;
  int epilogue;
};

struct alignas(8) WTile {
  int item;
  int row_block;
};

// Everything the roles need to know about one tile, staged in shared memory at kernel start so that no role chases
// pointers through global memory at a tile boundary (a 128-row x 1024-column tile lasts under two microseconds).
struct alignas(16) STile {
  const CUtensorMap * tmap_w;
  const uint8_t * w_scales;      // scale tiles of this row block
  const uint8_t * x_ops;
  const uint32_t * x_deep;
  const float * x_g;
  const WItem * item;
  __nv_bfloat16 * y;
  const __nv_bfloat16 * residual;
  int row_block, rows, k_steps, n_cols, deep_cols, deep_rows, tokens, digits, ldy, ldr, epilogue;
  float s2, s2_up;
};
constexpr int kMaxTilesInSmem = 40;

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
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "elect.sync _|p, 0xffffffff;\n\t"
    "selp.u32 %0, 1, 0, p;\n\t}"
    : "=r"(pred));
  return pred != 0;
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
// K-major operand tile, 128B swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t desc_k_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// Scale-factor slab for tcgen05.cp: no swizzle, 8 rows of 16 bytes per core matrix, core matrices 128 bytes apart.
__device__ __forceinline__ uint64_t desc_sf(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(128 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}
// With few operand columns an MMA is far shorter than the tensor pipe's latency, and four MMAs per stage that all
// accumulate into the same TMEM columns run one after the other at that latency (measured: 1500 cycles per stage,
// against 900 for the stage's bytes to arrive from HBM).  So the MMAs of a stage go to different partial
// accumulators (as many as fit beside each other in a buffer), each of which then sees one MMA per stage, and the
// epilogue adds the partials.
__device__ __forceinline__ int partial_accumulators(int n_cols, int deep_cols) {
  return 4 * n_cols + deep_cols <= kAccBufCols ? 4 : (2 * n_cols + deep_cols <= kAccBufCols ? 2 : 1);
}
// ... and of the deep digits' rows behind them
__device__ __forceinline__ int deep_accumulators(int used, int deep_cols) { return used + 2 * deep_cols <= kAccBufCols ? 2 : 1; }

// kind::mxf4nvf4: E2M1 x E2M1, K-major, UE4M3 scales, M = 128, N = n_cols.
__device__ __forceinline__ uint32_t instr_desc(int n_cols) {
  uint32_t d = 0;
  d |= 1u << 7;
  d |= 1u << 10;
  d |= static_cast<uint32_t>(n_cols >> 3) << 17;
  d |= static_cast<uint32_t>(kRows >> 4) << 24;
  return d;
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t tmem_sfa,
                                     uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "setp.ne.b32 p, %4, 0;\n\t"
    "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
    : "memory");
}
__device__ __forceinline__ void utccp_sf(uint32_t tmem_dst, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Waits for the loads before it.  The registers are operands, or the compiler might use them before the wait.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[4][8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]), "+r"(r[0][4]), "+r"(r[0][5]), "+r"(r[0][6]), "+r"(r[0][7]),
                 "+r"(r[1][0]), "+r"(r[1][1]), "+r"(r[1][2]), "+r"(r[1][3]), "+r"(r[1][4]), "+r"(r[1][5]), "+r"(r[1][6]), "+r"(r[1][7]),
                 "+r"(r[2][0]), "+r"(r[2][1]), "+r"(r[2][2]), "+r"(r[2][3]), "+r"(r[2][4]), "+r"(r[2][5]), "+r"(r[2][6]), "+r"(r[2][7]),
                 "+r"(r[3][0]), "+r"(r[3][1]), "+r"(r[3][2]), "+r"(r[3][3]), "+r"(r[3][4]), "+r"(r[3][5]), "+r"(r[3][6]), "+r"(r[3][7])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// CTA b walks tiles[cta_begin[b] .. cta_begin[b + 1]).
__global__ void __launch_bounds__(kLaunchBound, 1)
gemm_wstream_kernel(const WItem * __restrict__ items, const WTile * __restrict__ tiles, const int * __restrict__ cta_begin,
                    int stages, int b_slot_bytes, int deep_bytes, unsigned int * status, uint32_t wait_limit) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t * smem_a = smem;
  uint8_t * smem_b = smem_a + stages * kABytes;
  uint8_t * smem_sfa = smem_b + stages * b_slot_bytes;     // a slot of smem_b holds a step's operand codes and scale tiles,
                                                           // its last deep_bytes those of the deep digits
  uint64_t * bars = reinterpret_cast<uint64_t *>(smem_sfa + stages * kSfBytes);
  uint64_t * full = bars;                           // [stages]: both producers' bytes have landed
  uint64_t * empty = bars + kMaxStages;             // [stages]: the MMAs that read the stage have retired
  uint64_t * tmem_full = bars + 2 * kMaxStages;     // [2]: accumulator complete
  uint64_t * tmem_empty = tmem_full + 2;            // [2]: the epilogue warps have read the accumulator out
  uint64_t * mma_done = tmem_empty + 2;             // after an expired wait: every MMA issued has retired
  uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
  __shared__ STile stile[kMaxTilesInSmem];
  __shared__ uint32_t stage_deep[kMaxStages];              // the stage's step has deep digits; set before its bytes are asked for

  __shared__ uint32_t gave_up;                             // some role of this CTA has
  __shared__ uint32_t issued[2];                           // K steps whose weights, and whose activations, were asked for

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tile_begin = cta_begin[blockIdx.x], n_tiles = cta_begin[blockIdx.x + 1] - tile_begin;
  auto describe = [&](int ti, STile & d) {
    const WTile t = tiles[tile_begin + ti];
    const int rb = t.row_block;
    const WItem * it = items + t.item;
    d.item = it;
    d.tmap_w = &it->tmap_w;
    d.k_steps = it->k_steps;
    d.w_scales = it->w_scales + static_cast<size_t>(rb) * d.k_steps * kSfBytes;
    d.x_ops = it->x_ops;
    d.x_deep = it->x_deep;
    d.x_g = it->x_g;
    d.y = it->y;
    d.residual = it->residual;
    d.row_block = rb;
    d.rows = it->rows;
    d.n_cols = it->n_cols;
    d.deep_cols = it->deep_cols;
    d.deep_rows = it->deep_rows;
    d.tokens = it->tokens;
    d.digits = it->digits;
    d.ldy = it->ldy;
    d.ldr = it->ldr;
    d.epilogue = it->epilogue;
    d.s2 = it->s2;
    d.s2_up = it->s2_up;
  };
  // tile descriptors are constant for the life of a work list (and of a launch): read them before anything else
  for (int ti = threadIdx.x; ti < min(n_tiles, kMaxTilesInSmem); ti += blockDim.x) {
    describe(ti, stile[ti]);
    if (ti == 0 || tiles[tile_begin + ti - 1].item != tiles[tile_begin + ti].item) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(stile[ti].tmap_w) : "memory");
    }
  }
  // tiles beyond the staged ones (a CTA with a very long list) are described on the fly
  auto tile_at = [&](int ti, STile & spill) -> const STile * {
    if (ti < kMaxTilesInSmem) return stile + ti;
    describe(ti, spill);
    return &spill;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(smem_u32(full + i), 2);
      mbar_init(smem_u32(empty + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(tmem_full + i), 1);
      mbar_init(smem_u32(tmem_empty + i), blockDim.x / 32 - 3);
    }
    mbar_init(smem_u32(mma_done), 1);
    gave_up = 0;
    issued[0] = issued[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // The next kernel of the stream may be scheduled from here on; this one touches nothing an earlier kernel may
  // still be writing (activations, scales, outputs) before its own griddepcontrol.wait below.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------ weight producer (constant data: no wait)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0, steps = 0;
      bool ok = true;
      STile spill;
      for (int ti = 0; ti < n_tiles && ok; ++ti) {
        const STile * it = tile_at(ti, spill);
        const int k_steps = it->k_steps, rb = it->row_block;
        const uint8_t * sf = it->w_scales;
        for (int ks = 0; ks < k_steps; ++ks) {
          // the first turn of the ring was free; from here on it depends on the activations, which an earlier kernel may take
          // any time to deliver, and a bounded wait must not
          if (steps == static_cast<uint32_t>(stages)) asm volatile("griddepcontrol.wait;" ::: "memory");
          if (!mbar_wait(smem_u32(empty + stage), phase ^ 1, wait_limit)) {
            atomicExch(status, kWeightWait);
            gave_up = 1;
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(full + stage);
          mbar_expect_tx(bar, kABytes + kSfBytes);
          tma_load_2d(smem_u32(smem_a + stage * kABytes), it->tmap_w, bar, ks * kStepBytes, rb * kRows);
          bulk_load(smem_u32(smem_sfa + stage * kSfBytes), sf + static_cast<size_t>(ks) * kSfBytes, kSfBytes, bar);
          issued[0] = ++steps;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ activation producer
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int stage = 0;
    uint32_t phase = 0, steps = 0;
    bool ok = true;
    STile spill;
    const uint32_t * deep_of = nullptr;
    int deep_block = 0;
    uint32_t masks = 0;  // of token lane & 7, steps 128 * deep_block + 32 * (lane >> 3) and on; read once per projection
    for (int ti = 0; ti < n_tiles && ok; ++ti) {
      const STile * it = tile_at(ti, spill);
      const int k_steps = it->k_steps;
      for (int base = 0; base < k_steps && ok; base += 32) {
        if (deep_bytes > 0 && (it->x_deep != deep_of || base >> 7 != deep_block)) {
          deep_of = it->x_deep;
          deep_block = base >> 7;
          const int word = 4 * deep_block + (lane >> 3);
          masks = 32 * word < k_steps ? __ldcg(deep_of + 8 * word + (lane & 7)) : 0u;
        }
        const uint32_t deep = __reduce_or_sync(0xffffffffu, lane >> 3 == (base >> 5 & 3) ? masks : 0u);
        const uint8_t * ops = it->x_ops + static_cast<size_t>(base) * b_slot_bytes;
        if (elect_one()) {
          for (int i = 0; i < min(k_steps - base, 32); ++i) {
            if (!mbar_wait(smem_u32(empty + stage), phase ^ 1, wait_limit)) {
              atomicExch(status, kActWait);
              gave_up = 1;
              ok = false;
              break;
            }
            const uint32_t bar = smem_u32(full + stage), has = deep >> i & 1u;
            const uint32_t bytes = static_cast<uint32_t>(has != 0u ? b_slot_bytes : b_slot_bytes - deep_bytes);
            stage_deep[stage] = has;
            mbar_expect_tx(bar, bytes);
            bulk_load(smem_u32(smem_b + stage * b_slot_bytes), ops + static_cast<size_t>(i) * b_slot_bytes, bytes, bar);
            issued[1] = ++steps;
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
        // the elected lane is the same one every time and keeps the ring's position; whether it gave up, all have to know
        ok = __all_sync(0xffffffffu, ok);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // Per stage: eight scale-factor copies into one of two TMEM column sets, then four MMAs; a stage's turn takes about 500
    // cycles, its bytes 800 to come from HBM.  The issuing threads are chosen with elect.sync: by a test of the lane number
    // the same code took 600 ns per stage (0.8B-class step of one token 73 us instead of 44).
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait for activations before they can be there
      int stage = 0;
      uint32_t phase = 0, sf_turn = 0;
      bool ok = true;
      STile spill;
      for (int ti = 0; ti < n_tiles && ok; ++ti) {
        const STile * it = tile_at(ti, spill);
        const int k_steps = it->k_steps;
        const uint32_t idesc = instr_desc(it->n_cols), idesc_deep = instr_desc(it->deep_cols);
        uint32_t deep_seen = 0;
        const uint32_t ab = ti & 1;
        if (!mbar_wait(smem_u32(tmem_empty + ab), ((ti >> 1) & 1) ^ 1, wait_limit)) {
          atomicExch(status, kMmaDrainWait);
          gave_up = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + ab * kAccBufCols;
        const int n_cols = it->n_cols, deep_cols = it->deep_cols, parts = partial_accumulators(n_cols, deep_cols);
        const int deep_parts = deep_accumulators(parts * n_cols, deep_cols);
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!mbar_wait(smem_u32(full + stage), phase, wait_limit)) {
            atomicExch(status, kMmaWait);
            gave_up = 1;
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t a_desc = desc_k_sw128(smem_u32(smem_a + stage * kABytes));
          const uint64_t b_desc = desc_k_sw128(smem_u32(smem_b + stage * b_slot_bytes));
          const uint64_t sfa_desc = desc_sf(smem_u32(smem_sfa + stage * kSfBytes));
          const uint64_t sfb_desc = desc_sf(smem_u32(smem_b + (stage + 1) * b_slot_bytes - deep_bytes - kSfBytes));
          const uint32_t sf_set = tmem_base + (sf_turn ^= 1u) * kSfSetCols;
#pragma unroll
          for (int j = 0; j < kMmaPerStage; ++j) {
            utccp_sf(sf_set + kSfaCol + j * 4, sfa_desc + j * (kSfChunk >> 4));
            utccp_sf(sf_set + kSfbCol + j * 4, sfb_desc + j * (kSfChunk >> 4));
          }
#pragma unroll
          for (int j = 0; j < kMmaPerStage; ++j) {
            umma(acc + (j & (parts - 1)) * n_cols, a_desc + j * 2, b_desc + j * 2, idesc, sf_set + kSfaCol + j * 4,
                 sf_set + kSfbCol + j * 4, (ks * kMmaPerStage + j) >= parts ? 1u : 0u);
          }
          if (stage_deep[stage] != 0u) {
            // The copies overwrite the scale columns of the MMAs above, behind which they stand in the tensor pipe.
            const uint64_t bd_desc = desc_k_sw128(smem_u32(smem_b + (stage + 1) * b_slot_bytes - deep_bytes));
            const uint64_t sfd_desc = desc_sf(smem_u32(smem_b + (stage + 1) * b_slot_bytes - kSfBytes));
#pragma unroll
            for (int j = 0; j < kMmaPerStage; ++j) utccp_sf(sf_set + kSfbCol + j * 4, sfd_desc + j * (kSfChunk >> 4));
#pragma unroll
            for (int j = 0; j < kMmaPerStage; ++j) {
              umma(acc + parts * n_cols + (j & (deep_parts - 1)) * deep_cols, a_desc + j * 2, bd_desc + j * 2, idesc_deep, sf_set + kSfaCol + j * 4,
                   sf_set + kSfbCol + j * 4, deep_seen != 0u || j >= deep_parts ? 1u : 0u);
            }
            deep_seen = 1;
          }
          umma_commit(smem_u32(empty + stage));
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit(smem_u32(tmem_full + ab));
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: lane = weight row, column = operand row
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int quarter = warp & 3, first_token = (warp - 3) >> 2, turns = (static_cast<int>(blockDim.x) - 96) >> 7;
    const int row_in_tile = quarter * 32 + lane;
    STile spill;
    const float * scales_of = nullptr;
    float scales = 0.0f;      // of token `lane`, read once per projection and before the wait (one load per token cost 1 us a tile)
    uint32_t deep_tokens = 0; // tokens with deep digits; the sums of the others have nothing in those rows
    for (int ti = 0; ti < n_tiles; ++ti) {
      const STile * it = tile_at(ti, spill);
      const uint32_t ab = ti & 1;
      if (it->x_g != scales_of) {
        scales_of = it->x_g;
        uint32_t any = 0;
        if (lane < it->tokens) {
          scales = __ldcg(scales_of + lane);
          if (it->x_deep != nullptr) {
            for (int w = 0; 32 * w < it->k_steps; ++w) any |= __ldcg(it->x_deep + 8 * w + lane);
          }
        }
        deep_tokens = __ballot_sync(0xffffffffu, any != 0u);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(tmem_full + ab), (ti >> 1) & 1, wait_limit))) {  // the whole warp goes on, or none of it
        if (lane == 0) {
          atomicExch(status, kEpilogueWait);
          gave_up = 1;
        }
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int rows = it->rows, tokens = it->tokens, digits = it->digits, n_cols = it->n_cols, deep_cols = it->deep_cols;
      const int row = it->row_block * kRows + row_in_tile;
      const bool gate_up = it->epilogue == kEpiGateUp;
      const float s2 = it->s2, s2_up = it->s2_up;
      const uint32_t taddr = tmem_base + ab * kAccBufCols + (static_cast<uint32_t>(quarter * 32) << 16);
      const int parts = partial_accumulators(n_cols, deep_cols);
      // the deep digits' sums: columns among the others', or accumulators of their own behind them
      const uint32_t deep_addr = taddr + (deep_cols > 0 ? parts * n_cols : it->deep_rows);
      const int deep_stride = deep_cols > 0 ? deep_cols : n_cols, deep_parts = deep_cols > 0 ? deep_accumulators(parts * n_cols, deep_cols) : parts;
      // One token at a time, in a compact loop: a small part of a tile's time as long as its code stays resident (with all
      // columns unrolled a 0.8B-class step of eight tokens took 99 us instead of 54).
#pragma unroll 1
      for (int token = first_token; token < tokens; token += turns) {
        uint32_t col = taddr + token * digits;
        int stride = n_cols, count = digits, sums = parts;
        float g = __shfl_sync(0xffffffffu, scales, token);
        float sum = 0.0f, weight = 1.0f;  // of digit j: 8^-j
#pragma unroll 1
        for (bool again = (deep_tokens >> token & 1u) != 0u;; again = false) {
          uint32_t r[4][8] = {};
          tmem_ld8(col, r[0]);  // digits <= 8: what lies behind them is not used
          if (sums > 1) tmem_ld8(col + stride, r[1]);
          if (sums > 2) {
            tmem_ld8(col + 2 * stride, r[2]);
            tmem_ld8(col + 3 * stride, r[3]);
          }
          tmem_wait_ld(r);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j < count) {
              sum = fmaf((__uint_as_float(r[0][j]) + __uint_as_float(r[1][j])) + (__uint_as_float(r[2][j]) + __uint_as_float(r[3][j])), weight, sum);
              weight *= 0.125f;
            }
          }
          if (!again) break;
          // the same code once more for the deep digits: code of its own, seldom run, is fetched from afar every time
          // (out of line a 0.8B-class step of eight tokens took 71 us)
          col = deep_addr + token * kDeepDigits;
          stride = deep_stride;
          count = kDeepDigits;
          sums = deep_parts;
        }
        if (!(g < INFINITY)) {
          // a token with NaNs has nothing else to give: a NaN times anything is one
          sum = g != g ? g : infinite_dot(it->item->w_codes, it->item->w_scales, it->item->x + static_cast<size_t>(token) * it->k_steps * 256, rows, it->k_steps * 256, 0, it->k_steps * 256, row, lane);
          g = 1.0f;
        }
        // g is a power of two, possibly a subnormal one: it comes last, so that nothing underflows before the result does
        if (gate_up) {
          // rows alternate 8 gate / 8 up: lane l holds gate row j, lane l ^ 8 the matching up row
          const float other = __shfl_xor_sync(0xffffffffu, sum, 8);
          if ((row & 8) == 0 && row + 8 < rows) {
            const int j = (row >> 4) * 8 + (row & 7);
            const float gate = sum * s2 * g, up = other * s2_up * g;
            it->y[static_cast<size_t>(token) * it->ldy + j] = __float2bfloat16_rn(gate / (1.0f + expf(-gate)) * up);
          }
        } else if (row < rows) {
          const float rv = it->residual != nullptr ? __bfloat162float(it->residual[static_cast<size_t>(token) * it->ldr + row]) : 0.0f;
          it->y[static_cast<size_t>(token) * it->ldy + row] = __float2bfloat16_rn(fmaf(sum * s2, g, rv));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(tmem_empty + ab));
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (gave_up != 0) {
    // Nothing is issued any more.  What was issued lands in this CTA's memory, so it has to land before the CTA ends: the
    // thread that issued the MMAs waits for them, and another one for the copies.  A step that one producer asked for and the
    // other did not lacks an arrival at its barrier; the ring is never more than one turn ahead of the slower producer.
    if (warp == 1 && elect_one()) {
      umma_commit(smem_u32(mma_done));
      mbar_wait(smem_u32(mma_done), 0, kDrainLimit);
    } else if (warp == 0 && elect_one()) {
      const int first = static_cast<int>(min(issued[0], issued[1])), last = static_cast<int>(max(issued[0], issued[1]));
      for (int n = first; n < last; ++n) mbar_arrive(smem_u32(full + n % stages));
      for (int n = max(last - stages, 0); n < last; ++n) mbar_wait(smem_u32(full + n % stages), (n / stages) & 1, kDrainLimit);
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
  }
}

// ---- decode: BF16 activations -> octal digits in NVFP4 ----------------------------------------------------------

// What a CTA per token expands: columns 8 * begin .. 8 * end (whole K steps) of one item's activations.
struct ExpandItem {
  const __nv_bfloat16 * x;   // [tokens, k], k a multiple of 256
  uint8_t * ops;             // see WItem::x_ops; operand row = token * digits + digit, and likewise of the deep digits
  uint32_t * deep;           // see WItem::x_deep
  float * g;                 // [tokens]: scale of each token's expansion
  int k;
  int begin, end;
  int step_bytes;            // of a K step of ops
  int scales_at;             // its scale tiles
  int deep_row, deep_at, deep_scales_at;  // the deep digits' first operand row, their codes and scale tiles
};

constexpr int kSplitThreads = 256;
// Of eight columns that a CTA expands, a multiple of 32.  A CTA per token of [.., 9216] was still at work 15 us after the first ones
// had started, and every CTA of the projection kernel waits for the last.  0.8B-class step one token 42.1 -> 41.2 us, eight 51.7 ->
// 50.9, 4B-class one 290.0 -> 289.8, four 311.7 -> 308.4; 512 chunks 42.1, 52.2, 292.0 and 306.3, 128 42.5, 52.1, 290.1 and 310.3.
constexpr int kSplitChunks = 256;
constexpr int kDeepWords = 64;   // of 32 K steps each: 524288 columns, more than a list on either path can have

// One CTA per (projection, token); digits.cuh has what they are.
// With deep digits (a list that has to be as exact as BF16 activations converted to fp16 by one power of two per token,
// which keep multiples of 2^-38 of the token's largest binade): where the first eight leave something of any value of a K
// step, six more are written, fourteen in all, which hold multiples of 2^-40 of the block's largest binade; the step is
// marked in the token's mask.  A step that was marked in the run before and is not any more gets zero scales there, since
// another token's deep digits may be used in it.  A warp takes one K step at a time.
// The deep digits cost one microsecond here with one token (4.9 -> 5.9 us; with eight the wider unrolling gives it back, 9.9
// -> 9.1) and about one in the projection.  In runs of 0.2 s, us: 0.8B-class step one token 44.2 -> 45.5, eight 54.4 -> 54.9,
// 4B-class one 305 -> 308, four 335 -> 339; always fourteen digits: 45.7, 68, 308 and 362.
// A token with a NaN, or else an infinity, gets that for its scale if `propagate`, and the epilogue works its outputs out from
// these elements; else they count as zero.
__global__ void __launch_bounds__(kSplitThreads) split_digits_kernel(const ExpandItem * __restrict__ items, int digits, int propagate) {
  // small CTAs that are soon all resident: the projection kernel may start streaming its weights
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const ExpandItem it = items[blockIdx.x];
  const int token = blockIdx.y, k = it.k, chunks = k >> 3;
  const uint4 * src = reinterpret_cast<const uint4 *>(it.x + static_cast<size_t>(token) * k);
  __shared__ uint32_t red[kSplitThreads / 32];
  __shared__ uint32_t deep_now[kDeepWords], deep_before[kDeepWords];
  const int words = (chunks + 1023) >> 10;
  auto load = [&](int c) {
    uint4 q = __ldca(src + c);
    if (!propagate) {
      uint32_t * r = reinterpret_cast<uint32_t *>(&q);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if ((r[i] & 0x7f80u) == 0x7f80u) r[i] &= 0xffff0000u;
        if ((r[i] & 0x7f800000u) == 0x7f800000u) r[i] &= 0xffffu;
      }
    }
    return q;
  };
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel before
  uint32_t best = 0, before = 0;
  if (it.deep != nullptr && static_cast<int>(threadIdx.x) < words) before = __ldcg(it.deep + 8 * threadIdx.x + token);
  for (int c = threadIdx.x; c < chunks; c += kSplitThreads) best = max(best, bf16x8_abs_max(load(c)));
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  if (threadIdx.x < kDeepWords) {
    deep_before[threadIdx.x] = before;
    deep_now[threadIdx.x] = 0u;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSplitThreads / 32; ++i) best = max(best, red[i]);
  const int top = max(static_cast<int>(best >> 7), 1);  // exponent field of the token's largest value
  if (threadIdx.x == 0 && it.begin == 0) {
    it.g[token] = best > 0x7f80u ? __uint_as_float(0x7fffffffu) : (best == 0x7f80u ? __uint_as_float(0x7f800000u) : digits_scale(top));
  }
  for (int c = it.begin + threadIdx.x; c < it.end; c += kSplitThreads) {  // whole warps: both are multiples of 32
    const uint4 q = best < 0x7f80u ? load(c) : make_uint4(0u, 0u, 0u, 0u);  // the epilogue has no use for the digits then
    uint32_t b = bf16x8_abs_max(q);
    b = max(b, __shfl_xor_sync(0xffffffffu, b, 1));
    const int e = digits_exponent(b, top);
    float v[8];
    digits_begin(q, e, v);
    uint8_t * step = it.ops + static_cast<size_t>(c >> 5) * it.step_bytes;
    // writes the next digit as an operand row
    auto write_digit = [&](uint8_t * codes, int row) {
      *reinterpret_cast<uint32_t *>(codes + row * kStepBytes + ((((c >> 2) ^ row) & 7) << 4) + ((c & 3) << 2)) = digits_next(v);
    };
    // the scale bytes of eight lanes' four blocks make one word of the tiled layout, the same for every digit
    const uint32_t byte = digits_scale_byte(e, top);
    uint32_t word = byte << (8 * ((threadIdx.x >> 1) & 3));
    word |= __shfl_xor_sync(0xffffffffu, word, 2);
    word |= __shfl_xor_sync(0xffffffffu, word, 4);
    const int j = threadIdx.x & 7;
    auto write_scales = [&](uint8_t * tiles, int row, int count, uint32_t value) {
      if (j < count) *reinterpret_cast<uint32_t *>(tiles + ((c >> 3) & 3) * kSfChunk + ((row + j) & 31) * 16 + ((row + j) >> 5) * 4) = value;
    };
    for (int i = 0; i < digits; ++i) write_digit(step, token * digits + i);
    write_scales(step + it.scales_at, token * digits, digits, word);
    if (it.deep != nullptr) {
      uint32_t rest = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) rest |= __float_as_uint(v[i]);
      const int row = it.deep_row + token * kDeepDigits;
      const int at = c >> 10, bit = c >> 5 & 31;
      if (__any_sync(0xffffffffu, (rest & 0x7fffffffu) != 0u)) {
#pragma unroll 1
        for (int i = 0; i < kDeepDigits; ++i) write_digit(step + it.deep_at, row + i);
        write_scales(step + it.deep_scales_at, row, kDeepDigits, word);
        if ((threadIdx.x & 31) == 0) atomicOr(deep_now + at, 1u << bit);
      } else if ((deep_before[at] >> bit & 1u) != 0u) {
        // zero scales again: in this step another token's deep digits may be used
        write_scales(step + it.deep_scales_at, row, kDeepDigits, 0u);
      }
    }
  }
  if (it.deep != nullptr) {
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < words) {
      // this CTA's steps of the word: the others' bits are others' to change
      const int lo = max(it.begin / 32 - 32 * static_cast<int>(threadIdx.x), 0), hi = min(it.end / 32 - 32 * static_cast<int>(threadIdx.x), 32);
      const uint32_t own = hi > lo ? (hi == 32 ? ~0u : (1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
      const uint32_t now = deep_now[threadIdx.x], gone = before & own & ~now, come = now & ~before;
      if (gone != 0u) atomicAnd(it.deep + 8 * threadIdx.x + token, ~gone);
      if (come != 0u) atomicOr(it.deep + 8 * threadIdx.x + token, come);
    }
  }
}

int plan_stages(int b_slot_bytes) {
  const int stage = kABytes + kSfBytes + b_slot_bytes;
  return std::max(2, std::min(kMaxStages, (kSmemBudget - 1024 - 256) / stage));
}
int smem_for(int stages, int b_slot_bytes) { return stages * (kABytes + kSfBytes + b_slot_bytes) + 1024 + 256; }

int ensure_attr() {
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  Q35B_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  if (!attr_set[dev & 63].load(std::memory_order_acquire)) {
    Q35B_CUDA_TRY(cudaFuncSetAttribute(gemm_wstream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget),
                  "cudaFuncSetAttribute(weight-streaming gemm smem)");
    attr_set[dev & 63].store(true, std::memory_order_release);
  }
  return Q35B_OK;
}

}  // namespace

// ---- decode work list on the tensor path ------------------------------------------------------------------------

struct WBatch {
  int m = 0, digits = 0, expand_count = 0, grid = 0, stages = 0, b_slot = 0, deep_bytes = 0, smem = 0;
  void * dev_base = nullptr;
  WItem * items = nullptr;
  WTile * tiles = nullptr;
  int * cta_begin = nullptr;
  ExpandItem * expand = nullptr;
  unsigned int * status = nullptr;
  size_t bytes_per_run = 0;
  bool wide = false;        // more epilogue warps
  bool exact = false;       // all bits of the activations, their infinities and NaNs too, reach the outputs
  uint32_t wait_limit = kWaitLimit;
};

namespace {

// K steps of every tile of a list, and two for what a tile costs besides.
std::vector<long> tile_costs(const q35b_gemv_item * items, int count) {
  std::vector<long> cost;
  for (int i = 0; i < count; ++i) cost.insert(cost.end(), (items[i].weight->rows + kRows - 1) / kRows, items[i].weight->k / 256 + 2);
  return cost;
}

// What each CTA of a grid does: the tiles, longest first, each to the CTA that has least so far (Graham 1969: the longest share is
// at most 4/3 of the best one, and even to a tile's shortest where there are many); a CTA's own in the list's order.  With
// contiguous runs the longest share of a 0.8B-class step was 100 K steps of 85.6 and its last CTA ended 7 us after half of them
// had: one token 44.9 -> 42.1 us, eight 53.5 -> 51.7; 4B-class step (746 of 709) one token 305.6 -> 290.0, four 331.8 -> 311.7.
std::vector<std::vector<int>> deal_tiles(const std::vector<long> & cost, int grid) {
  std::vector<int> order(cost.size());
  for (size_t t = 0; t < order.size(); ++t) order[t] = static_cast<int>(t);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
  std::priority_queue<std::pair<long, int>, std::vector<std::pair<long, int>>, std::greater<>> least;  // (share, CTA)
  for (int c = 0; c < grid; ++c) least.emplace(0, c);
  std::vector<std::vector<int>> dealt(grid);
  for (int t : order) {
    const auto [share, c] = least.top();
    least.pop();
    dealt[c].push_back(t);
    least.emplace(share + cost[t], c);
  }
  for (auto & tiles : dealt) std::sort(tiles.begin(), tiles.end());
  return dealt;
}

}  // namespace

double wbatch_longest_share(const q35b_gemv_item * items, int count) {
  const std::vector<long> cost = tile_costs(items, count);
  if (cost.empty()) return 0.0;
  const int grid = std::min<int>(sm_count(), static_cast<int>(cost.size()));
  long total = 0, longest = 0;
  for (const auto & tiles : deal_tiles(cost, grid)) {
    long share = 0;
    for (int t : tiles) share += cost[t];
    longest = std::max(longest, share);
    total += share;
  }
  return static_cast<double>(longest) * sm_count() / total;
}

int wbatch_build(const q35b_gemv_item * items, int count, int m, int digits, bool exact, WBatch ** out) {
  if (items == nullptr || out == nullptr || count <= 0) return fail(Q35B_ERR_ARGUMENT, "Invalid NVFP4 projection work list.");
  *out = nullptr;
  if (m < 1 || m > 8) return fail(Q35B_ERR_SHAPE, "NVFP4 decode projection supports 1..8 tokens.");
  if (digits < 1 || digits > 8 || m * digits > kMaxCols) {
    return fail(Q35B_ERR_ARGUMENT, "The tensor-core decode path takes 1..8 digits per token.");
  }
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    if (w == nullptr || items[i].x_bf16 == nullptr || items[i].y_bf16 == nullptr) {
      return fail(Q35B_ERR_ARGUMENT, "NVFP4 projection work list holds a null weight or buffer.");
    }
    if (const int st = check_weight_device(w)) return st;
    if ((w->k % 256) != 0 || w->rows <= 0 || !w->has_maps) {
      return fail(Q35B_ERR_SHAPE, "The tensor-core decode path needs cols to be a multiple of 256.");
    }
    if (w->negative_scales) return fail(Q35B_ERR_FORMAT, "The tensor-core decode path needs unsigned E4M3 block scales.");
    if (w->gate_up && items[i].residual_bf16 != nullptr) return fail(Q35B_ERR_ARGUMENT, "A gate/up projection takes no residual.");
    if (items[i].after != 0) {
      return fail(Q35B_ERR_ARGUMENT, "The tensor-core decode path runs independent items only: an item that reads another "
                                     "item's output needs its activations expanded after that item has finished "
                                     "(use q35b_gemv_batch_create for such lists, or one list per level).");
    }
    if ((reinterpret_cast<uintptr_t>(items[i].x_bf16) & 15u) != 0) {
      return fail(Q35B_ERR_ARGUMENT, "Activations of the NVFP4 projection work list must be 16-byte aligned.");
    }
  }
  if (const int st = ensure_attr()) return st;
  auto * b = new WBatch();
  b->m = m;
  b->digits = digits;
  b->exact = exact;
  const int op_rows = m * digits;
  const int n_cols = round_up_int(op_rows, 16);
  const bool inside = exact && m * (digits + kDeepDigits) <= n_cols;  // the deep digits' rows fit into the padding (one token)
  const int deep_cols = exact && !inside ? round_up_int(m * kDeepDigits, 16) : 0;
  b->deep_bytes = deep_cols > 0 ? deep_cols * kStepBytes + kSfBytes : 0;
  b->b_slot = n_cols * kStepBytes + kSfBytes + b->deep_bytes;
  b->stages = plan_stages(b->b_slot);
  b->smem = smem_for(b->stages, b->b_slot);

  // layout of the one allocation: items | tiles | cta_begin | expand items | status | per-item digit buffers
  std::vector<WTile> all;
  const std::vector<long> cost = tile_costs(items, count);
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    for (int rb = 0; rb < (w->rows + kRows - 1) / kRows; ++rb) all.push_back(WTile{i, rb});
    b->bytes_per_run += w->codes_bytes + w->scales_bytes;
  }
  long steps = 0;
  for (const WTile & t : all) steps += items[t.item].weight->k / 256;
  b->wide = m >= kWideTokens && steps < static_cast<long>(kWideSteps) * static_cast<long>(all.size());
  const int grid = std::max(1, std::min<int>(sm_count(), static_cast<int>(all.size())));
  b->grid = grid;
  std::vector<WTile> h_tiles;
  std::vector<int> h_begin;
  for (const auto & tiles : deal_tiles(cost, grid)) {
    h_begin.push_back(static_cast<int>(h_tiles.size()));
    for (int t : tiles) h_tiles.push_back(all[t]);
  }
  h_begin.push_back(static_cast<int>(h_tiles.size()));
  auto up = [](size_t v, size_t a) { return (v + a - 1) / a * a; };
  size_t expand_count = 0;
  for (int i = 0; i < count; ++i) expand_count += (items[i].weight->k / 8 + kSplitChunks - 1) / kSplitChunks;
  const size_t o_tiles = up(sizeof(WItem) * count, 256);
  const size_t o_begin = up(o_tiles + sizeof(WTile) * all.size(), 256);
  const size_t o_expand = up(o_begin + sizeof(int) * (grid + 1), 256);
  const size_t o_status = up(o_expand + sizeof(ExpandItem) * expand_count, 256);
  size_t o_data = o_status + 256;
  std::vector<size_t> o_ops(count), o_g(count), o_deep(count);
  for (int i = 0; i < count; ++i) {
    o_ops[i] = o_data;
    o_data = up(o_data + static_cast<size_t>(items[i].weight->k / 256) * b->b_slot, 256);
    o_g[i] = o_data;
    o_data += 256;
    o_deep[i] = o_data;
    if (exact) o_data = up(o_data + static_cast<size_t>((items[i].weight->k / 256 + 31) / 32) * 32, 256);
  }
  cudaError_t e = cudaMalloc(&b->dev_base, o_data);
  if (e != cudaSuccess) {
    delete b;
    return fail_cuda(e, "cudaMalloc(tensor-core projection work list)");
  }
  auto * base = static_cast<uint8_t *>(b->dev_base);
  b->items = reinterpret_cast<WItem *>(base);
  b->tiles = reinterpret_cast<WTile *>(base + o_tiles);
  b->cta_begin = reinterpret_cast<int *>(base + o_begin);
  b->expand = reinterpret_cast<ExpandItem *>(base + o_expand);
  b->status = reinterpret_cast<unsigned int *>(base + o_status);
  std::vector<WItem> h_items(count);
  std::vector<ExpandItem> h_expand;
  for (int i = 0; i < count; ++i) {
    const q35b_weight * w = items[i].weight;
    WItem & it = h_items[i];
    it = WItem{};
    it.tmap_w = w->tmap_codes_128;
    it.w_scales = w->scales_tiled;
    it.x_ops = base + o_ops[i];
    it.x_deep = exact ? reinterpret_cast<const uint32_t *>(base + o_deep[i]) : nullptr;
    it.x_g = reinterpret_cast<const float *>(base + o_g[i]);
    it.w_codes = w->codes;
    it.x = static_cast<const __nv_bfloat16 *>(items[i].x_bf16);
    it.y = static_cast<__nv_bfloat16 *>(items[i].y_bf16);
    it.residual = static_cast<const __nv_bfloat16 *>(items[i].residual_bf16);
    it.rows = w->rows;
    it.k_steps = w->k / 256;
    it.n_cols = n_cols;
    it.deep_cols = deep_cols;
    it.deep_rows = inside ? op_rows : 0;
    it.tokens = m;
    it.digits = digits;
    it.ldy = w->gate_up ? w->rows / 2 : w->rows;
    it.ldr = w->rows;
    it.s2 = w->s2;
    it.s2_up = w->s2_up;
    it.epilogue = w->gate_up ? kEpiGateUp : kEpiPlain;
    for (int begin = 0; begin < w->k / 8; begin += kSplitChunks) {
      h_expand.push_back(ExpandItem{static_cast<const __nv_bfloat16 *>(items[i].x_bf16), base + o_ops[i],
                                    exact ? reinterpret_cast<uint32_t *>(base + o_deep[i]) : nullptr, reinterpret_cast<float *>(base + o_g[i]), w->k, begin,
                                    std::min(begin + kSplitChunks, w->k / 8), b->b_slot, n_cols * kStepBytes, inside ? op_rows : 0,
                                    inside ? 0 : n_cols * kStepBytes + kSfBytes,
                                    inside ? n_cols * kStepBytes : (n_cols + deep_cols) * kStepBytes + kSfBytes});
    }
  }
  b->expand_count = static_cast<int>(h_expand.size());
  e = cudaMemset(b->dev_base, 0, o_data);
  if (e == cudaSuccess) e = cudaMemcpy(b->items, h_items.data(), sizeof(WItem) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->tiles, h_tiles.data(), sizeof(WTile) * h_tiles.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->cta_begin, h_begin.data(), sizeof(int) * (grid + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->expand, h_expand.data(), sizeof(ExpandItem) * h_expand.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(b->dev_base);
    delete b;
    return fail_cuda(e, "uploading the tensor-core projection work list");
  }
  *out = b;
  return Q35B_OK;
}

int wbatch_launch(const WBatch * b, cudaStream_t s) {
  // 1. the digits of every item's activations (one CTA per item and token); 2. the streaming kernel, whose weight
  // producer starts at once while its activation producer waits for the expansion
  cudaError_t le = launch_pdl(split_digits_kernel, dim3(b->expand_count, b->m), dim3(kSplitThreads), 0, s,
                              static_cast<const ExpandItem *>(b->expand), b->digits, b->exact ? 1 : 0);
  count_launch();
  Q35B_CUDA_TRY(le, "split_digits_kernel launch");
  le = launch_pdl(gemm_wstream_kernel, dim3(b->grid), dim3(threads_for(b->wide ? kEpilogueWarpsWide : kEpilogueWarps)), static_cast<size_t>(b->smem), s,
                  static_cast<const WItem *>(b->items), static_cast<const WTile *>(b->tiles), static_cast<const int *>(b->cta_begin),
                  b->stages, b->b_slot, b->deep_bytes, b->status, b->wait_limit);
  count_launch();
  Q35B_CUDA_TRY(le, "gemm_wstream_kernel launch");
  return Q35B_OK;
}

void wbatch_free(WBatch * b) {
  if (b == nullptr) return;
  if (b->dev_base != nullptr) cudaFree(b->dev_base);
  delete b;
}

int wbatch_status(const WBatch * b, unsigned int * out) {
  Q35B_CUDA_TRY(cudaMemcpy(out, b->status, sizeof(unsigned int), cudaMemcpyDeviceToHost), "cudaMemcpy(work list status)");
  return Q35B_OK;
}

int wbatch_debug_wait(WBatch * b, unsigned int wait_limit) {
  b->wait_limit = wait_limit;
  Q35B_CUDA_TRY(cudaMemset(b->status, 0, sizeof(unsigned int)), "cudaMemset(work list status)");
  return Q35B_OK;
}

size_t wbatch_bytes(const WBatch * b) { return b->bytes_per_run; }

}  // namespace q35b
