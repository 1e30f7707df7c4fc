// W4A4 prefill GEMM for sm_100a, weight rows on the 128-row side of the tensor-core tile, K split over a cluster:
// C[M, N] (bf16) = (Aq . Wq^T) * g * s2 with tcgen05.mma kind::mxf4nvf4 (block16, UE4M3 scale factors), TMEM
// accumulators, TMA-fed shared-memory ring.
//
// Replaces the reference's cuBLASLt FP4 call and the passes around it
// (src/runtime/cuda_bench.cu:1056-1167 run_nvfp4_cublaslt_prefill_projection_device,
// the fp32->bf16 pass at src/kernels/cuda/prefill.cu:639) and the SM120
// mma.sync projection (src/runtime/cuda_bench.cu:431-484) for problems too small to fill the chip with the
// 256 x 256 tiles of gemm_w4a4_2cta.cu.
//
// Operands in HBM
//   W codes  [N, K/2]  E2M1 pairs, K-major (checkpoint order, untouched)      -> UMMA A, 128 rows
//   X codes  [M, K/2]  E2M1 pairs, K-major (activation quantiser output)      -> UMMA B, 16..128 tokens
//   scales   128x4 tiles of 512 bytes (row-block major), one tile = the scale
//            factors of a 128-row x 64-column operand slab = exactly the
//            shared-memory image tcgen05.cp 32x128b.warpx4 copies to TMEM.
//
// What bounds it: such a problem is a few megabytes of weights, about a microsecond of HBM, so what counts is how many
// SMs pull them and how long the serial chain of K steps is.  One CTA per 128 x 128 tile leaves [2560, 9216] on 20 SMs
// with 36 steps each.  Here `split` CTAs (1, 2, 4 or 8, a cluster) share a tile, each taking a contiguous part of its
// K steps; they leave their fp32 accumulators in shared memory, meet at a cluster barrier, and every CTA adds up and
// stores its share of the tokens, reading the others' partial sums over distributed shared memory in rank order (the
// result does not depend on timing, and no workspace in HBM is needed).  The sums come back from shared memory with
// lanes along the weight rows, so output rows are stored in whole 256-byte pieces, and rows that start at an odd
// address still in 64-byte ones.
//
// Every mbarrier wait is bounded: on expiry the kernel writes a code to
// *status, abandons the tile, still meets its cluster, frees its TMEM and returns.
// *status counts only as read after griddepcontrol.wait: an earlier kernel of the stream may be what sets it to zero.
// By then the weight loads are under way, so a code found there stops the stores, not the loads, and the CTAs of a
// cluster decide together.  A CTA that reads a code at its start waits at once and reads again: after an expired wait
// the rest of the grid drains instead of running into the same one tile by tile.
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "engine.h"
#include "gemm_epilogue.cuh"
#include "nvfp4_codec.cuh"

namespace q35b {
namespace {

constexpr int kRows = 128;               // weight rows per tile (UMMA M)
constexpr int kMaxCols = 128;            // tokens per tile (UMMA N, a multiple of 16)
constexpr int kStepBytes = 128;          // one 128B swizzle row = 256 FP4 elements of K
constexpr int kMmaPerStage = 4;          // four K=64 MMAs per stage
constexpr int kSfChunk = 512;            // scale factors of 128 rows x 64 columns
constexpr int kABytes = kRows * kStepBytes;
constexpr int kSfBytes = kMmaPerStage * kSfChunk;
constexpr int kThreads = 512;            // warps 0-2 weight loads, MMA, activation loads; all sixteen the epilogue
constexpr int kMaxStages = 8;
constexpr int kMaxSplit = 8;
constexpr int kPitch = kRows + 4;        // floats per token of the partial sums in shared memory
constexpr int kAccCols = 128;            // accumulators: up to four partial ones of few tokens side by side
constexpr int kSfSetCols = 32;           // two sets of scale-factor columns, used by stages in turn
constexpr int kTmemCols = 256;
constexpr int kFixedBytes = 1024 /*alignment slack*/ + 256 /*barriers*/;
// Two CTAs per SM where the grid has that many: one's prologue and epilogue run under the other's loads.
constexpr int kSmemHalf = 112 * 1024, kSmemFull = 224 * 1024;
constexpr uint32_t kWaitLimit = 1u << 20;  // try_wait polls before giving up (4 us each on B200, 4 s in all)

enum StatusCode : unsigned { kStatusProducerWait = 1, kStatusMmaWait = 2, kStatusEpilogueWait = 3, kStatusActWait = 4 };

// ---- PTX wrappers -----------------------------------------------------------

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

// Bounded wait on a phase parity; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < kWaitLimit; ++i) {
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

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "elect.sync _|p, 0xffffffff;\n\t"
    "selp.u32 %0, 1, 0, p;\n\t}"
    : "=r"(pred));
  return pred != 0;
}

// Shared-memory matrix descriptor (tcgen05): K-major operand, 128B swizzle,
// 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t desc_k_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);         // start address
  d |= static_cast<uint64_t>(0) << 16;                         // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                 // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                         // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;                         // SWIZZLE_128B
  return d;
}

// Descriptor of a scale-factor slab for tcgen05.cp: no swizzle, 8 rows of 16
// bytes per core matrix, core matrices 128 bytes apart.
__device__ __forceinline__ uint64_t desc_sf(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(128 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}

// Instruction descriptor, kind::mxf4nvf4: A,B = E2M1 (1), K-major, UE4M3
// scale factors (0), M = 128, N = n_cols, dense K = 64.
__device__ __forceinline__ uint32_t instr_desc(int n_cols) {
  uint32_t d = 0;
  d |= 1u << 7;                                  // a_format = E2M1
  d |= 1u << 10;                                 // b_format = E2M1
  d |= static_cast<uint32_t>(n_cols >> 3) << 17;   // n_dim
  d |= 0u << 23;                                 // scale format UE4M3
  d |= static_cast<uint32_t>(kRows >> 4) << 24;    // m_dim
  return d;
}

__device__ __forceinline__ void umma_mxf4nvf4(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
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

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
    : "r"(taddr)
    : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Sum over the cluster's partial sums at byte offset `off` of every rank's `src`, in rank order.
template <int SPLIT>
__device__ __forceinline__ float4 sum4(const uint32_t (&src)[SPLIT], uint32_t off) {
  float4 v[SPLIT];
#pragma unroll
  for (int q = 0; q < SPLIT; ++q) {
    if constexpr (SPLIT == 1) {
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w) : "r"(src[q] + off));
    } else {
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w) : "r"(src[q] + off));
    }
  }
#pragma unroll
  for (int q = 1; q < SPLIT; ++q) {
    v[0].x += v[q].x; v[0].y += v[q].y; v[0].z += v[q].z; v[0].w += v[q].w;
  }
  return v[0];
}

// With few tokens an MMA is far shorter than the tensor pipe's latency, and the four MMAs of a stage, if they all
// accumulate into the same columns, run one after the other at that latency.  They go to different partial
// accumulators then (as many as fit), which the epilogue adds.
__device__ __forceinline__ int partial_accumulators(int n_cols) { return 4 * n_cols <= kAccCols ? 4 : (2 * n_cols <= kAccCols ? 2 : 1); }

enum Epi : int { kEpiPlain = 0, kEpiGateUp = 1, kEpiNvfp4 = 2 };

// The first `count` of four BF16 values, element by element.
__device__ __forceinline__ void store4_narrow(__nv_bfloat16 * dst, uint2 p, int count) {
  uint16_t * d = reinterpret_cast<uint16_t *>(dst);
  if (count > 0) d[0] = static_cast<uint16_t>(p.x);
  if (count > 1) d[1] = static_cast<uint16_t>(p.x >> 16);
  if (count > 2) d[2] = static_cast<uint16_t>(p.y);
  if (count > 3) d[3] = static_cast<uint16_t>(p.y >> 16);
}

// The same store on every other rank of a gathering launch; out of line, so that launches without peers do not fetch it.
__device__ __noinline__ void store4_to_peers(const GemmEpilogue & ep, size_t at, uint2 p, int count, bool whole) {
#pragma unroll 1
  for (int i = 0; i < ep.n_peers; ++i) {
    if (whole) {
      *reinterpret_cast<uint2 *>(ep.peer_c[i] + at) = p;
    } else {
      store4_narrow(ep.peer_c[i] + at, p, count);
    }
  }
}

// ---- kernel -------------------------------------------------------------------

// grid (weight row blocks, token tiles, SPLIT), cluster (1, 1, SPLIT).
template <int SPLIT, int EPI>
__global__ void __launch_bounds__(kThreads, 2)
gemm_w4a4_ksplit_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                        const uint8_t * __restrict__ sfw, const uint8_t * __restrict__ sfx,
                        const float * __restrict__ g_dev, const __grid_constant__ GemmEpilogue ep, int m, int n, int k_bytes, int stages,
                        int ring_bytes, int box_cols, int tile_cols, int accumulators, int vec, __nv_bfloat16 * __restrict__ c, int ldc, unsigned int * status) {
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment for the 128B-swizzled operand tiles.
  uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int b_bytes = box_cols * kStepBytes;
  uint8_t * smem_a = smem;
  uint8_t * smem_b = smem_a + stages * kABytes;
  uint8_t * smem_sfa = smem_b + stages * b_bytes;
  uint8_t * smem_sfb = smem_sfa + stages * kSfBytes;
  uint64_t * bars = reinterpret_cast<uint64_t *>(smem + ring_bytes);
  uint64_t * full = bars;                  // [stages]: both producers' bytes have landed
  uint64_t * empty = bars + kMaxStages;    // [stages]: the MMAs that read the stage have retired
  uint64_t * acc_full = bars + 2 * kMaxStages;
  uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
  float * part = reinterpret_cast<float *>(smem);  // [tokens][kPitch] partial sums, over the ring once it is done with

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rb = blockIdx.x;
  const int token0 = static_cast<int>(blockIdx.y) * tile_cols;
  const int rank = SPLIT > 1 ? static_cast<int>(cluster_rank()) : 0;
  const int tokens = min(tile_cols, m - token0);
  const int n_cols = (tokens + 15) & ~15;
  const int sf_col_blocks = k_bytes >> 5;                        // K/64: 512-byte scale tiles per row block
  const int k_steps = (sf_col_blocks + kMmaPerStage - 1) / kMmaPerStage;
  const int ks0 = rank * k_steps / SPLIT, ks1 = (rank + 1) * k_steps / SPLIT;
  const int parts = min(partial_accumulators(n_cols), accumulators);

  __shared__ unsigned int s_abort;  // nonzero: an error was on record when this CTA started, it loads nothing
  __shared__ unsigned int s_stop;   // nonzero: it stores nothing (that, an error found later, or an expired wait)
  if (threadIdx.x == 0) {
    unsigned int code = *reinterpret_cast<volatile unsigned int *>(status);
    if (code != 0u) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      code = *reinterpret_cast<volatile unsigned int *>(status);
    }
    s_abort = s_stop = code;
    for (int i = 0; i < stages; ++i) {
      mbar_init(smem_u32(full + i), 2);
      mbar_init(smem_u32(empty + i), 1);
    }
    mbar_init(smem_u32(acc_full), 1);
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
  const bool aborted = s_abort != 0u;
  // Launched with programmatic stream serialisation: weights are constant and the first ring of them starts loading at
  // once; activations, residuals and every store come after griddepcontrol.wait, when all earlier work of the stream is
  // complete.  So does every mbarrier wait that can block: its bound is meant for this kernel's own loads and MMAs, not
  // for however long the kernel before still runs.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ---------------- weight loads ----------------
    if (elect_one() && !aborted) {
      const uint8_t * sf = sfw + static_cast<size_t>(rb) * sf_col_blocks * kSfChunk;
      int stage = 0;
      uint32_t phase = 0;
      for (int ks = ks0; ks < ks1; ++ks) {
        if (ks - ks0 == stages) asm volatile("griddepcontrol.wait;" ::: "memory");  // the stages so far were free
        if (!mbar_wait(smem_u32(empty + stage), phase ^ 1)) {
          atomicExch(status, kStatusProducerWait);
          break;
        }
        const uint32_t sf_bytes = min(kMmaPerStage, sf_col_blocks - ks * kMmaPerStage) * kSfChunk;
        const uint32_t bar = smem_u32(full + stage);
        mbar_expect_tx(bar, kABytes + sf_bytes);
        tma_load_2d(smem_u32(smem_a + stage * kABytes), &tmap_w, bar, ks * kStepBytes, rb * kRows);
        bulk_load(smem_u32(smem_sfa + stage * kSfBytes), sf + static_cast<size_t>(ks) * kSfBytes, sf_bytes, bar);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 2) {
    // ---------------- activation loads ----------------
    if (elect_one() && !aborted) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const uint8_t * sf = sfx + static_cast<size_t>(token0 >> 7) * sf_col_blocks * kSfChunk;
      int stage = 0;
      uint32_t phase = 0;
      for (int ks = ks0; ks < ks1; ++ks) {
        if (!mbar_wait(smem_u32(empty + stage), phase ^ 1)) {
          atomicExch(status, kStatusActWait);
          break;
        }
        const uint32_t sf_bytes = min(kMmaPerStage, sf_col_blocks - ks * kMmaPerStage) * kSfChunk;
        const uint32_t bar = smem_u32(full + stage);
        mbar_expect_tx(bar, b_bytes + sf_bytes);
        tma_load_2d(smem_u32(smem_b + stage * b_bytes), &tmap_x, bar, ks * kStepBytes, token0);
        bulk_load(smem_u32(smem_sfb + stage * kSfBytes), sf + static_cast<size_t>(ks) * kSfBytes, sf_bytes, bar);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one() && !aborted) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const uint32_t idesc = instr_desc(n_cols);
      const uint32_t sfb_off = static_cast<uint32_t>(token0 & 127) >> 5;  // a 64-token tile may start in the middle of a scale tile
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int ks = ks0; ks < ks1; ++ks) {
        const int it = ks - ks0;
        if (!mbar_wait(smem_u32(full + stage), phase)) {
          atomicExch(status, kStatusMmaWait);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int valid = min(kMmaPerStage, sf_col_blocks - ks * kMmaPerStage);
        // the address field of a descriptor counts 16-byte units, so stepping one is an add
        const uint64_t a_desc = desc_k_sw128(smem_u32(smem_a + stage * kABytes));
        const uint64_t b_desc = desc_k_sw128(smem_u32(smem_b + stage * b_bytes));
        const uint64_t sfa_desc = desc_sf(smem_u32(smem_sfa + stage * kSfBytes));
        const uint64_t sfb_desc = desc_sf(smem_u32(smem_sfb + stage * kSfBytes));
        const uint32_t sf_set = tmem_base + kAccCols + (it & 1) * kSfSetCols;
#pragma unroll
        for (int j = 0; j < kMmaPerStage; ++j) {
          if (j < valid) {
            utccp_sf(sf_set + j * 4, sfa_desc + j * (kSfChunk >> 4));
            utccp_sf(sf_set + 16 + j * 4, sfb_desc + j * (kSfChunk >> 4));
          }
        }
#pragma unroll
        for (int j = 0; j < kMmaPerStage; ++j) {
          if (j < valid) {
            umma_mxf4nvf4(tmem_base + (j & (parts - 1)) * n_cols, a_desc + j * 2, b_desc + j * 2, idesc, sf_set + j * 4,
                          sf_set + 16 + j * 4 + sfb_off, (it * kMmaPerStage + j) >= parts ? 1u : 0u);
          }
        }
        umma_commit(smem_u32(empty + stage));  // frees the stage when these MMAs and copies retire
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) umma_commit(smem_u32(acc_full));  // accumulator complete, and with it every load of the ring consumed
    }
  } else if (warp == 3) {
    // ---------------- an error on record? ----------------
    if (elect_one() && !aborted) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (*reinterpret_cast<volatile unsigned int *>(status) != 0u) s_stop = 1u;
    }
  }
  __syncwarp();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the tensors' scales, on their way while the sums are waited for (asked for behind them: 1 us of a 9.4 us call)
  const float g = __ldcg(g_dev), q_g = EPI == kEpiNvfp4 ? __ldcg(ep.q_g) : 1.0f;

  // ---------------- epilogue: TMEM -> shared memory -> sum over the cluster -> global ----------------
  bool ran = !aborted;
  if (ran && !__all_sync(0xffffffffu, mbar_wait(smem_u32(acc_full), 0))) {  // the whole warp goes on, or none of it
    if (lane == 0) {
      atomicExch(status, kStatusEpilogueWait);
      s_stop = 1u;
    }
    ran = false;
  }
  if (ran) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int quarter = warp & 3;                 // TMEM lanes this warp may touch
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    // partial accumulators that were written: a slice of one short step has fewer MMAs than there are of them
    const int mmas = min((ks1 - ks0) * kMmaPerStage, sf_col_blocks - ks0 * kMmaPerStage);
    const int used = min(parts, mmas);
    float * dst = part + quarter * 32 + lane;
#pragma unroll 1
    for (int c0 = 16 * (warp >> 2); c0 < n_cols; c0 += 4 * (kThreads / 32)) {
      uint32_t r[16];
      tmem_ld16(taddr + c0, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll 1
      for (int p = 1; p < used; ++p) {
        uint32_t r2[16];
        tmem_ld16(taddr + p * n_cols + c0, r2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[(c0 + i) * kPitch] = __uint_as_float(r[i]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if constexpr (SPLIT > 1) cluster_sync(); else __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
  }
  // One CTA's expired wait leaves no sums for the others to add: the whole cluster stores, or none of it does.  Every
  // lane asks one CTA, and the lanes are asked only when the first sums are there (0.2 us of a 7 us kernel).
  const bool stop_lane = (SPLIT > 1 ? ld_cluster_u32(map_to_rank(smem_u32(&s_stop), lane & (SPLIT - 1))) : s_stop) != 0u;
  {
    // this CTA's share of the tokens
    const int t_begin = rank * n_cols / SPLIT, t_end = min((rank + 1) * n_cols / SPLIT, tokens);
    const float alpha = g * ep.s2, alpha_up = g * ep.s2_up;
    uint32_t src[SPLIT];
#pragma unroll
    for (int q = 0; q < SPLIT; ++q) src[q] = SPLIT > 1 ? map_to_rank(smem_u32(part), q) : smem_u32(part);
    const int row0 = rb * kRows;
    // Compact loops: this code runs once per CTA, so what it costs is mostly the fetching of its instructions
    // (unrolled four times and with the peers' stores inline it took 4.5 us at 128 tokens).
    if constexpr (EPI == kEpiNvfp4) {
      // one thread per token and 32 weight rows = one block of 16 outputs (n % 128 == 0 is checked on the host);
      // lanes along the tokens, whose pitch spreads them over the banks
      const GemmQuantScale q = {q_g, __frcp_rn(q_g), nullptr};
      const int live = __any_sync(0xffffffffu, stop_lane) ? 0 : t_end - t_begin;
      for (int u = threadIdx.x; u < live * (kRows / 32); u += kThreads) {
        const int t = t_begin + u % live, blk = u / live;
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 a = sum4<SPLIT>(src, static_cast<uint32_t>(t * kPitch + 32 * blk + i) * 4u);
          r[i] = __float_as_uint(a.x); r[i + 1] = __float_as_uint(a.y); r[i + 2] = __float_as_uint(a.z); r[i + 3] = __float_as_uint(a.w);
        }
        store_nvfp4_chunk32<false>(r, token0 + t, row0 + 32 * blk, alpha, alpha_up, ep, q);
      }
    } else {
      // one warp per token, four consecutive weight rows per lane
      const int row = row0 + 4 * lane;
      // output column of the lane's first value; a gate/up weight's rows alternate 8 gate / 8 up, so lanes l and l ^ 2
      // hold matching gate and up rows and the first of them stores
      const int col = EPI == kEpiGateUp ? (row >> 4) * 8 + (row & 7) : row;
      const int count = EPI == kEpiGateUp ? ((lane & 2) == 0 ? n - (row + 8) : 0) : n - row;
      const bool whole = vec != 0 && count >= 4;
      const __nv_bfloat16 * res = ep.residual + static_cast<size_t>(token0 + t_begin + warp) * ep.ldr + row;
      size_t at = static_cast<size_t>(token0 + t_begin + warp) * ldc + col;
#pragma unroll 1
      for (int t = t_begin + warp; t < t_end; t += kThreads / 32) {
        const float4 a = sum4<SPLIT>(src, static_cast<uint32_t>(t * kPitch + 4 * lane) * 4u);
        if (__any_sync(0xffffffffu, stop_lane)) break;
        float v[4] = {a.x, a.y, a.z, a.w};
        if constexpr (EPI == kEpiGateUp) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float up = __shfl_xor_sync(0xffffffffu, v[e], 2);
            v[e] = silu_mul(v[e] * alpha, up * alpha_up);
          }
        } else {
          float rv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (ep.residual != nullptr) {
            if (whole) {
              const uint2 p = __ldcg(reinterpret_cast<const uint2 *>(res));
              rv[0] = __uint_as_float(p.x << 16); rv[1] = __uint_as_float(p.x & 0xffff0000u);
              rv[2] = __uint_as_float(p.y << 16); rv[3] = __uint_as_float(p.y & 0xffff0000u);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) if (e < count) rv[e] = __bfloat162float(res[e]);
            }
            res += static_cast<size_t>(ep.ldr) * (kThreads / 32);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = fmaf(v[e], alpha, rv[e]);
        }
        const uint2 p = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        if (whole) {
          *reinterpret_cast<uint2 *>(c + at) = p;
        } else {
          store4_narrow(c + at, p, count);
        }
        if (ep.n_peers > 0) store4_to_peers(ep, at, p, count, whole);
        at += static_cast<size_t>(ldc) * (kThreads / 32);
      }
    }
  }

  gemm_signal_peers(ep, status);
  __syncwarp();
  if constexpr (SPLIT > 1) cluster_sync();  // no CTA may leave while another still reads its partial sums
}

// ---- host side ---------------------------------------------------------------

}  // namespace

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void * p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

// 2-D map over a K-major code matrix [rows, k_bytes] of bytes; box = box_rows x 128 bytes, 128B swizzle.
// Shared with the streaming decode kernel, whose tiles are 128-row boxes of the same matrix.
int make_code_map(CUtensorMap * map, const void * base, int rows, int k_bytes, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return fail(Q35B_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the CUDA driver.");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kStepBytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    return fail(Q35B_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult " + std::to_string(static_cast<int>(r)) + ".");
  }
  return Q35B_OK;
}

namespace {

// Tokens per tile and CTAs per tile.
//
// Estimates in nanoseconds, fitted to CUDA-graph timings on B200: a K step takes 250, tokens cost 6.6 each in loads and
// epilogue, and the exchange of a split costs 400 + 3.3 per token + 7 per token and doubling ([64, 2560] x [1024, 2560]:
// 5.1 us unsplit, 4.9 split in two or four, 5.0 in eight; [9, 5760] x [108, 5760]: 7.9, 5.5, 4.0, 3.4 us;
// [128, 9216] x [512, 9216]: 12.2, 8.9, 7.1, 6.9 us with 128 tokens per tile, 11.9, 8.3, 6.3, 5.8 us with 64).
// Halving the tiles or splitting K pays only while all CTAs run at once ([128, 2560] x [18432, 2560], 144 tiles:
// 7.3 us, 9.3 split in two, 9.0 with 64 tokens per tile), and a split has to gain 0.3 us to be worth it.
struct Shape {
  int tile_cols, split;
};
Shape choose_shape(int m, int row_blocks, int k_steps, int sms, int max_split) {
  Shape best = {kMaxCols, 1};
  int best_ns = 0;
  for (int cols = kMaxCols; cols >= 64; cols /= 2) {
    const int tiles = row_blocks * ((m + cols - 1) / cols), live = std::min(cols, round_up_int(m, 16));
    if (cols < kMaxCols && (m <= cols || tiles > sms)) break;
    for (int split = 1, log2 = 0; split <= max_split; split *= 2, ++log2) {
      if (split > 1 && (tiles * split > sms || k_steps < 2 * split)) break;
      const int ns = (k_steps + split - 1) / split * 250 + live * 66 / 10 +
                     (split > 1 ? 400 + live * 33 / 10 + live * 7 * log2 : 0);
      if (best_ns == 0 || ns + (split > best.split ? 300 : 0) < best_ns) {
        best = {cols, split};
        best_ns = ns;
      }
    }
  }
  return best;
}

// The kernel and the shape for a projection of m tokens, and with them the order in which its K is summed.
//
// Up to kSplitTokens tokens a tile's K steps may be split over CTAs and the MMAs of a step over partial accumulators; how
// depends on m, K and the rows of the whole tensor, not on those of the shard, so that the columns of a row shard are bit
// for bit those of the unsharded projection.  Above, every kernel sums K in order into one accumulator, so that a token's
// outputs depend neither on the shard nor on how many other tokens there are: ranks that share out the tokens, and groups
// of tokens projected one after the other, get the bits of the whole.
//
// Large problems: pairs of CTAs on 256 x 256 tiles, persistent (gemm_w4a4_2cta.cu).  They need many tiles to win: up
// to two 128 x 128 tiles per SM the kernel above is faster (us, this kernel / pairs: [512, 2560] x [9216, 2560]
// 8.9 / 10.5, [768, ..] 15.6 / 14.4; [1024, 4096] x [4096, 4096] 10.8 / 12.2, [1536, ..] 19.4 / 17.7), up to three
// where K is short ([2048, 1024] x [3584, 1024] 10.7 / 11.0, [3072, ..] 15.3 / 13.9), only one where K is long
// ([768, 9216] x [2560, 9216] 13.6 / 17.3, [1536, ..] 19.8 / 18.3).  The pairs also store rows that are not 32-byte
// aligned element by element ([4096, 640] x [5000, 640] 24 / 133).
//
// What the order costs, us in order / split ([m, 9216] x [2560, 9216]): 64 tokens 12.1 / 7.4, 128 12.3 / 8.4, 192
// 12.4 / 9.6, 384 12.9 / 10.4, 512 13.8 / 13.6; [192, 8192] x [512, 8192] 11.0 / 6.2; with K up to 2560 nothing.
constexpr int kSplitTokens = 128;
struct GemmPlan {
  bool pairs;
  int tile_cols, split, accumulators;
};
GemmPlan plan_gemm(int m, int rows, int n_total, int k, int sms, bool gather, bool rows_aligned) {
  const int k_steps = (k + 255) / 256, row_blocks = (rows + kRows - 1) / kRows;
  if (m <= kSplitTokens) {
    const Shape shape = choose_shape(m, (n_total + kRows - 1) / kRows, k_steps, sms, kMaxSplit);
    return {false, shape.tile_cols, shape.split, kMmaPerStage};
  }
  const long token_tiles = (m + kMaxCols - 1L) / kMaxCols, tiles = row_blocks * token_tiles;
  const long few = static_cast<long>(sms) * (k_steps <= 4 ? 3 : (k_steps <= 20 ? 2 : 1));
  // token tiles are the grid's y here, at most 65535 of them; the pairs walk any number
  const bool pairs = gather || (tiles > few && rows_aligned) || token_tiles > 65535;
  if (pairs && gemm_2cta_eligible(rows, m, k)) return {true, 0, 1, 1};
  return {false, choose_shape(m, row_blocks, k_steps, sms, 1).tile_cols, 1, 1};
}

int launch_gemm_ksplit(const q35b_weight * w, const uint8_t * a_codes, const uint8_t * a_scales, const float * g_dev, int m,
                       void * c, int ldc, const GemmEpilogue & ep, const GemmPlan & plan, unsigned int * status, cudaStream_t s) {
  const int row_blocks = (w->rows + kRows - 1) / kRows, k_steps = (w->k + 255) / 256;
  const int tile_cols = plan.tile_cols, split = plan.split;
  const int box_cols = std::min(tile_cols, round_up_int(m, 16));
  CUtensorMap tmap_x;
  if (const int st = make_code_map(&tmap_x, a_codes, m, w->k / 2, box_cols)) return st;
  const int token_tiles = (m + tile_cols - 1) / tile_cols;
  const int ctas = row_blocks * token_tiles * split;
  const int stage_bytes = kABytes + box_cols * kStepBytes + 2 * kSfBytes;
  const int budget = ctas > sm_count() ? kSmemHalf : kSmemFull;
  const int stages = std::min({kMaxStages, (budget - kFixedBytes) / stage_bytes, std::max(2, (k_steps + split - 1) / split)});
  // the partial sums reuse the ring, and want at least their own size
  const int ring = round_up_int(std::max(stages * stage_bytes, box_cols * kPitch * 4), 128);
  // 8-byte pieces of every row of the output (and of the residual and the peers' copies) are aligned
  bool vec = (ldc % 4) == 0 && (reinterpret_cast<uintptr_t>(c) & 7u) == 0;
  if (ep.residual != nullptr) vec = vec && (ep.ldr % 4) == 0 && (reinterpret_cast<uintptr_t>(ep.residual) & 7u) == 0;
  for (int i = 0; i < ep.n_peers; ++i) vec = vec && (reinterpret_cast<uintptr_t>(ep.peer_c[i]) & 7u) == 0;
  using Kernel = decltype(&gemm_w4a4_ksplit_kernel<1, kEpiPlain>);
  static constexpr Kernel kernels[3][4] = {
    {gemm_w4a4_ksplit_kernel<1, kEpiPlain>, gemm_w4a4_ksplit_kernel<2, kEpiPlain>, gemm_w4a4_ksplit_kernel<4, kEpiPlain>, gemm_w4a4_ksplit_kernel<8, kEpiPlain>},
    {gemm_w4a4_ksplit_kernel<1, kEpiGateUp>, gemm_w4a4_ksplit_kernel<2, kEpiGateUp>, gemm_w4a4_ksplit_kernel<4, kEpiGateUp>, gemm_w4a4_ksplit_kernel<8, kEpiGateUp>},
    {gemm_w4a4_ksplit_kernel<1, kEpiNvfp4>, gemm_w4a4_ksplit_kernel<2, kEpiNvfp4>, gemm_w4a4_ksplit_kernel<4, kEpiNvfp4>, gemm_w4a4_ksplit_kernel<8, kEpiNvfp4>}};
  const int epi = ep.q_codes != nullptr ? kEpiNvfp4 : (ep.gate_up ? kEpiGateUp : kEpiPlain), log2_split = split == 8 ? 3 : split >> 1;
  const Kernel kernel = kernels[epi][log2_split];
  // Only the instantiation that runs: setting the attribute loads the kernel, and all twelve made the first projection of a
  // process take 0.93 ms instead of 0.31.
  static std::atomic<bool> attr_set[64][3][4];
  std::atomic<bool> & set = attr_set[w->device & 63][epi][log2_split];
  if (!set.load(std::memory_order_acquire)) {
    // idempotent, so two threads getting here together is harmless
    Q35B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemFull), "cudaFuncSetAttribute(gemm smem)");
    set.store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(row_blocks), static_cast<unsigned>(token_tiles), static_cast<unsigned>(split));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(ring + kFixedBytes);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = static_cast<unsigned>(split);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, w->tmap_codes_128, tmap_x, static_cast<const uint8_t *>(w->scales_tiled),
                                            a_scales, g_dev, ep, m, w->rows, w->k / 2, stages, ring, box_cols, tile_cols, plan.accumulators, vec ? 1 : 0,
                                            static_cast<__nv_bfloat16 *>(c), ldc, status);
  count_launch();
  Q35B_CUDA_TRY(le, "gemm_w4a4_ksplit_kernel launch");
  return Q35B_OK;
}

// What the entry points use as *status when the caller passes none: two words per device inside the library (no allocation
// anywhere on that path), the prefill GEMMs', which a GEMM that finds a code in it stores nothing after, and that of single decode
// projections, which keeps nothing else from running.
__device__ unsigned int g_default_status[2];

}  // namespace

int gemm_plan_debug(int m, int rows, int n_total, int k, int sms, bool gather, bool rows_aligned, int * pairs, int * tile_cols,
                    int * split, int * accumulators) {
  if (m < 1 || rows < 1 || n_total < rows || k < 64 || (k % 64) != 0 || sms < 1 || pairs == nullptr || tile_cols == nullptr ||
      split == nullptr || accumulators == nullptr) {
    return fail(Q35B_ERR_ARGUMENT, "Invalid arguments for the plan of an NVFP4 prefill projection.");
  }
  const GemmPlan p = plan_gemm(m, rows, n_total, k, sms, gather, rows_aligned);
  *pairs = p.pairs ? 1 : 0;
  *tile_cols = p.tile_cols;
  *split = p.split;
  *accumulators = p.accumulators;
  return Q35B_OK;
}

int default_status_word(unsigned int ** out, DefaultStatus which) {
  static std::mutex mutex;
  static unsigned int * word[64] = {nullptr};
  int dev = 0;
  Q35B_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev < 0 || dev >= 64) return fail(Q35B_ERR_ARGUMENT, "Device ordinal out of range.");
  std::lock_guard<std::mutex> lock(mutex);
  if (word[dev] == nullptr) {
    // the symbol's name is only a handle in host code; its address on the current device comes from the runtime
    void * p = nullptr;
    Q35B_CUDA_TRY(cudaGetSymbolAddress(&p, g_default_status), "cudaGetSymbolAddress(default status word)");
    word[dev] = static_cast<unsigned int *>(p);
  }
  *out = word[dev] + which;
  return Q35B_OK;
}

}  // namespace q35b

extern "C" int q35b_gemm_default_status(unsigned int * status_out) {
  using namespace q35b;
  if (status_out == nullptr) return fail(Q35B_ERR_ARGUMENT, "Null status pointer.");
  unsigned int * word = nullptr;
  if (const int st = default_status_word(&word)) return st;
  unsigned int codes[2];
  Q35B_CUDA_TRY(cudaMemcpy(codes, word, sizeof codes, cudaMemcpyDeviceToHost), "cudaMemcpy(default status words)");
  *status_out = codes[0] != 0u ? codes[0] : codes[1];
  if (*status_out != 0u) Q35B_CUDA_TRY(cudaMemset(word, 0, sizeof codes), "cudaMemset(default status words)");
  return Q35B_OK;
}

namespace q35b {

int launch_gemm_w4a4(const q35b_weight * w, const uint8_t * a_codes, const uint8_t * a_scales_tiled, const float * g_dev,
                     int m, void * c_bf16, int ldc, const void * residual_bf16, int ldr, unsigned int * status_dev,
                     cudaStream_t s, const GemmQuantOut * qout, const GemmGather * gather) {
  if (w == nullptr || a_codes == nullptr || a_scales_tiled == nullptr || g_dev == nullptr ||
      (c_bf16 == nullptr && qout == nullptr)) {
    return fail(Q35B_ERR_ARGUMENT, "NVFP4 prefill projection received a null device buffer.");
  }
  const int out_cols = w->gate_up ? w->rows / 2 : w->rows;
  if (m <= 0 || (qout == nullptr && ldc < out_cols)) return fail(Q35B_ERR_SHAPE, "Invalid dimensions for NVFP4 prefill projection.");
  if (qout != nullptr) {
    if (!w->gate_up) return fail(Q35B_ERR_ARGUMENT, "NVFP4 output of the prefill projection needs a gate/up weight.");
    if (qout->codes == nullptr || qout->scales_tiled == nullptr || qout->g_dev == nullptr) {
      return fail(Q35B_ERR_ARGUMENT, "NVFP4 prefill projection received a null device buffer.");
    }
    if ((out_cols % 64) != 0) return fail(Q35B_ERR_SHAPE, "NVFP4 output of the prefill projection needs rows / 2 to be a multiple of 64.");
    if ((w->row_begin % 128) != 0 || qout->total_cols < w->row_begin / 2 + out_cols || (qout->total_cols % 64) != 0) {
      return fail(Q35B_ERR_SHAPE, "NVFP4 output of the prefill projection: the shard's columns do not fit the given width.");
    }
    if ((reinterpret_cast<uintptr_t>(qout->codes) & 7u) != 0) {
      return fail(Q35B_ERR_ARGUMENT, "NVFP4 prefill projection buffers must be 16-byte aligned.");
    }
  }
  if (residual_bf16 != nullptr && (w->gate_up || ldr < w->rows)) {
    return fail(Q35B_ERR_ARGUMENT, "Invalid residual for NVFP4 prefill projection.");
  }
  GemmEpilogue ep;
  ep.s2 = w->s2;
  ep.s2_up = w->s2_up;
  ep.gate_up = w->gate_up ? 1 : 0;
  ep.residual = static_cast<const __nv_bfloat16 *>(residual_bf16);
  ep.ldr = ldr;
  if (qout != nullptr) {
    ep.q_codes = qout->codes + w->row_begin / 4;   // two output columns per byte, two weight rows per output column
    ep.q_scales = qout->scales_tiled;
    ep.q_g = qout->g_dev;
    ep.q_slots = round_up_int(qout->total_cols / 16, 4);
    ep.q_ld = qout->total_cols / 2;
    ep.q_slot0 = w->row_begin / 32;
  }
  if (gather != nullptr) {
    static_assert(sizeof(gather->peer_c) / sizeof(gather->peer_c[0]) == GemmEpilogue::kMaxPeers, "peer table size");
    if (qout != nullptr || residual_bf16 != nullptr) return fail(Q35B_ERR_ARGUMENT, "The gathering NVFP4 prefill projection takes no residual and writes BF16.");
    ep.n_peers = gather->n_peers;
    for (int i = 0; i < gather->n_peers; ++i) {
      ep.peer_c[i] = static_cast<__nv_bfloat16 *>(gather->peer_c[i]);
      ep.peer_flag[i] = gather->peer_flag[i];
    }
    ep.done_counter = gather->done_counter;
    ep.epoch = gather->epoch;
    ep.send_seq = gather->send_seq;
    // whole-row forwarding moves aligned 32-byte pieces; any other geometry takes the per-lane peer stores
    bool aligned = (ldc % 16) == 0 && (out_cols % 16) == 0 && (reinterpret_cast<uintptr_t>(c_bf16) & 31u) == 0;
    for (int i = 0; i < gather->n_peers; ++i) aligned = aligned && (reinterpret_cast<uintptr_t>(gather->peer_c[i]) & 31u) == 0;
    ep.forward_rows = aligned ? 1 : 0;
  }
  if ((w->k % 64) != 0) return fail(Q35B_ERR_SHAPE, "NVFP4 W4A4 GEMM needs cols to be a multiple of 64.");
  if ((reinterpret_cast<uintptr_t>(a_codes) & 15u) != 0 || (reinterpret_cast<uintptr_t>(a_scales_tiled) & 15u) != 0) {
    return fail(Q35B_ERR_ARGUMENT, "NVFP4 prefill projection buffers must be 16-byte aligned.");
  }
  if (w->rows == 0) return Q35B_OK;
  if (const int st = check_weight_device(w)) return st;
  if (!w->has_maps) return fail(Q35B_ERR_ARGUMENT, "NVFP4 weight has no tensor maps (it was not built by q35b_weight_create*).");
  if (status_dev == nullptr) {
    // the library's own word: kernels only ever write a nonzero code into it, q35b_gemm_default_status reads and
    // clears it (no memset in front of the launch: it would sit between this kernel and the one it overlaps with)
    if (const int st = default_status_word(&status_dev)) return st;
  }
  const bool rows_aligned = qout != nullptr || ((ldc % 16) == 0 && (reinterpret_cast<uintptr_t>(c_bf16) & 31u) == 0 &&
                            (residual_bf16 == nullptr || ((ldr % 8) == 0 && (reinterpret_cast<uintptr_t>(residual_bf16) & 15u) == 0)));
  const GemmPlan plan = plan_gemm(m, w->rows, w->n_total, w->k, sm_count(), gather != nullptr, rows_aligned);
  if (plan.pairs) return launch_gemm_w4a4_2cta(w, a_codes, a_scales_tiled, g_dev, m, c_bf16, ldc, ep, status_dev, s);
  return launch_gemm_ksplit(w, a_codes, a_scales_tiled, g_dev, m, c_bf16, ldc, ep, plan, status_dev, s);
}

int launch_project_prefill(const q35b_weight * w, const void * x, bool f32, int m, float global_scale, uint8_t * codes, uint8_t * scales_tiled, float * g_dev,
                           void * workspace, const void * residual_bf16, int ldr, void * c_bf16, int ldc, unsigned int * status_dev, cudaStream_t s) {
  // One launch where the operand is made in shared memory (gemm_resident.cu); whatever is not in order goes the general way,
  // which says so.  So does a call whose output or scratch lies over the activations: in one launch some CTAs store while others
  // still read x, of two the first has read all of it.
  auto apart = [&](const void * written, size_t bytes) {
    const auto a = reinterpret_cast<uintptr_t>(x), b = reinterpret_cast<uintptr_t>(written);
    return a + static_cast<size_t>(m) * w->k * (f32 ? 4 : 2) <= b || b + bytes <= a;
  };
  auto aligned = [](const void * p) { return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (w != nullptr && m >= 1 && m <= kSplitTokens && w->rows > 0 && w->has_maps && (w->k % 64) == 0 && aligned(x) && aligned(codes) && aligned(scales_tiled) && g_dev != nullptr &&
      (global_scale > 0.0f || workspace != nullptr) && c_bf16 != nullptr && ldc >= (w->gate_up ? w->rows / 2 : w->rows) &&
      (residual_bf16 == nullptr || (!w->gate_up && ldr >= w->rows))) {
    const GemmPlan plan = plan_gemm(m, w->rows, w->n_total, w->k, sm_count(), false, true);
    int stages = 0, smem = 0;
    if (!plan.pairs && plan.tile_cols >= m && prefill_resident_shape(w, m, global_scale, plan.split, &stages, &smem) &&
        apart(c_bf16, (static_cast<size_t>(m - 1) * ldc + (w->gate_up ? w->rows / 2 : w->rows)) * 2) &&
        apart(codes, q35b_act_codes_bytes(m, w->k)) && apart(scales_tiled, q35b_act_scales_bytes(m, w->k))) {
      if (const int st = check_weight_device(w)) return st;
      if (status_dev == nullptr) {
        if (const int st = default_status_word(&status_dev)) return st;
      }
      return launch_prefill_resident(w, x, f32, m, codes, scales_tiled, g_dev, plan.split, stages, smem, residual_bf16, ldr, c_bf16, ldc, status_dev, s);
    }
  }
  const int k = w != nullptr ? w->k : 0;
  if (const int st = f32 ? launch_quantize_f32(static_cast<const float *>(x), m, k, global_scale, codes, scales_tiled, g_dev, workspace, s)
                         : launch_quantize_bf16(x, m, k, global_scale, codes, scales_tiled, g_dev, workspace, s)) {
    return st;
  }
  return launch_gemm_w4a4(w, codes, scales_tiled, g_dev, m, c_bf16, ldc, residual_bf16, ldr, status_dev, s);
}

}  // namespace q35b
