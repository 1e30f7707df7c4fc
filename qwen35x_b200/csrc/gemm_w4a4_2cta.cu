// W4A4 prefill GEMM, 2-CTA persistent variant for sm_100a.
//
// Same contract as gemm_w4a4_tcgen05.cu (C[M,N] bf16 = (Aq . Wq^T) * g * s2, replacing
// run_nvfp4_cublaslt_prefill_projection_device, src/runtime/cuda_bench.cu:1056-1167), built for large M:
//
//   - a pair of CTAs on neighbouring SMs (cluster of 2) computes one 256 x 256 output tile with
//     tcgen05.mma.cta_group::2: each CTA stages only its own 128 rows of A and its own 128 rows of B.  No TMA
//     multicast is used: every load lands in the issuing CTA's own shared memory;
//   - persistent: 74 pairs walk the tile list (M-tiles fastest, so the pairs in flight share B tiles in L2);
//     barriers, TMEM and tensor maps are set up once per CTA, not once per tile;
//   - per K step (256 FP4 columns) a CTA lands A 16 KB + B 16 KB (128B-swizzled TMA boxes) and the scale
//     factors SFA 2 KB + SFB 4 KB (TMA boxes over the 512-byte scale tiles); 5-stage ring;
//   - the leader CTA's MMA thread copies scale factors to TMEM in both CTAs (tcgen05.cp.cta_group::2) and
//     issues four M=256, N=256, K=64 block-scaled MMAs per K step; tcgen05.commit multicasts stage release and
//     accumulator-ready to both CTAs;
//   - two accumulators alternate, so that a tile's MMAs run while the one before is converted and stored.  Beside 48
//     columns of scale factors 512 columns of TMEM do not hold two of 256: the second starts at column 208 and shares 48
//     with the first (OVERLAP below).  The 64 columns that hold them are read out of a tile first, and the next tile's MMAs
//     wait for these alone; all others have a tile's time to leave.
//
// What bounds it: the power cap.  At [4096, 2560] x [18432, 2560] the SM clock falls to 1.5 GHz within a millisecond and to
// 1.35 GHz in a loop.  A K step takes some 560 cycles (542 at the tensor cores' nominal rate); with one accumulator 1900 of a
// tile's 8300 cycles went by between its last MMA and the next tile's first one.
//
// Every mbarrier wait is bounded; an expired wait records a code in *status and the role stops, the kernel
// still runs to its cluster barrier and frees TMEM.
#include <cuda_bf16.h>

#include "engine.h"
#include "gemm_epilogue.cuh"
#include "nvfp4_codec.cuh"

namespace q35b {
namespace {

constexpr int kCtaRows = 128;            // rows of A staged per CTA
constexpr int kTileM = 256;              // output tile of the pair: 256 tokens ...
constexpr int kTileN = 256;              // ... by 256 weight rows
constexpr int kCtaBRows = kTileN / 2;    // rows of B staged per CTA
constexpr int kStepBytes = 128;          // 256 FP4 columns
constexpr int kMmaPerStage = 4;
constexpr int kSfChunk = 512;
constexpr int kABytes = kCtaRows * kStepBytes;
constexpr int kBBytes = kCtaBRows * kStepBytes;
constexpr int kSfaBytes = kMmaPerStage * kSfChunk;
constexpr int kSfbBytes = 2 * kMmaPerStage * kSfChunk;
constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;   // 38912
constexpr int kStages = 5;
// Epilogue warps per CTA (template parameter of the kernel), a multiple of four: kEpilogueWarps / 4 per TMEM lane
// quarter, which take turns at the 32-column chunks of the accumulator.  Eight for the plain and the residual epilogue,
// whose chunks leave through shared memory as TMA boxes of 32 x 32 values, two per warp in turn; sixteen for the epilogues that do
// arithmetic on what they drain (SiLU, NVFP4 output) and for launches that forward rows to peers, which store per lane.
// Either is a loop of few instructions: unrolled over the chunks it fetched them anew for every tile, 3900 cycles for 128
// columns, and pushed the MMA issuer's out of the instruction cache.  With loop and boxes [4096, 2560] x [18432, 2560] went
// from 81.5 to 80.5 us, and quantise + GEMM in a loop at the power cap from 113.3 to 110.7.
constexpr int kEpiWarpsWide = 16;
constexpr int kEpiWarpsPlain = 8;
constexpr int kChunkCols = 32;
constexpr int kChunks = kTileN / kChunkCols;
constexpr int kBoxBytes = 32 * kChunkCols * 2;
constexpr int kBoxOffset = kStages * kStageBytes + 512;  // of the boxes, behind the barriers; the swizzle repeats every 512 bytes
constexpr int kSmemBytes = 1024 + kBoxOffset;
constexpr int kSmemBytesPlain = kSmemBytes + kEpiWarpsPlain * 2 * kBoxBytes;
static_assert(kSmemBytesPlain <= 227 * 1024 && kBoxOffset % 512 == 0, "shared memory");
constexpr int kSfaCols = kMmaPerStage * 4;
constexpr int kSfbCols = kMmaPerStage * 8;
constexpr int kTmemCols = 512;
// OVERLAP: the second accumulator ends where the scale factors begin.
constexpr int kAcc1 = kTmemCols - kSfaCols - kSfbCols - kTileN;  // its first column, 208
static_assert(kAcc1 < kTileN && kTileN - kAcc1 <= 2 * kChunkCols, "the shared columns lie in the first accumulator's last two chunks and the second one's first two");
constexpr uint32_t kWaitLimit = 1u << 20;
constexpr uint32_t kPeerMask = 0xFEFFFFFFu;  // clears the CTA-rank bit of a shared::cluster address: the pair's leader

enum StatusCode : unsigned { kProducerWait = 21, kMmaWait = 22, kEpilogueWait = 23, kMmaDrainWait = 24 };

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Arrive on the barrier at this offset in the pair's leader.  What it tells is that registers hold what TMEM held
// (tcgen05.wait::ld), so no scope beyond the CTA is asked for: with .release.cluster the arrival waits for the output
// stores under way, 1400 cycles in which the tensor cores had nothing to do.
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar & kPeerMask) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < kWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
    if (ok) return true;
  }
  return false;
}
// TMA box load into this CTA's shared memory, completion bytes go to the pair leader's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap * map, uint32_t leader_bar, int x, int y) {
  asm volatile(
    "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
      "r"(dst),
    "l"(map), "r"(leader_bar), "r"(x), "r"(y)
    : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap * map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
               "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap * map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
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
__device__ __forceinline__ uint64_t desc_k_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
__device__ __forceinline__ uint64_t desc_sf(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(128 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}
// kind::mxf4nvf4 instruction descriptor: E2M1 x E2M1, K-major, UE4M3 scales, M = 256 (pair), N = 256.
__device__ __forceinline__ uint32_t instr_desc_pair() {
  uint32_t d = 0;
  d |= 1u << 7;
  d |= 1u << 10;
  d |= static_cast<uint32_t>(kTileN >> 3) << 17;
  d |= static_cast<uint32_t>(kTileM >> 4) << 24;
  return d;
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t tmem_sfa,
                                          uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "setp.ne.b32 p, %4, 0;\n\t"
    "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
    : "memory");
}
__device__ __forceinline__ void utccp_sf_pair(uint32_t tmem_dst, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(sdesc) : "memory");
}
// Arrive (once all earlier tcgen05 work of this thread has retired) on the barrier at this offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
      "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
      "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
    : "r"(taddr)
    : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The first `count` (up to eight) of eight BF16 values into 16-byte aligned memory.
__device__ __noinline__ void store_bf16_tail(__nv_bfloat16 * p, uint4 v, int count) {
  if (count >= 8) {
    *reinterpret_cast<uint4 *>(p) = v;
    return;
  }
  const uint64_t w[2] = {v.x | static_cast<uint64_t>(v.y) << 32, v.z | static_cast<uint64_t>(v.w) << 32};
  for (int i = 0; i < count; ++i) reinterpret_cast<unsigned short *>(p)[i] = static_cast<unsigned short>(w[i >> 2] >> (16 * (i & 3)));
}

template <int kEpilogueWarps>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((2 + kEpilogueWarps) * 32, 1)
gemm_w4a4_2cta_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                      const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_res,  // output and residual of the plain epilogue
                      const float * __restrict__ g_dev, const GemmEpilogue ep, int m, int n, int k_bytes, int m_tiles, int num_tiles,
                      __nv_bfloat16 * __restrict__ c, int ldc, unsigned int * status) {
  constexpr int kColWarps = kEpilogueWarps / 4, kTurns = kChunks / kColWarps;  // chunks of a tile that one epilogue warp takes
  static_assert(kEpilogueWarps % 4 == 0 && kColWarps >= 2 && kTurns * kColWarps == kChunks, "epilogue column split");
  extern __shared__ uint8_t smem_raw[];
  uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t * smem_a = smem;
  uint8_t * smem_b = smem_a + kStages * kABytes;
  uint8_t * smem_sfa = smem_b + kStages * kBBytes;
  uint8_t * smem_sfb = smem_sfa + kStages * kSfaBytes;
  uint64_t * bars = reinterpret_cast<uint64_t *>(smem_sfb + kStages * kSfbBytes);
  uint64_t * full = bars;                       // used in the leader: bytes of both CTAs
  uint64_t * empty = bars + kStages;            // in each CTA: its own stages are free
  uint64_t * tmem_full = bars + 2 * kStages;    // in each CTA: the tile's accumulator is complete
  uint64_t * drained = tmem_full + 1;           // used in the leader: both CTAs' epilogue warps have read the columns that the next tile's accumulator shares
  uint64_t * res_full = drained + 1;            // [2 per epilogue warp of the plain epilogue]: the residual's box has landed
  uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(res_full + 2 * kEpiWarpsPlain);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int sf_col_blocks = k_bytes >> 5;
  const int k_steps = (sf_col_blocks + kMmaPerStage - 1) / kMmaPerStage;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(full + i), 1);
      mbar_init(smem_u32(empty + i), 1);
    }
    mbar_init(smem_u32(tmem_full), 1);
    mbar_init(smem_u32(drained), 2 * kEpilogueWarps);
    for (int i = 0; i < 2 * kEpiWarpsPlain; ++i) mbar_init(smem_u32(res_full + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // both CTAs' barriers exist before anything signals across the pair
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_acc = tmem_base;
  const uint32_t tmem_sfa = tmem_base + kAcc1 + kTileN;
  const uint32_t tmem_sfb = tmem_sfa + kSfaCols;
  // Launched with programmatic stream serialisation: everything above (barriers, TMEM, the pair's rendezvous) may run
  // under the tail of the previous kernel; nothing below touches global memory before that kernel is complete.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // An error recorded by an earlier launch: run no tiles (every CTA still goes through alloc, barriers, dealloc).
  const bool aborted = *reinterpret_cast<volatile unsigned int *>(status) != 0u;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (elect_one() && !aborted) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        const int tm = tile % m_tiles;
        const int tn = tile / m_tiles;
        const int a_row = tm * kTileM + static_cast<int>(rank) * kCtaRows;
        const int b_row = tn * kTileN + static_cast<int>(rank) * kCtaBRows;
        const int sfa_chunk0 = (tm * 2 + static_cast<int>(rank)) * sf_col_blocks;
        const int sfb_rb = (tn * kTileN) >> 7;  // first of the two 128-row scale tiles
        const int sfb_chunk0 = sfb_rb * sf_col_blocks;
        const int sfb_chunk1 = (sfb_rb + 1) * sf_col_blocks;
        // The weights of the pair's next tile come from HBM, where they queue up behind the output that is being written (waits
        // of up to 1700 cycles, longer than the ring): into L2 with them now, the K steps shared out among the pairs that
        // will read them.  With the order of waits in the MMA issuer 80.5 -> 75.4 us.
        if (const int next = tile + num_pairs; next < num_tiles) {
          const int next_row = next / m_tiles * kTileN;
          for (int ks = next % m_tiles; ks < k_steps; ks += m_tiles) {
            tma_prefetch_2d(&tmap_b, ks * kStepBytes, next_row + static_cast<int>(rank) * kCtaBRows);
            tma_prefetch_2d(&tmap_sfb, 0, ((next_row >> 7) + static_cast<int>(rank)) * sf_col_blocks + ks * kMmaPerStage);
          }
        }
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!mbar_wait(smem_u32(empty + stage), phase ^ 1)) {
            atomicExch(status, kProducerWait);
            ok = false;
            break;
          }
          const uint32_t leader_full = smem_u32(full + stage) & kPeerMask;
          if (rank == 0) mbar_expect_tx(smem_u32(full + stage), 2 * kStageBytes);
          tma_load_2d_pair(smem_u32(smem_a + stage * kABytes), &tmap_a, leader_full, ks * kStepBytes, a_row);
          tma_load_2d_pair(smem_u32(smem_b + stage * kBBytes), &tmap_b, leader_full, ks * kStepBytes, b_row);
          tma_load_2d_pair(smem_u32(smem_sfa + stage * kSfaBytes), &tmap_sfa, leader_full, 0, sfa_chunk0 + ks * kMmaPerStage);
          tma_load_2d_pair(smem_u32(smem_sfb + stage * kSfbBytes), &tmap_sfb, leader_full, 0, sfb_chunk0 + ks * kMmaPerStage);
          tma_load_2d_pair(smem_u32(smem_sfb + stage * kSfbBytes + kSfaBytes), &tmap_sfb, leader_full, 0,
                           sfb_chunk1 + ks * kMmaPerStage);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (rank == 0 && elect_one() && !aborted) {
      const uint32_t idesc = instr_desc_pair();
      int stage = 0;
      uint32_t phase = 0;
      uint32_t li = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++li) {
        const uint32_t acc = tmem_acc + (li & 1) * kAcc1;
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!mbar_wait(smem_u32(full + stage), phase)) {
            atomicExch(status, kMmaWait);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int valid = min(kMmaPerStage, sf_col_blocks - ks * kMmaPerStage);
          // descriptors of this stage: the address field counts 16-byte units, so stepping a descriptor is an add
          const uint64_t a_desc = desc_k_sw128(smem_u32(smem_a + stage * kABytes));
          const uint64_t b_desc = desc_k_sw128(smem_u32(smem_b + stage * kBBytes));
          const uint64_t sfa_desc = desc_sf(smem_u32(smem_sfa + stage * kSfaBytes));
          const uint64_t sfb_desc = desc_sf(smem_u32(smem_sfb + stage * kSfbBytes));
#pragma unroll
          for (int j = 0; j < kMmaPerStage; ++j) {
            if (j < valid) {
              utccp_sf_pair(tmem_sfa + j * 4, sfa_desc + j * (kSfChunk >> 4));
              utccp_sf_pair(tmem_sfb + j * 8, sfb_desc + j * (kSfChunk >> 4));
              utccp_sf_pair(tmem_sfb + j * 8 + 4, sfb_desc + (kSfaBytes >> 4) + j * (kSfChunk >> 4));
            }
          }
          // the scale factors are on their way; the shared columns of the tile before are read out, and with them all of
          // the one before that
          if (ks == 0) {
            if (!mbar_wait(smem_u32(drained), (li & 1) ^ 1)) {
              atomicExch(status, kMmaDrainWait);
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
#pragma unroll
          for (int j = 0; j < kMmaPerStage; ++j) {
            if (j < valid) {
              umma_pair(acc, a_desc + j * 2, b_desc + j * 2, idesc, tmem_sfa + j * 4, tmem_sfb + j * 8,
                        (ks | j) != 0 ? 1u : 0u);
            }
          }
          umma_commit_pair(smem_u32(empty + stage));
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(smem_u32(tmem_full));
      }
    }
  } else {
    // ---------------- epilogue (both CTAs): this CTA's 128 rows of the pair's tile ----------------
    const int quarter = warp & 3;                 // TMEM lanes 32 * quarter .. + 31 (fixed by the warp's index)
    const int col_warp = (warp - 2) >> 2;
    const float g = __ldcg(g_dev);
    const float alpha = g * ep.s2;
    GemmQuantScale q;
    if constexpr (kEpilogueWarps == kEpiWarpsWide) {
      __shared__ float q_table[128];
      if (ep.q_codes != nullptr) {
        q.g = __ldcg(ep.q_g);
        q.rg = __frcp_rn(q.g);
        q.table = q_table;
        const int at = threadIdx.x - 64;
        if (at < 127) q_table[at] = bf16_block_multiplier(at, q.g);
        asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueWarps * 32) : "memory");  // the epilogue warps only
      }
    }
    uint32_t li = 0;
    bool ok = !aborted;
    int res_loads = 0;  // lane 0: residual boxes asked for
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++li) {
      const int tm = tile % m_tiles;
      const int tn = tile / m_tiles;
      const int row0 = tm * kTileM + static_cast<int>(rank) * kCtaRows + quarter * 32;
      const uint32_t taddr = tmem_acc + (li & 1) * kAcc1 + (static_cast<uint32_t>(quarter * 32) << 16);
      // the chunks with the shared columns come first: the last two of the first accumulator, the first two of the second
      const int chunk0 = (li & 1) != 0u ? col_warp : col_warp + kChunks - 2;
      if constexpr (kEpilogueWarps == kEpiWarpsPlain) {
        const uint32_t box0 = smem_u32(smem + kBoxOffset) + (warp - 2) * 2 * kBoxBytes;
#pragma unroll 1
        for (int turn = 0; turn < kTurns; ++turn) {
          const int chunk = (chunk0 + turn * kColWarps) & (kChunks - 1);
          const int col0 = tn * kTileN + chunk * kChunkCols;
          // The residual's boxes come by TMA into the boxes that the sums leave from, each while the one before is worked on;
          // the first one of a tile under the tile before.
          auto load_residual = [&](int at_tile, int at_turn, uint32_t at_li) {
            const int at_chunk = (col_warp + ((at_li & 1) != 0u ? 0 : kChunks - 2) + at_turn * kColWarps) & (kChunks - 1);
            const uint32_t at_box = box0 + (at_turn & 1) * kBoxBytes, bar = smem_u32(res_full + 2 * (warp - 2) + (at_turn & 1));
            ++res_loads;
            mbar_expect_tx(bar, kBoxBytes);
            tma_load_2d(at_box, &tmap_res, bar, at_tile / m_tiles * kTileN + at_chunk * kChunkCols,
                        at_tile % m_tiles * kTileM + static_cast<int>(rank) * kCtaRows + quarter * 32);
          };
          if (ep.residual != nullptr && lane == 0) {
            if (li == 0 && turn == 0) load_residual(tile, 0, 0);
            // the box after this one: its last store has been read
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            if (turn + 1 < kTurns) {
              load_residual(tile, turn + 1, li);
            } else if (tile + num_pairs < num_tiles) {
              load_residual(tile + num_pairs, 0, li + 1);
            }
          }
          if (turn == 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(tmem_full), li & 1));  // the whole warp goes on, or none of it
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          uint32_t r[32];
          tmem_ld32(taddr + chunk * kChunkCols, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (turn == 0) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(smem_u32(drained));
          }
          const uint32_t box = box0 + (turn & 1) * kBoxBytes;
          if (ep.residual != nullptr) {
            ok = mbar_wait(smem_u32(res_full + 2 * (warp - 2) + (turn & 1)), (li * (kTurns / 2) + turn / 2) & 1);
            if (!__all_sync(0xffffffffu, ok)) {
              ok = false;
              break;
            }
          } else {
            // the box before last has been read
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
          }
          const bool whole = col0 + kChunkCols <= n;  // a box that is cut off in the middle of 16 bytes writes them all
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // 64-byte swizzle: eight lanes' pieces lie in eight different sixteenths of the 128-byte span of the banks
            const uint32_t piece = box + lane * 64 + ((i ^ (lane >> 1 & 3)) << 4);
            uint32_t rw[4] = {0u, 0u, 0u, 0u}, p[4];
            if (ep.residual != nullptr) {
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(rw[0]), "=r"(rw[1]), "=r"(rw[2]), "=r"(rw[3]) : "r"(piece) : "memory");
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              p[e] = pack_bf16(fmaf(__uint_as_float(r[8 * i + 2 * e]), alpha, __uint_as_float(rw[e] << 16)),
                               fmaf(__uint_as_float(r[8 * i + 2 * e + 1]), alpha, __uint_as_float(rw[e] & 0xffff0000u)));
            }
            if (!whole) {
              if (row0 + lane < m && col0 + 8 * i < n) store_bf16_tail(c + static_cast<size_t>(row0 + lane) * ldc + col0 + 8 * i, make_uint4(p[0], p[1], p[2], p[3]), n - col0 - 8 * i);
              continue;
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(piece), "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]) : "memory");
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            // rows past m are not written
            if (whole && row0 < m) {
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&tmap_c), "r"(box), "r"(col0), "r"(row0) : "memory");
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      } else {
        // plain BF16 output of a gathering launch: store locally, then forward whole rows, whose chunks are neighbours then;
        // the fused epilogues (and a launch without peers) store per lane
        const bool forward = ep.n_peers > 0 && !ep.gate_up && ep.forward_rows != 0;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(tmem_full), li & 1));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int turn = 0; turn < kTurns; ++turn) {
          const int chunk = forward ? col_warp * kTurns + turn : (chunk0 + turn * kColWarps) & (kChunks - 1);
          uint32_t r[32];
          tmem_ld32(taddr + chunk * kChunkCols, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (turn == (forward ? kTurns - 1 : 0)) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(smem_u32(drained));
          }
          if (row0 + lane < m) gemm_store_chunk32(r, row0 + lane, tn * kTileN + chunk * kChunkCols, n, g, ep, c, ldc, !forward, q);
          __syncwarp();
        }
        if (forward) gemm_forward_rows_to_peers<kTurns * kChunkCols>(ep, c, ldc, row0, m, tn * kTileN + col_warp * kTurns * kChunkCols, n, lane);
      }
    }
    if (!ok && !aborted && lane == 0) atomicExch(status, kEpilogueWait);
    // the boxes stay until they have been stored, and until what was asked for has landed
    if (!ok) {
      for (int i = max(res_loads - 2, 0); i < res_loads; ++i) mbar_wait(smem_u32(res_full + 2 * (warp - 2) + (i & 1)), i >> 1 & 1);
    }
    if (kEpilogueWarps == kEpiWarpsPlain && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  gemm_signal_peers(ep, status);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // neither CTA may leave while its partner can still signal its barriers or read its tiles
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
  }
}

}  // namespace

namespace {
int encode_map(CUtensorMap * map, CUtensorMapDataType type, const void * base, cuuint64_t inner, cuuint64_t outer, cuuint64_t stride, cuuint32_t box_inner,
               cuuint32_t box_outer, CUtensorMapSwizzle swizzle, const char * what) {
  using Fn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                          const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                          CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Fn fn = nullptr;
  if (fn == nullptr) {
    void * p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
      return fail(Q35B_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the CUDA driver.");
    }
    fn = reinterpret_cast<Fn>(p);
  }
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {stride};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(map, type, 2, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    return fail(Q35B_ERR_CUDA, std::string("cuTensorMapEncodeTiled(") + what + ") failed with CUresult " + std::to_string(static_cast<int>(r)) + ".");
  }
  return Q35B_OK;
}

// 2-D map over the BF16 output or residual [m, n] with rows ldc apart: boxes of 32 x 32 values.
int make_output_map(CUtensorMap * map, const void * c, int m, int n, int ldc) {
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, c, static_cast<cuuint64_t>(n), static_cast<cuuint64_t>(m), static_cast<cuuint64_t>(ldc) * 2,
                    kChunkCols, 32, CU_TENSOR_MAP_SWIZZLE_64B, "output");
}
}  // namespace

// 2-D map over a tiled scale array seen as [chunks, 128 x u32]: box = 4 consecutive 512-byte chunks.
int make_sf_map(CUtensorMap * map, const void * base, long long chunks) {
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, base, 128, static_cast<cuuint64_t>(chunks), 512, 128, 4, CU_TENSOR_MAP_SWIZZLE_NONE, "scale factors");
}

int build_weight_maps(q35b_weight * w) {
  if (w->rows <= 0 || (w->k % 64) != 0) return Q35B_OK;  // such a weight never reaches a GEMM
  if (const int st = make_code_map(&w->tmap_codes_128, w->codes, w->rows, w->k / 2, 128)) return st;
  if (const int st = make_code_map(&w->tmap2_codes, w->codes, w->rows, w->k / 2, kCtaBRows)) return st;
  const long long chunks = static_cast<long long>((w->rows + 127) / 128) * (w->k / 64);
  if (const int st = make_sf_map(&w->tmap2_sf, w->scales_tiled, chunks)) return st;
  w->has_maps = true;
  return Q35B_OK;
}

bool gemm_2cta_eligible(int rows, int m, int k) { return rows >= 192 && m >= 256 && (k % 64) == 0; }

int launch_gemm_w4a4_2cta(const q35b_weight * w, const uint8_t * a_codes, const uint8_t * a_scales_tiled, const float * g_dev,
                          int m, void * c_bf16, int ldc, const GemmEpilogue & ep, unsigned int * status_dev,
                          cudaStream_t s) {
  static std::atomic<bool> attr_set[64];
  if (!attr_set[w->device & 63].load(std::memory_order_acquire)) {
    Q35B_CUDA_TRY(cudaFuncSetAttribute(gemm_w4a4_2cta_kernel<kEpiWarpsWide>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes),
                  "cudaFuncSetAttribute(2-CTA gemm smem)");
    Q35B_CUDA_TRY(cudaFuncSetAttribute(gemm_w4a4_2cta_kernel<kEpiWarpsPlain>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytesPlain),
                  "cudaFuncSetAttribute(2-CTA gemm smem)");
    attr_set[w->device & 63].store(true, std::memory_order_release);
  }
  CUtensorMap tmap_a, tmap_sfa;
  if (const int st = make_code_map(&tmap_a, a_codes, m, w->k / 2, kCtaRows)) return st;
  if (const int st = make_sf_map(&tmap_sfa, a_scales_tiled, static_cast<long long>((m + 127) / 128) * (w->k / 64))) return st;
  const int m_tiles = (m + kTileM - 1) / kTileM;
  const int n_tiles = (w->rows + kTileN - 1) / kTileN;
  const int num_tiles = m_tiles * n_tiles;
  const int pairs = std::max(1, std::min(num_tiles, sm_count() / 2));
  // plain and residual epilogues without peers whose rows a TMA box can be stored to
  const bool plain = !ep.gate_up && ep.q_codes == nullptr && ep.n_peers == 0 && (ldc % 8) == 0 && (reinterpret_cast<uintptr_t>(c_bf16) & 15u) == 0 &&
                     (ep.residual == nullptr || ((ep.ldr % 8) == 0 && (reinterpret_cast<uintptr_t>(ep.residual) & 15u) == 0));
  CUtensorMap tmap_c = tmap_a, tmap_res = tmap_a;
  if (plain) {
    if (const int st = make_output_map(&tmap_c, c_bf16, m, w->rows, ldc)) return st;
    if (ep.residual != nullptr) {
      if (const int st = make_output_map(&tmap_res, ep.residual, m, w->rows, ep.ldr)) return st;
    }
  }
  const int epi_warps = plain ? kEpiWarpsPlain : kEpiWarpsWide;
  const auto kernel = plain ? gemm_w4a4_2cta_kernel<kEpiWarpsPlain> : gemm_w4a4_2cta_kernel<kEpiWarpsWide>;
  const cudaError_t le = launch_pdl(kernel, dim3(2 * pairs), dim3((2 + epi_warps) * 32), plain ? kSmemBytesPlain : kSmemBytes, s, tmap_a, w->tmap2_codes,
                                    tmap_sfa, w->tmap2_sf, tmap_c, tmap_res, g_dev, ep, m, w->rows, w->k / 2, m_tiles, num_tiles,
                                    static_cast<__nv_bfloat16 *>(c_bf16), ldc, status_dev);
  count_launch();
  Q35B_CUDA_TRY(le, "gemm_w4a4_2cta_kernel launch");
  return Q35B_OK;
}

}  // namespace q35b
