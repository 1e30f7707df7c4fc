// Projections of few tokens whose whole operand is made and kept in shared memory, for sm_100a: one launch from BF16 or fp32
// activations to outputs.
//
// Weight rows are the 128-row tensor-core operand as in gemm_w4a4_tcgen05.cu and gemm_wstream.cu, streamed through a ring that
// fills before griddepcontrol.wait, K split over a cluster of up to eight CTAs.  The other operand does not come from memory:
// every CTA reads its columns of the activations and makes it itself,
//
//   W4A4    NVFP4 codes and block scales.  A cluster covers all of K, so with one token tile the tensor's amax is the largest of
//           its CTAs' maxima, exchanged over distributed shared memory: no meeting of the grid, no second launch.  The codes,
//           scales and scale word also go to the caller's scratch, K steps dealt out over the clusters.
//   W4A16   octal digits (digits.cuh), eight rows per token and six of deep digits, which are multiplied only where the CTA's
//           columns have some.  A token is counted against the largest exponent in the CTA's columns, whose power of two the
//           sums are multiplied with before they are sent.  What fourteen digits leave of a value (which has to be some 2^-33 of
//           its block's largest, or less) the epilogue adds in fp32: nothing of an activation is lost.
//
// The partial sums are pushed into the shared memory of the CTA that stores them (it owns some of the tile's 16-row groups),
// so that behind the cluster barrier there are only local reads.
//
// What bounds it: latency, a chain of about half a microsecond each: activations from L2, the operand, a quarter of a
// microsecond per K step (eight scale copies and four MMAs), the sums' way out of TMEM and over the cluster, the stores, and one
// microsecond until the next kernel's griddepcontrol.wait returns.  The operand is made anew by every row block, so this pays
// only where a CTA's share of it is small (the rules at the launchers).
//
// Every wait is bounded; an expired one records a code in *status, the cluster stores nothing, and the CTA waits (again with a
// limit) for what it has under way.  `wait_limit` is that of the waits for copies, operand and maxima; the sums are always sent, and
// waited for with the longer limit.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "digits.cuh"
#include "engine.h"
#include "gemm_epilogue.cuh"
#include "nvfp4_codec.cuh"
#include "nvfp4_quant_block.cuh"

namespace q35b {
namespace {

constexpr int kRows = 128;               // weight rows per tile (UMMA M)
constexpr int kStepBytes = 128;          // 256 FP4 columns of K per ring stage
constexpr int kMmaPerStage = 4;          // K = 64 per MMA
constexpr int kSfChunk = 512;            // scale factors of 128 rows x 64 columns
constexpr int kABytes = kRows * kStepBytes;
constexpr int kSfBytes = kMmaPerStage * kSfChunk;
constexpr int kMaxStages = 8;
constexpr int kMaxSplit = 8;
constexpr int kMakers = 14;              // warps 2..15 make the operand; warp 0 loads weights, warp 1 issues MMAs; all store
constexpr int kMakerThreads = kMakers * 32;
constexpr int kThreads = 64 + kMakerThreads;
constexpr int kGroupRows = 16;           // rows of a tile that one CTA of the cluster stores together (8 gate / 8 up)
constexpr int kGroups = kRows / kGroupRows;
constexpr int kAccCols = 192;            // accumulators, up to four partial ones side by side ...
constexpr int kSfSetCols = 32;           // ... and two sets of scale-factor columns, used by stages in turn
constexpr int kTmemCols = 256;
constexpr int kFixedBytes = 1024 /*alignment slack*/ + 256 /*barriers*/;
constexpr int kSmemHalf = 110 * 1024, kSmemFull = 220 * 1024;  // two CTAs per SM where they fit, or one
constexpr uint32_t kWaitLimit = 1u << 20;
constexpr uint32_t kDrainLimit = 1u << 20;

enum StatusCode : unsigned { kWeightWait = 51, kMmaWait = 52, kOperandWait = 53, kEpilogueWait = 54, kAmaxWait = 55, kSumsWait = 56 };
enum Op : int { kDigits = 0, kNvfp4Bf16 = 1, kNvfp4F32 = 2 };

struct ResidentArgs {
  const uint8_t * w_scales;        // weight scale tiles
  const uint8_t * w_codes;         // W4A16: for infinite activations
  const void * x;                  // [m, k]
  __nv_bfloat16 * y;
  const __nv_bfloat16 * residual;  // NULL or [m, ldr]
  int ldy, ldr;
  int m, n, k;
  // K steps of the cluster's CTAs, the 16-row groups of a tile that they store, and which one stores a group: worked out by the
  // host, since a division by a number that the compiler does not know takes as long as the loads it is waited for with
  short step_begin[kMaxSplit + 1], group_begin[kMaxSplit + 1], group_owner[kGroups];
  int most_steps;
  int stages, cols_plain, cols_deep;  // ring stages; operand rows (UMMA N) without and with the deep digits
  int sf_cols;                     // TMEM columns of operand scales per MMA: 32 rows each (2 or 4)
  float s2, s2_up;
  int gate_up;
  // what the launch after this one will stream, to be brought into L2 under this one (or NULL)
  const uint8_t * next_codes, * next_scales;
  unsigned long long next_codes_bytes, next_scales_bytes;
  uint32_t next_codes_share, next_scales_share;  // of a CTA
  // Of a chain: two words of this launch and of the one before it (or NULL).  The first is set where a CTA gives up; then the
  // launch after it stores nothing, since what it would read may be an earlier run's, and sets its own.  Its CTAs count themselves
  // in the second, and the last one clears both for the next run.  Otherwise a launch reads a word that nobody writes (a word per
  // CTA, written in every run, cost half a microsecond of 10 to 18).
  unsigned int * gave, * before;
  int absent;                      // test hook: 1: in every other row block, the first included, the operand is never complete
  // W4A4: the caller's scratch
  uint8_t * codes, * scales;
  float * g_out;
  unsigned int * status;
  uint32_t wait_limit;
};

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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
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
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void makers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kMakerThreads) : "memory"); }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// A word into a CTA's shared memory, whose barrier counts its bytes.
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}

// A CTA's share of `bytes` (both multiples of 16) into L2.
__device__ __forceinline__ void prefetch_share(const uint8_t * p, uint32_t share, unsigned long long bytes, unsigned cta) {
  const unsigned long long begin = static_cast<unsigned long long>(share) * cta;
  for (unsigned long long at = begin; at < min(begin + share, bytes); at += 16384) {
    const uint32_t n = static_cast<uint32_t>(min(16384ull, min(begin + share, bytes) - at));
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + at), "r"(n) : "memory");
  }
}

// With few operand rows an MMA is far shorter than the tensor pipe's latency; the four of a stage go to different partial
// accumulators then, as many as fit.
__device__ __forceinline__ int partial_accumulators(int n_cols) { return 4 * n_cols <= kAccCols ? 4 : (2 * n_cols <= kAccCols ? 2 : 1); }

// W4A16: a token's 256 columns of one K step, of which a maker warp takes every fourteenth.
struct Unit {
  int token, it;
};
__device__ __forceinline__ Unit next_unit(Unit u, int steps) {
  u.it += kMakers;
  while (u.it >= steps) {
    u.it -= steps;
    ++u.token;
  }
  return u;
}

// Above this exponent field of the largest value the smallest BF16 values vanish in units of it, before there are digits.
constexpr int kTopUnderflows = 144;

// What the digits of a token's columns k0 .. k1 (k0 a multiple of 256) leave, times the weights of `row` of `rows` (one per lane),
// without the tensor's scale: 256 columns at a time a warp looks for values far enough below their block's largest one, makes
// their digits again and takes the products of the remainders.  It is for the few values that outliers leave behind.  [4096, 2560], four
// tokens, us: none 6.6, one value 7.1, one column in a hundred 19.3, all but an outlier per block 62; the rows kernel, which unpacks
// all weights, 9.1.
__device__ __noinline__ float left_dot(const uint8_t * w_codes, const uint8_t * w_scales, const __nv_bfloat16 * x_row, int rows, int k, int k0, int k1, int row,
                                       int top, int lane) {
  constexpr int kDigits14 = 8 + kDeepDigits;
  const bool live = row < rows;
  const uint8_t * codes = w_codes + static_cast<size_t>(live ? row : 0) * (k >> 1);
  const uint4 * x = reinterpret_cast<const uint4 *>(x_row);
  float sum = 0.0f;
#pragma unroll 1
  for (int base = k0 >> 3; base < k1 >> 3; base += 32) {
    const uint4 q = base + lane < k1 >> 3 ? __ldcg(x + base + lane) : make_uint4(0u, 0u, 0u, 0u);
    uint32_t b = bf16x8_abs_max(q);
    b = max(b, __shfl_xor_sync(0xffffffffu, b, 1));
    const int e = digits_exponent(b, top);
    const uint32_t r[4] = {q.x, q.y, q.z, q.w};
    uint32_t low = 0;  // bit i: value i has bits below the last digit's unit, or may have
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int magnitude = r[i >> 1] >> (16 * (i & 1)) & 0x7fffu;
      if (magnitude != 0 && max(magnitude >> 7, 1) + 3 * kDigits14 - 9 < e) low |= 1u << i;
    }
    uint32_t lanes = __ballot_sync(0xffffffffu, low != 0u);
    if (lanes == 0u) continue;
    float v[8];
    digits_begin(q, e, v);
#pragma unroll 1
    for (int i = 0; i < kDigits14; ++i) digits_next(v);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // v: 8^14 times what is left, in units of 2^(e - 128).  Far below its block a value has no digits, and may have vanished
      // in these units.
      const float whole = __uint_as_float((i & 1) != 0 ? r[i >> 1] & 0xffff0000u : r[i >> 1] << 16);
      const int field = static_cast<int>(__float_as_uint(whole) >> 23 & 255u);
      v[i] = field + 60 < e ? whole : ldexpf(v[i], e - 128 - 3 * kDigits14);
    }
    for (; lanes != 0u; lanes &= lanes - 1) {
      const int src = __ffs(lanes) - 1, c = base + src;  // eight columns of one block
      const uint32_t word = *reinterpret_cast<const uint32_t *>(codes + c * 4);
      const float scale = live ? decode_e4m3(w_scales[tiled_scale_offset(row, c >> 1, round_up_int(k >> 4, 4))]) : 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sum = fmaf(decode_e2m1(static_cast<uint8_t>(word >> (4 * i) & 15u)) * __shfl_sync(0xffffffffu, v[i], src), scale, sum);
      }
    }
  }
  return sum;
}

// grid (row blocks, 1, split), cluster (1, 1, split).
template <int OP>
__global__ void __launch_bounds__(kThreads, 2)
gemm_resident_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ ResidentArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rb = blockIdx.x, rank = blockIdx.z, split = gridDim.z;
  const int sf_col_blocks = a.k >> 6;                       // 512-byte scale tiles per row block
  const int ks0 = a.step_begin[rank], steps = a.step_begin[rank + 1] - ks0;
  const int op_bytes = a.cols_deep * kStepBytes;
  // The operand's scales: a column of TMEM holds four bytes (one MMA's) of 32 rows.  With no more than 64 rows the columns of two
  // MMAs share a tile, and a step takes two copies instead of four.  (An MMA's scales start at an even column: at an odd one
  // it faults.)  Offset of the word of `row` for MMA j:
  auto scale_word = [&](int row, int j) {
    const int col = j * a.sf_cols + (row >> 5);
    return (col >> 2) * kSfChunk + (row & 31) * 16 + (col & 3) * 4;
  };
  uint8_t * smem_a = smem;
  uint8_t * smem_op = smem_a + a.stages * kABytes;          // [most_steps] operand codes as the MMAs read them
  uint8_t * smem_sfa = smem_op + a.most_steps * op_bytes;
  uint8_t * smem_sfo = smem_sfa + a.stages * kSfBytes;      // [most_steps] the operand's scale tiles
  float * recv = reinterpret_cast<float *>(smem_sfo + a.most_steps * kSfBytes);  // [split][m][rows this CTA stores at most]
  const int recv_rows = a.group_begin[1] * kGroupRows;  // the first CTA has the most
  const int group0 = a.group_begin[rank], rows_here = (a.group_begin[rank + 1] - group0) * kGroupRows;  // rows of the tile that this CTA stores
  uint64_t * bars = reinterpret_cast<uint64_t *>(recv + split * a.m * recv_rows);
  uint64_t * full = bars;                          // [stages]: weights have landed
  uint64_t * empty = bars + kMaxStages;            // [stages]: the MMAs that read the stage have retired
  uint64_t * acc_full = bars + 2 * kMaxStages;
  uint64_t * op_ready = acc_full + 1;              // the operand is made
  uint64_t * amax_bar = op_ready + 1;              // the cluster's maxima have arrived
  uint64_t * sums = amax_bar + 1;                  // the cluster's sums for the rows this CTA stores have arrived
  uint64_t * mma_done = sums + 1;                  // after an expired wait: every MMA issued has retired
  uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
  __shared__ uint32_t gave_up, issued;             // 1: some role of this CTA gave up, 2: an earlier error is on record; K steps whose weights were asked for
  __shared__ float red[kMakers];
  __shared__ uint32_t s_amax[kMaxSplit], s_good[kMaxSplit];  // every CTA's maximum, and whether its sums count
  __shared__ uint32_t s_top[8], s_deep;            // W4A16: largest magnitude of every token here; 1: some value has deep digits, 256 << token: which leave something
  __shared__ float s_scale;                        // W4A4: the tensor's scale
  __shared__ float table[128];

  if (threadIdx.x == 0) {
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(smem_u32(full + i), 1);
      mbar_init(smem_u32(empty + i), 1);
    }
    mbar_init(smem_u32(acc_full), 1);
    mbar_init(smem_u32(op_ready), kMakers + (OP == kDigits ? a.absent & ~rb : 0));
    mbar_init(smem_u32(amax_bar), 1);
    mbar_init(smem_u32(mma_done), 1);
    mbar_init(smem_u32(sums), 1);
    gave_up = issued = s_deep = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (split > 1) {
      if (OP != kDigits) mbar_expect_tx(smem_u32(amax_bar), 4 * split);
      mbar_expect_tx(smem_u32(sums), 4 * split * (a.m * rows_here + 1));
    }
  }
  if (threadIdx.x < 8) s_top[threadIdx.x] = 0u;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (split > 1) cluster_arrive();  // this CTA's barriers and words can be written from now on; the wait is behind the roles' own
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  auto give_up = [&](unsigned code) {
    atomicCAS(a.status, 0u, code);
    atomicOr(&gave_up, 1u);
  };

  if (warp == 0) {
    // ---------------- weight loads (constant data: the first turn of the ring does not wait) ----------------
    if (elect_one()) {
      const uint8_t * sf = a.w_scales + static_cast<size_t>(rb) * sf_col_blocks * kSfChunk;
      int stage = 0;
      uint32_t phase = 1;
      for (int it = 0; it < steps; ++it) {
        const int ks = ks0 + it;
        if (it == a.stages) {
          // The ring is full, and HBM has nothing to do until the operand is made: what comes later into L2.
          for (int later = it; later < steps; ++later) {
            asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(&tmap_w), "r"((ks0 + later) * kStepBytes), "r"(rb * kRows) : "memory");
          }
          asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait before the activations can be there
        }
        if (!mbar_wait(smem_u32(empty + stage), phase, a.wait_limit)) {
          give_up(kWeightWait);
          break;
        }
        const uint32_t sf_bytes = min(kMmaPerStage, sf_col_blocks - ks * kMmaPerStage) * kSfChunk, bar = smem_u32(full + stage);
        mbar_expect_tx(bar, kABytes + sf_bytes);
        tma_load_2d(smem_u32(smem_a + stage * kABytes), &tmap_w, bar, ks * kStepBytes, rb * kRows);
        bulk_load(smem_u32(smem_sfa + stage * kSfBytes), sf + static_cast<size_t>(ks) * kSfBytes, sf_bytes, bar);
        issued = it + 1;
        if (it == min(a.stages, steps) - 1 && a.next_codes != nullptr) {
          // ... and what the next launch will stream
          prefetch_share(a.next_codes, a.next_codes_share, a.next_codes_bytes, rb * split + rank);
          prefetch_share(a.next_scales, a.next_scales_share, a.next_scales_bytes, rb * split + rank);
        }
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      bool ok = mbar_wait(smem_u32(op_ready), 0, a.wait_limit);
      if (!ok) give_up(kOperandWait);
      const int n_cols = OP == kDigits && *reinterpret_cast<volatile uint32_t *>(&s_deep) == 0u ? a.cols_plain : a.cols_deep;
      const int parts = partial_accumulators(n_cols);
      const uint32_t idesc = instr_desc(n_cols);
      // A step's scale factors are copied before the MMAs of the step before, so that these do not wait for copies.
      int ahead = 0;  // the ring's stage of the copies, and its phase
      uint32_t phase = 0;
      auto copy_scales = [&](int it) {
        if (!mbar_wait(smem_u32(full + ahead), phase, a.wait_limit)) {
          give_up(kMmaWait);
          return false;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t sfa_desc = desc_sf(smem_u32(smem_sfa + ahead * kSfBytes)), sfb_desc = desc_sf(smem_u32(smem_sfo + it * kSfBytes));
        const uint32_t sf_set = tmem_base + kAccCols + (it & 1) * kSfSetCols;
        const int valid = min(kMmaPerStage, sf_col_blocks - (ks0 + it) * kMmaPerStage);
#pragma unroll
        for (int j = 0; j < kMmaPerStage; ++j) {
          if (j < valid) utccp_sf(sf_set + j * 4, sfa_desc + j * (kSfChunk >> 4));
          if (j < a.sf_cols) utccp_sf(sf_set + 16 + j * 4, sfb_desc + j * (kSfChunk >> 4));
        }
        if (++ahead == a.stages) {
          ahead = 0;
          phase ^= 1;
        }
        return true;
      };
      ok = ok && copy_scales(0);
      int stage = 0;
#pragma unroll 1
      for (int it = 0; it < steps && ok; ++it) {
        if (it + 1 < steps && !copy_scales(it + 1)) {
          ok = false;
          break;
        }
        const int valid = min(kMmaPerStage, sf_col_blocks - (ks0 + it) * kMmaPerStage);
        const uint64_t a_desc = desc_k_sw128(smem_u32(smem_a + stage * kABytes)), b_desc = desc_k_sw128(smem_u32(smem_op + it * op_bytes));
        const uint32_t sf_set = tmem_base + kAccCols + (it & 1) * kSfSetCols;
#pragma unroll
        for (int j = 0; j < kMmaPerStage; ++j) {
          if (j < valid) {
            umma(tmem_base + (j & (parts - 1)) * n_cols, a_desc + j * 2, b_desc + j * 2, idesc, sf_set + j * 4, sf_set + 16 + j * a.sf_cols,
                 it * kMmaPerStage + j >= parts ? 1u : 0u);
          }
        }
        umma_commit(smem_u32(empty + stage));
        if (++stage == a.stages) stage = 0;
      }
      // also after giving up, which every warp then finds on record: none waits for what does not come
      if (ok) umma_commit(smem_u32(acc_full)); else mbar_arrive(smem_u32(acc_full));
    }
    __syncwarp();
  } else {
    // ---------------- the operand ----------------
    const int mt = threadIdx.x - 64, mw = warp - 2;
    if constexpr (OP == kDigits) {
      const int chunks = a.k >> 3;  // of eight columns
      const uint4 * x = static_cast<const uint4 *>(a.x);
      auto load = [&](const Unit & u) {
        const int token = u.token, c = (ks0 + u.it) * 32 + lane;
        return c < chunks ? __ldca(x + static_cast<size_t>(token) * chunks + c) : make_uint4(0u, 0u, 0u, 0u);
      };
      asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel before
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      const Unit start = next_unit(Unit{0, mw - kMakers}, steps);
      const uint4 first = start.token < a.m ? load(start) : zero;
      {
        uint4 q = first;
#pragma unroll 1
        for (Unit u = start; u.token < a.m;) {
          const uint32_t best = __reduce_max_sync(0xffffffffu, bf16x8_abs_max(q));
          if (lane == 0) atomicMax(&s_top[u.token], best);
          u = next_unit(u, steps);
          if (u.token < a.m) q = load(u);
        }
      }
      makers_sync();
      uint32_t deep = 0;
      uint4 q = first;
#pragma unroll 1
      for (Unit u = start; u.token < a.m;) {
        const int token = u.token, j = lane & 7;
        uint8_t * codes = smem_op + u.it * op_bytes, * tiles = smem_sfo + u.it * kSfBytes;
        const uint32_t best = s_top[token];
        const int top = max(static_cast<int>(best >> 7), 1);
        if (best >= 0x7f80u) q = zero;  // the epilogue has no use for the digits then
        u = next_unit(u, steps);
        const uint4 next = u.token < a.m ? load(u) : zero;
        uint32_t b = bf16x8_abs_max(q);
        b = max(b, __shfl_xor_sync(0xffffffffu, b, 1));
        const int e = digits_exponent(b, top);
        // the scale bytes of eight lanes' four blocks make one word of the tiled layout, the same for every digit
        uint32_t word = digits_scale_byte(e, top) << (8 * ((lane >> 1) & 3));
        word |= __shfl_xor_sync(0xffffffffu, word, 2);
        word |= __shfl_xor_sync(0xffffffffu, word, 4);
        auto write = [&](int row, uint32_t w) {
          *reinterpret_cast<uint32_t *>(codes + row * kStepBytes + ((((lane >> 2) ^ row) & 7) << 4) + ((lane & 3) << 2)) = w;
        };
        auto scales_of = [&](int row) { return reinterpret_cast<uint32_t *>(tiles + scale_word(row, lane >> 3)); };
        uint32_t rest = 0;
        float v[8];
        digits_begin(q, e, v);
        *scales_of(token * 8 + j) = word;
#pragma unroll
        for (int i = 0; i < 8; ++i) write(token * 8 + i, digits_next(v));
#pragma unroll
        for (int i = 0; i < 8; ++i) rest |= __float_as_uint(v[i]);
        const bool has = __any_sync(0xffffffffu, (rest & 0x7fffffffu) != 0u);
        const int deep_row = a.m * 8 + token * kDeepDigits;
        if (j < kDeepDigits) *scales_of(deep_row + j) = has ? word : 0u;  // zero scales make what lies there count for nothing
        if (has) {
#pragma unroll 1
          for (int i = 0; i < kDeepDigits; ++i) write(deep_row + i, digits_next(v));
          rest = 0;
#pragma unroll
          for (int i = 0; i < 8; ++i) rest |= __float_as_uint(v[i]);
          deep |= (rest & 0x7fffffffu) != 0u ? 256u << token | 1u : 1u;
        }
        q = next;
      }
      if (deep != 0u) atomicOr(&s_deep, deep);
    } else {
      using T = std::conditional_t<OP == kNvfp4Bf16, __nv_bfloat16, float>;
      constexpr int kVecs = sizeof(T);  // 16-byte loads per block
      // one block of sixteen per thread at most: block b of this CTA's columns of a token
      const int per_row = a.k >> 4, first = ks0 * 16, width = min(first + steps * 16, per_row) - first;
      const int token = static_cast<int>((static_cast<float>(mt) + 0.5f) * __fdividef(1.0f, static_cast<float>(width)));  // mt / width, up to 448 / 448
      const int b = mt - token * width;
      const bool has = token < a.m;
      uint32_t mine = 0;  // this CTA's K steps (28 at most) that its cluster writes to the scratch
      {
        int it = rb - ks0;
        while (it < 0) it += gridDim.x;
        for (; it < steps; it += gridDim.x) mine |= 1u << it;
      }
      asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel before, which may also read the scratch
      if (split > 1) cluster_wait();
      uint4 r[kVecs] = {};
      if (has) {
        const uint4 * src = static_cast<const uint4 *>(a.x) + (static_cast<size_t>(token) * per_row + first + b) * kVecs;
#pragma unroll
        for (int v = 0; v < kVecs; ++v) r[v] = __ldca(src + v);
      }
      float best = 0.0f;
#pragma unroll
      for (int v = 0; v < kVecs; ++v) best = abs_max<T>(r[v], best);
      // magnitudes: their bit patterns are ordered as they are
      const uint32_t warp_best = __reduce_max_sync(0xffffffffu, __float_as_uint(best));
      if (lane == 0) red[mw] = __uint_as_float(warp_best);
      makers_sync();
      float amax = red[0];
#pragma unroll
      for (int i = 1; i < kMakers; ++i) amax = fmaxf(amax, red[i]);
      if (split > 1) {
        if (mt < split) st_async(map_to_rank(smem_u32(&s_amax[rank]), mt), __float_as_uint(amax), map_to_rank(smem_u32(amax_bar), mt));
        if (!mbar_wait(smem_u32(amax_bar), 0, a.wait_limit)) {
          if (lane == 0) give_up(kAmaxWait);
        } else {
          for (int i = 0; i < split; ++i) amax = fmaxf(amax, __uint_as_float(*reinterpret_cast<volatile uint32_t *>(&s_amax[i])));
        }
      }
      const float g = amax > 0.0f ? __fdiv_rn(amax, 6.0f * 448.0f) : 1.0f;
      if (OP == kNvfp4Bf16) {
        if (mt < 127) table[mt] = bf16_block_multiplier(mt, g);  // the multipliers of quantize_block_bf16, per scale byte
        makers_sync();
      }
      if (mt == 0) s_scale = g;
      const float rg = __frcp_rn(g);
      if (a.g_out != nullptr && rb == 0 && rank == 0 && mt == 0) *a.g_out = g;
      if (has) {
        uint2 packed;
        const uint32_t sb = quantize_raw<T, OP == kNvfp4Bf16>(r, g, rg, table, packed);
        const int it = b >> 4, in = b & 15;
        *reinterpret_cast<uint2 *>(smem_op + it * op_bytes + token * kStepBytes + (((in >> 1) ^ (token & 7)) << 4) + (in & 1) * 8) = packed;
        smem_sfo[it * kSfBytes + scale_word(token, in >> 2) + (in & 3)] = static_cast<uint8_t>(sb);
        if ((mine >> it & 1u) != 0u) {
          *reinterpret_cast<uint2 *>(a.codes + (static_cast<size_t>(token) * per_row + first + b) * 8) = packed;
          a.scales[static_cast<size_t>(ks0 + it) * kSfBytes + (in >> 2) * kSfChunk + token * 16 + (in & 3)] = static_cast<uint8_t>(sb);  // fewer than 32 tokens
        }
      }
      // the scratch's scale bytes of rows m .. 127 are zero
      for (int it = 0; it < steps; ++it) {
        if ((mine >> it & 1u) == 0u) continue;
        const int valid = min(kMmaPerStage, sf_col_blocks - (ks0 + it) * kMmaPerStage);
        for (int i = mt; i < valid * kRows; i += kMakerThreads) {
          const int row = i & (kRows - 1);
          if (row >= a.m) *reinterpret_cast<uint32_t *>(a.scales + static_cast<size_t>(ks0 + it) * kSfBytes + (i >> 7) * kSfChunk + (row & 31) * 16 + (row >> 5) * 4) = 0u;
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs and the scale copies read what was written above
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(op_ready));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // One output of a token at a time; a gate/up weight's groups hold eight gate rows and the eight up rows for them.  Where a
  // thread's first one goes, and its residual, before the sums are waited for.
  const int row0 = rb * kRows + group0 * kGroupRows, outs = a.gate_up ? rows_here / 2 : rows_here;
  const float per_outs = __fdividef(1.0f, static_cast<float>(outs));
  struct Out {
    int token, r, row;
    float residual;
  };
  auto output = [&](int i) {
    Out o;
    o.token = static_cast<int>((static_cast<float>(i) + 0.5f) * per_outs);  // i / outs, up to 4096 / 8
    const int at = i - o.token * outs;
    o.r = a.gate_up ? (at >> 3) * kGroupRows + (at & 7) : at;
    o.row = row0 + o.r;
    o.residual = 0.0f;
    if (a.residual != nullptr && i < a.m * outs && o.row < a.n) {
      o.residual = __uint_as_float(static_cast<uint32_t>(__ldcg(reinterpret_cast<const unsigned short *>(a.residual) + static_cast<size_t>(o.token) * a.ldr + o.row)) << 16);
    }
    return o;
  };
  Out out = output(threadIdx.x);
  uint32_t held_back = 0;
  if (OP == kDigits && threadIdx.x == 0 && a.before != nullptr) held_back = __ldcg(a.before);
  if (split > 1 && (OP == kDigits || warp < 2)) cluster_wait();  // the makers of NVFP4 codes have

  // ---------------- TMEM -> the CTA that stores ----------------
  auto send_and_wait = [&] {
    if (OP != kDigits && warp == 2 && lane == 0 && *reinterpret_cast<volatile unsigned int *>(a.status) != 0u) atomicOr(&gave_up, 2u);  // an earlier error on record: store nothing
    bool ran = mbar_wait(smem_u32(acc_full), 0, kDrainLimit);
    if (!ran && lane == 0) give_up(kEpilogueWait);
    ran = __all_sync(0xffffffffu, ran);
    {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int quarter = warp & 3, group = warp >> 2;
      const int tile_row = quarter * 32 + lane, row_group = tile_row >> 4;
      const int owner = a.group_owner[row_group];
      // where this lane's sums go: [rank][token][row] of the owner
      float * mine = recv + rank * a.m * recv_rows + tile_row - a.group_begin[owner] * kGroupRows;
      const uint32_t dst = split > 1 ? map_to_rank(smem_u32(mine), owner) : 0u, dst_bar = split > 1 ? map_to_rank(smem_u32(sums), owner) : 0u;
      auto push = [&](int token, float v) {
        if (split > 1) {
          st_async(dst + token * recv_rows * 4, __float_as_uint(v), dst_bar);
        } else {
          mine[token * recv_rows] = v;
        }
      };
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t deep = OP == kDigits ? s_deep : 1u;
      const int n_cols = deep == 0u ? a.cols_plain : a.cols_deep;
      const int mmas = min(steps * kMmaPerStage, sf_col_blocks - ks0 * kMmaPerStage);
      const int parts = min(partial_accumulators(n_cols), mmas);  // accumulators that were written
      if constexpr (OP == kDigits) {
#pragma unroll 1
        for (int token = group; token < a.m; token += 4) {
          float sum = 0.0f, weight = 1.0f;  // of digit j: 8^-j
          uint32_t col = taddr + token * 8;
          int count = 8;
          const uint32_t best = s_top[token];
#pragma unroll 1
          for (bool again = deep != 0u;; again = false) {
            uint32_t r[4][8] = {};
            tmem_ld8(col, r[0]);  // what lies behind the deep digits is not used
            if (parts > 1) tmem_ld8(col + n_cols, r[1]);
            if (parts > 2) tmem_ld8(col + 2 * n_cols, r[2]);
            if (parts > 3) tmem_ld8(col + 3 * n_cols, r[3]);
            tmem_wait_ld(r);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j < count) {
                sum = fmaf((__uint_as_float(r[0][j]) + __uint_as_float(r[1][j])) + (__uint_as_float(r[2][j]) + __uint_as_float(r[3][j])), weight, sum);
                weight *= 0.125f;
              }
            }
            if (!again) break;
            col = taddr + a.m * 8 + token * kDeepDigits;  // the same code once more
            count = kDeepDigits;
          }
          // The token's scale is a power of two, possibly a subnormal one: it comes last, so that nothing underflows before the
          // output does.
          const float s2 = a.gate_up != 0 && (tile_row & 8) != 0 ? a.s2_up : a.s2;
          const int top = max(static_cast<int>(best >> 7), 1);
          float v = sum * s2 * digits_scale(top);
          if ((top > kTopUnderflows || (deep >> token & 256u) != 0u) && ran) {
            const __nv_bfloat16 * x = static_cast<const __nv_bfloat16 *>(a.x) + static_cast<size_t>(token) * a.k;
            const int k0 = ks0 * 256, k1 = min((ks0 + steps) * 256, a.k), row = rb * kRows + tile_row;
            if (best < 0x7f80u) {
              v = fmaf(left_dot(a.w_codes, a.w_scales, x, a.n, a.k, k0, k1, row, top, lane), s2, v);
            } else {
              // a token with NaNs has nothing else to give: a NaN times anything is one
              v = best > 0x7f80u ? __uint_as_float(0x7fffffffu) : infinite_dot(a.w_codes, a.w_scales, x, a.n, a.k, k0, k1, row, lane) * s2;
            }
          }
          push(token, ran ? v : 0.0f);
        }
      } else {
        const int c0 = group * 8;  // up to 32 columns
        if (c0 < a.m) {
          uint32_t r[8];
          tmem_ld8(taddr + c0, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll 1
          for (int p = 1; p < parts; ++p) {
            uint32_t r2[8];
            tmem_ld8(taddr + p * n_cols + c0, r2);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (c0 + i < a.m) push(c0 + i, ran ? __uint_as_float(r[i]) : 0.0f);
          }
        }
      }
    }
    // A CTA that gave up sends its sums too, so that nothing is under way to a CTA when it ends, and word that they do not
    // count: the whole cluster stores, or none of it does.
    if (split > 1) {
      if (threadIdx.x < static_cast<unsigned>(split)) {
        const bool good = ran && *reinterpret_cast<volatile uint32_t *>(&gave_up) == 0u;
        st_async(map_to_rank(smem_u32(&s_good[rank]), threadIdx.x), good ? 1u : 0u, map_to_rank(smem_u32(sums), threadIdx.x));
      }
      if (!mbar_wait(smem_u32(sums), 0, kDrainLimit)) {
        if (lane == 0) give_up(kSumsWait);
      } else if (lane < split && *reinterpret_cast<volatile uint32_t *>(&s_good[lane]) == 0u) {
        atomicOr(&gave_up, 2u);
      }
    }
    if (OP == kDigits && held_back != 0u) atomicOr(&gave_up, 2u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if ((gave_up & 1u) != 0u && elect_one()) {
        // nothing is issued any more; what was issued lands in this CTA's memory, so it has to land before the CTA ends
        umma_commit(smem_u32(mma_done));
        mbar_wait(smem_u32(mma_done), 0, kDrainLimit);
        const int last = static_cast<int>(issued);
        for (int it = max(last - a.stages, 0); it < last; ++it) mbar_wait(smem_u32(full + it % a.stages), it / a.stages & 1, kDrainLimit);
        if (split > 1) mbar_wait(smem_u32(sums), 0, kDrainLimit);
      }
      __syncwarp();
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<uint32_t>(kTmemCols)) : "memory");
    }
  };
  // ---------------- sums over the cluster, in rank order, and the stores ----------------
  auto finish = [&] {
    const float alpha = s_scale * a.s2, alpha_up = s_scale * a.s2_up;  // W4A4; the sums of W4A16 come scaled
#pragma unroll 1
    for (int i = threadIdx.x; i < a.m * outs;) {
      const float * src = recv + out.token * recv_rows + out.r;
      auto total = [&](const float * p) {
        float v[kMaxSplit], sum = 0.0f;
#pragma unroll
        for (int q = 0; q < kMaxSplit; ++q) v[q] = q < split ? p[q * a.m * recv_rows] : 0.0f;
#pragma unroll
        for (int q = 0; q < kMaxSplit; ++q) {
          if (q < split) sum = q == 0 ? v[q] : sum + v[q];
        }
        return sum;
      };
      float v = total(src);
      size_t at = static_cast<size_t>(out.token) * a.ldy + out.row;
      bool live = out.row < a.n;
      if (a.gate_up) {
        const float up = total(src + 8);
        if constexpr (OP == kDigits) {
          v = v / (1.0f + expf(-v)) * up;
        } else {
          v = silu_mul(v * alpha, up * alpha_up);
        }
        at = static_cast<size_t>(out.token) * a.ldy + (out.row >> 4) * 8 + (out.row & 7);
        live = out.row + 8 < a.n;
      } else {
        v = OP == kDigits ? v + out.residual : fmaf(v, alpha, out.residual);
      }
      if (live) a.y[at] = __float2bfloat16_rn(v);
      i += kThreads;
      if (i < a.m * outs) out = output(i);
    }
  };
  send_and_wait();
  if (gave_up == 0u) {
    finish();
  } else if (OP == kDigits && threadIdx.x == 0) {
    if (a.gave != nullptr) atomicExch(a.gave, 1u);
    if (held_back != 0u && atomicAdd(a.before + 1, 1u) == gridDim.x * gridDim.z - 1) a.before[0] = a.before[1] = 0u;
  }
  if ((gave_up & 1u) != 0u && split > 1) {
    __syncthreads();  // with warp 1, which has waited for the other CTAs' sums
    cluster_arrive();
    cluster_wait();
  }
}

// Shared memory of one shape of launch; false: it does not fit.
struct Shape {
  int split, stages, smem;
};
int most_groups(int split) { return (kGroups + split - 1) / split; }
bool shape_for(int row_blocks, int k, int m, int cols, int split, int sms, int ring, Shape * out) {
  const int k_steps = (k + 255) / 256;
  if (split > k_steps) return false;
  const int steps = (k_steps + split - 1) / split;
  const int fixed = kFixedBytes + steps * (cols * kStepBytes + kSfBytes) + split * m * most_groups(split) * kGroupRows * 4;
  // two CTAs per SM if the ring keeps `ring` stages then, which also leaves clusters room to be placed; else one, if the grid has no more
  for (const int budget : {kSmemHalf, kSmemFull}) {
    const int stages = std::min({kMaxStages, steps, (budget - fixed) / (kABytes + kSfBytes)});
    if (stages >= std::min({steps, ring, kMaxStages}) && (budget == kSmemHalf || row_blocks * split <= sms)) {
      *out = {split, stages, fixed + stages * (kABytes + kSfBytes)};
      return row_blocks * split <= 2 * sms;
    }
  }
  return false;
}

template <int OP>
int launch_resident(const q35b_weight * w, ResidentArgs & a, const Shape & shape, cudaStream_t s) {
  static std::atomic<bool> attr_set[64];
  std::atomic<bool> & set = attr_set[w->device & 63];
  if (!set.load(std::memory_order_acquire)) {
    Q35B_CUDA_TRY(cudaFuncSetAttribute(gemm_resident_kernel<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemFull), "cudaFuncSetAttribute(resident gemm smem)");
    set.store(true, std::memory_order_release);
  }
  a.w_scales = w->scales_tiled;
  a.w_codes = w->codes;
  a.n = w->rows;
  a.k = w->k;
  a.s2 = w->s2;
  a.s2_up = w->s2_up;
  a.gate_up = w->gate_up ? 1 : 0;
  a.stages = shape.stages;
  const int split = shape.split, k_steps = (w->k + 255) / 256;
  a.most_steps = (k_steps + split - 1) / split;
  for (int r = 0; r <= split; ++r) {
    a.step_begin[r] = static_cast<short>(r * k_steps / split);
    a.group_begin[r] = static_cast<short>((r * kGroups + split - 1) / split);
  }
  for (int g = 0; g < kGroups; ++g) a.group_owner[g] = static_cast<short>(g * split / kGroups);
  a.sf_cols = a.cols_deep <= 64 ? 2 : 4;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((w->rows + kRows - 1) / kRows), 1, static_cast<unsigned>(shape.split));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(shape.smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = static_cast<unsigned>(shape.split);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, gemm_resident_kernel<OP>, w->tmap_codes_128, a);
  count_launch();
  Q35B_CUDA_TRY(le, "gemm_resident_kernel launch");
  return Q35B_OK;
}

// ---- W4A16 ------------------------------------------------------------------------------------------------------

// The split, and the estimate it is chosen by (0: none fits), in nanoseconds: 230 per K step and SM, 450 for the digits of fourteen units of 256 columns, 250 for a
// step whose weights come when the ring has turned, 300 for the exchange.  chain: only shapes of which an SM holds two CTAs; the next
// launch's are then placed, and their weights on the way, while this one's run.  MLP block of two tokens, gate/up split / down
// split: [2560, 9216] 1/6 18.1 us, 2/6 18.2, 2/7 18.1, 2/8 17.4; [1024, 3584] 1/6 11.3, 2/6 11.2, 2/8 10.3.
double decode_shape(const q35b_weight * w, int m, bool chain, Shape * out) {
  if (w == nullptr || w->rows <= 0 || !w->has_maps || w->nan_scales || w->negative_scales || m < 1 || m > 8) return 0.0;
  const int cols = round_up_int(m * (8 + kDeepDigits), 16), row_blocks = (w->rows + kRows - 1) / kRows, sms = sm_count();
  double best = 0.0;
  for (int split = 1; split <= kMaxSplit; ++split) {
    Shape shape;
    if (!shape_for(row_blocks, w->k, m, cols, split, sms, 3, &shape) || (chain && shape.smem > kSmemHalf)) continue;
    const int steps = ((w->k + 255) / 256 + split - 1) / split;
    const double ns = (steps * 230 + (m * steps + kMakers - 1) / kMakers * 450) * std::max(1.0, static_cast<double>(row_blocks * split) / sms) +
                      std::max(0, steps - shape.stages) * 250 + (split > 1 ? 300 : 0);
    if (best == 0.0 || ns < best) {
      best = ns;
      *out = shape;
    }
  }
  return best;
}

// Clusters of a shape's split that the GPU holds at once, at half an SM or all of it per CTA: 148 SMs hold 296 CTAs of half an SM, but
// 56 clusters of five, 45 of six, 37 of seven and 33 of eight; of all of it 148, 74, 45, 33, 26, 22, 15 and 15.  Asked of a kernel of the
// same size that is never launched: the runtime counts on one CTA per SM of any kernel with tcgen05.alloc, which is so only until
// it gives up its right to allocate (clusters of two, 296 CTAs of 30 us each with 256 columns: 36 us).
__global__ void __launch_bounds__(kThreads, 2) resident_size_kernel(float * p) {
  extern __shared__ float words[];
  p[threadIdx.x] = words[threadIdx.x];
}
int clusters_at_once(const Shape & shape) {
  static std::atomic<int> known[64][2][kMaxSplit + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  const bool full = shape.smem > kSmemHalf;
  std::atomic<int> & held = known[dev][full ? 1 : 0][shape.split];
  int n = held.load(std::memory_order_relaxed);
  if (n != 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, 1, static_cast<unsigned>(shape.split));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(full ? kSmemFull : kSmemHalf);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(shape.split);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(resident_size_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemFull) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, resident_size_kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  held.store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace

double decode_resident_chain_ns(const q35b_weight * w, int m, bool * at_once) {
  Shape shape;
  const double ns = decode_shape(w, m, true, &shape);
  if (ns > 0.0) *at_once = (w->rows + kRows - 1) / kRows <= clusters_at_once(shape);
  return ns;
}

// Where not all clusters fit the GPU at once the rest, waiting for whole clusters' room, takes as long again, with all of an SM's shared
// memory per CTA several times as long: [6072, 4352] two tokens (48 clusters of six, 45 fit) 11.6 us, [4720, 4096] eight (37 of four, 33
// fit) 19.0, [4648, 9280] eight 35.1, where the plain estimate says 7.0, 7.1 and 11.6.  large: a weight that the streaming kernel would take; whole
// tiles then go in rounds, with all of an SM's shared memory per CTA nothing of the next call overlaps ([9088, 5632] four tokens 14.0, estimate 10.6;
// [11648, 4096] 18.8, 13.7), and more than twenty K steps per CTA are too long a way ([15992, 6400] two tokens 25.8, estimate 17.6, streaming 20.0; where only
// the rows kernel could have it, [14840, 5184] two 15.9 against 26.0).
double decode_resident_ns(const q35b_weight * w, int m, bool large) {
  Shape shape;
  double ns = decode_shape(w, m, false, &shape);
  if (ns == 0.0) return 0.0;
  const int row_blocks = (w->rows + kRows - 1) / kRows, steps = ((w->k + 255) / 256 + shape.split - 1) / shape.split, sms = sm_count();
  const bool full = shape.smem > kSmemHalf;
  if (large && steps > 20 && m > 1) return 0.0;
  if (large && shape.split == 1 && row_blocks > sms) {
    ns = (steps * 230 + (m * steps + kMakers - 1) / kMakers * 450) * ((row_blocks + sms - 1) / sms) + std::max(0, steps - shape.stages) * 250;
  }
  if (row_blocks > clusters_at_once(shape)) {
    ns *= full ? 4.5 : 2.5;
  } else if (full && large) {
    ns *= m <= 3 ? 1.2 : 1.5;
  }
  return 4500.0 + ns;
}

int launch_decode_resident(const q35b_weight * w, const void * x_bf16, int m, void * y_bf16, const void * residual_bf16,
                           const ResidentChain * chain, unsigned int * status, unsigned int wait_limit, cudaStream_t s) {
  Shape shape;
  if (decode_shape(w, m, chain != nullptr, &shape) == 0.0) return fail(Q35B_ERR_SHAPE, "NVFP4 projection does not fit the resident kernel.");
  ResidentArgs a = {};
  a.x = x_bf16;
  a.y = static_cast<__nv_bfloat16 *>(y_bf16);
  a.residual = static_cast<const __nv_bfloat16 *>(residual_bf16);
  a.ldy = w->gate_up ? w->rows / 2 : w->rows;
  a.ldr = w->rows;
  a.m = m;
  if (chain != nullptr) {
    a.gave = chain->gave;
    a.before = chain->before;
    a.absent = chain->absent ? 1 : 0;
  }
  if (const q35b_weight * next = chain != nullptr ? chain->next : nullptr) {
    a.next_codes = next->codes;
    a.next_codes_bytes = next->codes_bytes & ~size_t(15);
    a.next_scales = next->scales_tiled;
    a.next_scales_bytes = next->scales_tiled_bytes & ~size_t(15);
    const size_t ctas = static_cast<size_t>((w->rows + kRows - 1) / kRows) * shape.split;
    a.next_codes_share = static_cast<uint32_t>((a.next_codes_bytes / ctas + 16) & ~size_t(15));
    a.next_scales_share = static_cast<uint32_t>((a.next_scales_bytes / ctas + 16) & ~size_t(15));
  }
  a.cols_plain = round_up_int(m * 8, 16);
  a.cols_deep = round_up_int(m * (8 + kDeepDigits), 16);
  a.status = status;
  a.wait_limit = wait_limit;
  return launch_resident<kDigits>(w, a, shape, s);
}

// ---- W4A4 -------------------------------------------------------------------------------------------------------

// Whether a projection quantises its activations itself; `split` is the one of the plan, so that the sums are those of the
// two launches.  It pays where the two launches would meet twice (a scale from the tensor) and the quantising, which every row
// block does anew, is one block of sixteen per thread; and only if the ring holds the weights, or they come when the operand
// has been waited for.  us, two launches / one: [3, 5184] x [169, 5184] 9.1 / 6.1, [2, 2688] x [2077, 2688] 8.8 / 6.1, [4, 1664] x
// [8025, 1664] 9.1 / 7.4, [11, 1920] x [973, 1920] 8.5 / 6.2; more than one block per thread: [16, 2560] x [9216, 2560] 9.6 / 10.7, [20, 1280] x
// [870, 1280] 8.5 / 11.9; a given scale: [3, 2048] x [133, 2048] 4.9 / 4.8, [5, 3136] x [273, 3136] 5.3 / 5.5; weights that come later: [1, 3008] x
// [22014, 3008] 12.5 / 13.3.
bool prefill_resident_shape(const q35b_weight * w, int m, float scale, int split, int * stages, int * smem) {
  const int k_steps = (w->k + 255) / 256, steps = (k_steps + split - 1) / split;
  if (scale > 0.0f || m * steps * 16 > kMakerThreads) return false;  // so fewer than 32 tokens
  Shape shape;
  if (!shape_for((w->rows + kRows - 1) / kRows, w->k, m, round_up_int(m, 16), split, sm_count(), steps, &shape)) return false;
  *stages = shape.stages;
  *smem = shape.smem;
  return true;
}

int launch_prefill_resident(const q35b_weight * w, const void * x, bool f32, int m, uint8_t * codes, uint8_t * scales, float * g_dev, int split, int stages, int smem,
                            const void * residual, int ldr, void * c, int ldc, unsigned int * status, cudaStream_t s) {
  ResidentArgs a = {};
  a.x = x;
  a.y = static_cast<__nv_bfloat16 *>(c);
  a.residual = static_cast<const __nv_bfloat16 *>(residual);
  a.ldy = ldc;
  a.ldr = ldr;
  a.m = m;
  a.cols_plain = a.cols_deep = round_up_int(m, 16);
  a.codes = codes;
  a.scales = scales;
  a.g_out = g_dev;
  a.status = status;
  a.wait_limit = kWaitLimit;
  const Shape shape = {split, stages, smem};
  return f32 ? launch_resident<kNvfp4F32>(w, a, shape, s) : launch_resident<kNvfp4Bf16>(w, a, shape, s);
}

}  // namespace q35b
