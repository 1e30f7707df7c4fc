// NVFP4 quantisation on the GPU: BF16 (activations) or fp32 (weights) ->
// E2M1 codes, E4M3 block scales, fp32 per-tensor scale.
//
// Replaces nvfp4_quantize_{single_row,matrix,bf16_matrix}_for_cublaslt_kernel
// (src/runtime/cuda_bench.cu:98-213) and the cudaMemset pair that precedes
// them in every bridge (:2621-2624): padding scale bytes are written here.
//
// Recipe (bit-exact contract, all fp32, IEEE division, no fused contraction
// that could change a rounding):
//   g  = amax(X) / (6 * 448)   (1 if the tensor is all zero), or a given g
//   per 16-block: t  = amax_blk / 6
//                 sb = min(UE4M3(max(t / g, 1e-8)), 0x7e)
//                 d  = max(decode(sb), 1e-8) * g
//                 code_i = E2M1(x_i / d), element 2j in the low nibble
// UE4M3()/E2M1() are the reference's nearest-with-ties-down encoders
// (src/runtime/cuda_bench.cu:58-96).  0x7f is never emitted because the
// tensor-core UE4M3 format reads it as NaN.
//
// HBM traffic per [M,K] BF16 call: 2*M*K read once (what the second pass does
// not find in registers it finds in L2) + M*K/2 + M*K/16 written.
#include <cuda_bf16.h>

#include <algorithm>

#include "engine.h"
#include "nvfp4_codec.cuh"
#include "nvfp4_quant_block.cuh"

namespace q35b {
namespace {

constexpr int kThreads = 256;

// Per-tensor amax -> g of a weight.  ws[0] holds the running maximum (fp32 bits), ws[1] counts finished blocks; the last
// block publishes g and leaves both words zero for the next call.
__global__ void __launch_bounds__(kThreads)
amax_to_global_scale_kernel(const float * __restrict__ x, size_t n, unsigned int * __restrict__ ws, float * __restrict__ g_out) {
  // no early griddepcontrol.launch_dependents here: a dependent grid that became resident early would take the
  // registers this kernel's remaining blocks need; the implicit trigger at block exit overlaps the tail only
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may come from the kernel before
  float local = 0.0f;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  const float4 * v = reinterpret_cast<const float4 *>(x);
  const size_t nv = n >> 2;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nv; i += stride) {
    const float4 q = __ldcg(v + i);
    local = fmaxf(local, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, off));
  __shared__ float red[kThreads / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = red[0];
#pragma unroll
    for (int i = 1; i < kThreads / 32; ++i) m = fmaxf(m, red[i]);
    atomicMax(ws, __float_as_uint(m));
    __threadfence();
    const unsigned int ticket = atomicAdd(ws + 1, 1u);
    if (ticket == gridDim.x - 1) {
      __threadfence();
      const float amax = __uint_as_float(atomicExch(ws, 0u));
      *g_out = (amax > 0.0f) ? __fdiv_rn(amax, 6.0f * 448.0f) : 1.0f;
      ws[1] = 0u;
    }
  }
}

template <typename T>
__device__ __forceinline__ void load16(const T * p, float (&v)[16]);

template <>
__device__ __forceinline__ void load16<__nv_bfloat16>(const __nv_bfloat16 * p, float (&v)[16]) {
  const uint4 * q = reinterpret_cast<const uint4 *>(p);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint4 a = __ldca(q + i);
    const uint32_t r[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[i * 8 + j * 2] = __uint_as_float(r[j] << 16);
      v[i * 8 + j * 2 + 1] = __uint_as_float(r[j] & 0xffff0000u);
    }
  }
}

template <>
__device__ __forceinline__ void load16<float>(const float * p, float (&v)[16]) {
  const float4 * q = reinterpret_cast<const float4 *>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 a = __ldca(q + i);
    v[i * 4] = a.x;
    v[i * 4 + 1] = a.y;
    v[i * 4 + 2] = a.z;
    v[i * 4 + 3] = a.w;
  }
}

// Pass 2: one thread per 16-element block, so a warp reads 1 KB of contiguous activations and writes 256 bytes of
// contiguous codes; the four scale bytes of a 64-element group are gathered into lane 0 of each quad with
// shuffles and stored as one 32-bit word of the tiled layout (or four bytes of the row-major layout).
// The grid covers roundup(K/16, 4) block slots per row and rows_padded rows: slots past K and rows past `rows`
// only produce zero scale bytes (TILED layout).
template <typename T, int RECIPE, bool TILED>
__global__ void __launch_bounds__(kThreads, 6)  // 39 registers, six CTAs per SM: measured 4-5 % faster than five CTAs of 45
quantize_nvfp4_kernel(const T * __restrict__ x, int rows, int rows_padded, int k, const float * __restrict__ g_dev,
                      float g_fixed, float * __restrict__ g_out, int swap, uint8_t * __restrict__ codes,
                      uint8_t * __restrict__ scales) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the per-tensor scale, and x itself, may come from the kernel before
  const int scale_cols = k >> 4;
  const int slots = ((scale_cols + 3) >> 2) << 2;  // block slots per row, a multiple of 4
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(rows_padded) * slots;
  // whole quads run or exit together (slots % 4 == 0 and kThreads % 4 == 0), so the shuffles below are safe
  const bool live = idx < total;
  const int row = live ? static_cast<int>(idx / slots) : 0;
  const int b = live ? static_cast<int>(idx % slots) : 0;
  float g = 1.0f;
  if (RECIPE == kEngine) {
    // one load of the per-tensor scale per CTA, handed round in shared memory: every warp of a large grid loading
    // the same word would queue up on one L2 slice (measured: the kernel took 1.7x as long)
    __shared__ float g_shared;
    if (threadIdx.x == 0) g_shared = (g_dev != nullptr) ? __ldcg(g_dev) : g_fixed;
    __syncthreads();
    g = g_shared;
    if (g_out != nullptr && idx == 0) *g_out = g;
  }
  uint32_t sb = 0;
  if (live && row < rows && b < scale_cols) {
    float v[16];
    load16<T>(x + static_cast<size_t>(row) * k + static_cast<size_t>(b) * 16, v);
    uint2 packed;
    sb = quantize_block<RECIPE>(v, g, swap != 0, packed);
    *reinterpret_cast<uint2 *>(codes + (static_cast<size_t>(row) * k + static_cast<size_t>(b) * 16) / 2) = packed;
  }
  // gather the quad's four scale bytes
  const int lane = threadIdx.x & 31;
  uint32_t word = sb;
  word |= __shfl_sync(0xffffffffu, sb, (lane & ~3) + 1) << 8;
  word |= __shfl_sync(0xffffffffu, sb, (lane & ~3) + 2) << 16;
  word |= __shfl_sync(0xffffffffu, sb, (lane & ~3) + 3) << 24;
  if (!live || (lane & 3) != 0) return;
  if (TILED) {
    *reinterpret_cast<uint32_t *>(scales + tiled_scale_offset(row, b, slots)) = word;
  } else if (row < rows) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (b + j < scale_cols) scales[static_cast<size_t>(row) * scale_cols + b + j] = static_cast<uint8_t>(word >> (8 * j));
    }
  }
}

// ---- activations: amax, per-tensor scale and quantisation in one launch --------------------------------------------

// What bounds it, once a BF16 value costs one conversion (nvfp4_quant_block.cuh): about 150 instructions per block at 60 %
// of the issue slots, and for a tensor's own scale the first pass with the meeting at its end.  Four CTAs of 256 threads
// per SM leave registers for two held blocks and one on its way (five CTAs and one block: [4096, 2560] 15.0 us; three and
// four: 12.9, but 8.8 instead of 7.0 with a given scale).  us, amax launch + quantise launch with two conversions per
// value -> now, graph replays over more than L2: [16, 2560] 5.0 -> 3.5, [100, 9216] 6.2 -> 4.9, [4096, 2560] 17.3 -> 13.4,
// [4096, 9216] 48.7 -> 33.5; with a given scale 1.9 -> 1.6, 2.5 -> 2.1, 10.2 -> 7.0, 30.7 -> 18.9; fp32 [1000, 1024] 7.9 -> 5.4.
constexpr int kActCtas = 4;          // per SM
constexpr int kHold = 2;             // blocks a thread keeps in registers between the two passes
// Looks at the arrival counts, some 0.7 us each, before a CTA stops waiting for the others, and then for the ones that help.
struct AmaxWait {
  int polls = 64, help_polls = 1 << 12;
  unsigned int absent = 0;  // test hook: arrivals demanded on top of what the grid delivers
};

// Block slots of a tiled activation: `slots` (a multiple of four) per row, numbered through the rows.
struct SlotMap {
  uint32_t slots;
  uint32_t magic, shift;  // index / slots = umulhi(index, magic) >> shift for indexes below 2^31
};

__device__ __forceinline__ void locate(uint32_t i, const SlotMap & s, uint32_t & row, uint32_t & b) {
  row = __umulhi(i, s.magic) >> s.shift;
  b = i - row * s.slots;
}
__device__ __forceinline__ void locate(size_t i, const SlotMap & s, uint32_t & row, uint32_t & b) {
  row = static_cast<uint32_t>(i / s.slots);
  b = static_cast<uint32_t>(i % s.slots);
}

// Codes and scale byte of the block in `slot` (in: not one of the padding).
template <typename T, bool TABLE, typename Idx>
__device__ __forceinline__ void emit(Idx slot, bool in, const uint4 (&r)[sizeof(T)], const SlotMap & map, uint32_t scale_cols, Idx total, float g,
                                     float rg, const float * table, uint8_t * __restrict__ codes, uint8_t * __restrict__ scales) {
  uint32_t sb = 0, row, b;
  locate(slot, map, row, b);
  if (in) {
    uint2 packed;
    sb = quantize_raw<T, TABLE>(r, g, rg, table, packed);
    *(reinterpret_cast<uint2 *>(codes) + (static_cast<Idx>(row) * scale_cols + b)) = packed;
  }
  // the quad's four scale bytes (whole quads get here together: slots and kThreads are multiples of four)
  uint32_t word = sb << (8 * (threadIdx.x & 3));
  word |= __shfl_xor_sync(0xffffffffu, word, 1);
  word |= __shfl_xor_sync(0xffffffffu, word, 2);
  if ((threadIdx.x & 3) == 0 && slot < total) {
    const uint32_t tile = (row >> 7) * (map.slots >> 2) + (b >> 2);
    *reinterpret_cast<uint32_t *>(scales + static_cast<size_t>(tile) * 512 + ((row & 31) * 16 + (row >> 5 & 3) * 4)) = word;
  }
}

// One thread per 16-element block and turn, so a warp reads 1 KB (fp32: 2 KB) of contiguous activations and writes 256
// bytes of contiguous codes; the four scale bytes of a 64-element group meet in lane 0 of each quad and leave as one
// 32-bit word of the tiled layout.  Slots past K and rows past `rows` only produce zero scale bytes.
// DYNAMIC: the grid (never more CTAs than are resident together) reads everything once, meets at a counter, and quantises
// what it has kept in registers (the first kHold blocks of a thread) or reads again from L2.  No CTA depends on the others
// being there (kernels of other streams may hold their places for as long as they like): those that have waited some 45 us
// deal the whole tensor out among themselves, a CTA's share at a time, so that the amax costs one more pass over it and not
// one per CTA; and one that has waited much longer for these takes the maximum over everything by itself.
// ws: [0] running maximum (fp32 bits), [1] CTAs that have added theirs, [2] CTAs that have read it, [3] shares dealt out,
// [4] shares added; all zero between calls.
// Idx: type of a slot index, 32 bits up to 2^31 slots.
template <typename T, bool DYNAMIC, typename Idx>
__global__ void __launch_bounds__(kThreads, kActCtas)
quantize_activations_kernel(const T * __restrict__ x, uint32_t scale_cols, const SlotMap map, Idx live, Idx total, float g_fixed,
                            unsigned int parts, const AmaxWait wait, unsigned int * ws, float * __restrict__ g_out, uint8_t * __restrict__ codes,
                            uint8_t * __restrict__ scales) {
  constexpr int kVecs = sizeof(T);  // 16-byte loads per block
  constexpr int kHeld = DYNAMIC ? kHold : 1;
  __shared__ float table[128];
  __shared__ float red[kThreads / 32];
  __shared__ float shared_amax;
  __shared__ unsigned int shared_share;
  // every CTA of the grid is resident: the next kernel of the stream may move in beside them
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const Idx stride = static_cast<Idx>(gridDim.x) * kThreads, first = static_cast<Idx>(blockIdx.x) * kThreads;
  const bool even = map.slots == scale_cols;  // no padding slots: a slot's index is its block's
  float g = g_fixed, rg = 1.0f;
  // the multipliers pay as a table from the second turn on
  const bool many = sizeof(T) == 2 && stride < live;
  if constexpr (!DYNAMIC) {
    rg = __frcp_rn(g);
    if (many) {
      if (threadIdx.x < 127) table[threadIdx.x] = bf16_block_multiplier(threadIdx.x, g);
      __syncthreads();
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may come from the kernel before, which may also read the scratch

  // false: a slot of the padding
  auto load = [&](Idx slot, uint4 (&r)[kVecs]) -> bool {
    Idx f = slot;
    bool in = slot < live;
    if (!even) {
      uint32_t row, b;
      locate(slot, map, row, b);
      f = static_cast<Idx>(row) * scale_cols + b;
      in = in && b < scale_cols;
    }
    const uint4 * src = reinterpret_cast<const uint4 *>(x) + static_cast<size_t>(f) * kVecs;
    // through L1: a lane's loads share sectors, which each of them would fetch from L2 anew
#pragma unroll
    for (int i = 0; i < kVecs; ++i) r[i] = in ? __ldca(src + i) : make_uint4(0u, 0u, 0u, 0u);
    return in;
  };

  uint4 held[kHeld][kVecs];
  bool held_in[kHeld];
#pragma unroll
  for (int h = 0; h < kHeld; ++h) held_in[h] = load(first + h * stride + threadIdx.x, held[h]);
  if constexpr (DYNAMIC) {
    if (first < live) {  // the other CTAs only write padding
      float best = 0.0f;
#pragma unroll
      for (int h = 0; h < kHeld; ++h) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) best = abs_max<T>(held[h][i], best);
      }
#pragma unroll 2
      for (Idx at = first + kHeld * stride; at < live; at += stride) {
        uint4 r[kVecs];
        load(at + threadIdx.x, r);
#pragma unroll
        for (int i = 0; i < kVecs; ++i) best = abs_max<T>(r[i], best);
      }
      auto block_max = [&](float v) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        float m = red[0];
#pragma unroll
        for (int i = 1; i < kThreads / 32; ++i) m = fmaxf(m, red[i]);
        return m;
      };
      best = block_max(best);
      // whether all have added theirs, or those who wait have added every share, within `polls` looks (one thread)
      auto all_there = [&](int polls) {
        const unsigned int all = parts + wait.absent;
        for (int i = 0; i < polls; ++i) {
          unsigned int here, shares;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(here) : "l"(ws + 1) : "memory");
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(shares) : "l"(ws + 4) : "memory");
          if (here >= all || shares >= parts) return true;
        }
        return false;
      };
      // The counts only order what a fence stands on either side of: every maximum comes before its arrival, reading the
      // result comes after all arrivals (the last to arrive need not have polled) and before leaving, the reset after all
      // have left.
      auto read_amax = [&] {
        __threadfence();
        return __uint_as_float(*reinterpret_cast<volatile unsigned int *>(ws));
      };
      if (threadIdx.x == 0) {
        atomicMax(ws, __float_as_uint(best));
        __threadfence();
        const unsigned int here = atomicAdd(ws + 1, 1u) + 1u;
        shared_amax = here >= parts + wait.absent || all_there(wait.polls) ? read_amax() : -1.0f;
      }
      __syncthreads();
      float amax = shared_amax;
      if (amax < 0.0f) {
        auto share_max = [&](Idx from, Idx step) {
          float m = 0.0f;
          for (Idx at = from + threadIdx.x; at < live; at += step) {
            uint4 r[kVecs];
            load(at, r);
#pragma unroll
            for (int i = 0; i < kVecs; ++i) m = abs_max<T>(r[i], m);
          }
          __syncthreads();  // the words that hold the warps' maxima are free
          return block_max(m);
        };
        while (true) {
          if (threadIdx.x == 0) shared_share = atomicAdd(ws + 3, 1u);
          __syncthreads();
          const unsigned int share = shared_share;
          if (share >= parts) break;
          const float m = share_max(static_cast<Idx>(share) * kThreads, stride);
          if (threadIdx.x == 0) {
            atomicMax(ws, __float_as_uint(m));
            __threadfence();
            atomicAdd(ws + 4, 1u);
          }
        }
        if (threadIdx.x == 0) shared_amax = all_there(wait.help_polls) ? read_amax() : -1.0f;
        __syncthreads();
        amax = shared_amax;
        if (amax < 0.0f) amax = share_max(0, kThreads);
      }
      if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(ws + 2, 1u) == parts - 1u) {
          __threadfence();
#pragma unroll
          for (int i = 0; i < kQuantWorkspaceWords; ++i) ws[i] = 0u;
        }
      }
      g = amax > 0.0f ? __fdiv_rn(amax, 6.0f * 448.0f) : 1.0f;
      rg = __frcp_rn(g);
      if (many) {
        if (threadIdx.x < 127) table[threadIdx.x] = bf16_block_multiplier(threadIdx.x, g);
        __syncthreads();
      }
    }
  }
  if (g_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *g_out = g;

  if (!many) {
#pragma unroll
    for (int h = 0; h < kHeld; ++h) {
      if (first + h * stride < total) emit<T, false>(first + h * stride + threadIdx.x, held_in[h], held[h], map, scale_cols, total, g, rg, table, codes, scales);
    }
    for (Idx at = first + kHeld * stride; at < total; at += stride) {  // padding, or fp32
      uint4 r[kVecs];
      const bool in = load(at + threadIdx.x, r);
      emit<T, false>(at + threadIdx.x, in, r, map, scale_cols, total, g, rg, table, codes, scales);
    }
    return;
  }
  if constexpr (sizeof(T) == 2) {
    // the next block is on its way while one is quantised
    uint4 next[kVecs];
    Idx at = first + kHeld * stride;
    bool next_in = at < total && load(at + threadIdx.x, next);
#pragma unroll
    for (int h = 0; h < kHeld; ++h) {
      if (first + h * stride < total) emit<T, true>(first + h * stride + threadIdx.x, held_in[h], held[h], map, scale_cols, total, g, rg, table, codes, scales);
    }
#pragma unroll 1
    while (at < total) {
      uint4 r[kVecs];
#pragma unroll
      for (int i = 0; i < kVecs; ++i) r[i] = next[i];
      const bool in = next_in;
      const Idx slot = at + threadIdx.x;
      at += stride;
      next_in = at < total && load(at + threadIdx.x, next);
      emit<T, true>(slot, in, r, map, scale_cols, total, g, rg, table, codes, scales);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
tile_scales_kernel(const uint8_t * __restrict__ src, int rows, int rows_padded, int scale_cols,
                   uint8_t * __restrict__ tiled, unsigned int * __restrict__ flags) {
  const int groups = (scale_cols + 3) >> 2;
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<size_t>(rows_padded) * groups) return;
  const int row = static_cast<int>(idx / groups);
  const int grp = static_cast<int>(idx % groups);
  uint32_t sbytes = 0;
  if (row < rows) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = grp * 4 + j;
      if (b < scale_cols) sbytes |= static_cast<uint32_t>(src[static_cast<size_t>(row) * scale_cols + b]) << (8 * j);
    }
  }
  *reinterpret_cast<uint32_t *>(tiled + tiled_scale_offset(row, grp * 4, groups * 4)) = sbytes;
  if (flags != nullptr) {
    // some byte has its sign bit set; some byte is 0x7f or 0xff: adding one to the low seven bits carries into the eighth
    const uint32_t found = ((sbytes & 0x80808080u) != 0u ? 1u : 0u) | ((((sbytes & 0x7f7f7f7fu) + 0x01010101u) & 0x80808080u) != 0u ? 2u : 0u);
    if (found != 0u) atomicOr(flags, found);
  }
}

int check_quant_args(const void * x, int m, int k, const void * codes, const void * scales) {
  if (x == nullptr || codes == nullptr || scales == nullptr) {
    return fail(Q35B_ERR_ARGUMENT, "NVFP4 quantisation received a null buffer.");
  }
  if (m <= 0 || k <= 0 || (k % 16) != 0) return fail(Q35B_ERR_SHAPE, "Invalid dimensions for NVFP4 quantisation.");
  if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0 || (reinterpret_cast<uintptr_t>(codes) & 7u) != 0 ||
      (reinterpret_cast<uintptr_t>(scales) & 3u) != 0) {
    return fail(Q35B_ERR_ARGUMENT, "NVFP4 quantisation buffers must be 16-byte aligned.");
  }
  return Q35B_OK;
}

template <typename T>
int launch_quantize_activations(const T * x, int m, int k, float global_scale, uint8_t * codes, uint8_t * scales_tiled,
                                float * g_dev, void * workspace, cudaStream_t s, const AmaxWait & wait = AmaxWait()) {
  if (const int st = check_quant_args(x, m, k, codes, scales_tiled)) return st;
  if (g_dev == nullptr) return fail(Q35B_ERR_ARGUMENT, "NVFP4 quantisation needs a device word for the input scale.");
  const bool dynamic = !(global_scale > 0.0f);
  if (dynamic && workspace == nullptr) return fail(Q35B_ERR_ARGUMENT, "Dynamic NVFP4 quantisation needs its workspace.");
  const int rows_padded = round_up_int(m, 128);
  SlotMap map = {static_cast<uint32_t>((((k >> 4) + 3) >> 2) << 2), 0u, 0u};
  const size_t total = static_cast<size_t>(rows_padded) * map.slots, live = static_cast<size_t>(m) * map.slots;
  const size_t per_turn = static_cast<size_t>(sm_count()) * kActCtas * kThreads;
  const unsigned grid = static_cast<unsigned>(std::min((total + kThreads - 1) / kThreads, per_turn / kThreads));
  const unsigned parts = static_cast<unsigned>(std::min<size_t>(grid, (live + kThreads - 1) / kThreads));
  cudaError_t le;
  if (total + (kHold + 1) * per_turn < (1u << 31)) {
    // ceil(2^(31 + l) / slots) with 2^(l - 1) < slots <= 2^l divides every index below 2^31 exactly; slots >= 4, so l >= 2
    int l = 2;
    while ((1u << l) < map.slots) ++l;
    map.magic = static_cast<uint32_t>(((1ull << (31 + l)) + map.slots - 1) / map.slots);
    map.shift = static_cast<uint32_t>(l - 1);
    le = launch_pdl(dynamic ? quantize_activations_kernel<T, true, uint32_t> : quantize_activations_kernel<T, false, uint32_t>, dim3(grid),
                    dim3(kThreads), 0, s, x, static_cast<uint32_t>(k >> 4), map, live, total, global_scale, parts, wait,
                    static_cast<unsigned int *>(workspace), g_dev, codes, scales_tiled);
  } else {
    le = launch_pdl(dynamic ? quantize_activations_kernel<T, true, size_t> : quantize_activations_kernel<T, false, size_t>, dim3(grid),
                    dim3(kThreads), 0, s, x, static_cast<uint32_t>(k >> 4), map, live, total, global_scale, parts, wait,
                    static_cast<unsigned int *>(workspace), g_dev, codes, scales_tiled);
  }
  count_launch();
  Q35B_CUDA_TRY(le, "quantize_activations_kernel launch");
  return Q35B_OK;
}

}  // namespace

int launch_quantize_bf16(const void * x, int m, int k, float global_scale, uint8_t * codes, uint8_t * scales_tiled,
                         float * g_dev, void * workspace, cudaStream_t s) {
  return launch_quantize_activations(static_cast<const __nv_bfloat16 *>(x), m, k, global_scale, codes, scales_tiled, g_dev,
                                     workspace, s);
}

int launch_quantize_bf16_wait(const void * x, int m, int k, uint8_t * codes, uint8_t * scales_tiled, float * g_dev, void * workspace,
                              int polls, int help_polls, unsigned int absent, cudaStream_t s) {
  AmaxWait wait;
  wait.polls = polls;
  wait.help_polls = help_polls;
  wait.absent = absent;
  return launch_quantize_activations(static_cast<const __nv_bfloat16 *>(x), m, k, 0.0f, codes, scales_tiled, g_dev, workspace, s, wait);
}

int launch_quantize_f32(const float * x, int m, int k, float global_scale, uint8_t * codes, uint8_t * scales_tiled,
                        float * g_dev, void * workspace, cudaStream_t s) {
  return launch_quantize_activations(x, m, k, global_scale, codes, scales_tiled, g_dev, workspace, s);
}

int launch_quantize_reference_recipe(const void * x, int m, int k, int swap, uint8_t * codes, uint8_t * scales_tiled,
                                     cudaStream_t s) {
  if (const int st = check_quant_args(x, m, k, codes, scales_tiled)) return st;
  const int rows_padded = round_up_int(m, 128);
  const size_t threads = static_cast<size_t>(rows_padded) * ((((k >> 4) + 3) >> 2) << 2);
  const unsigned blocks = static_cast<unsigned>((threads + kThreads - 1) / kThreads);
  quantize_nvfp4_kernel<__nv_bfloat16, kReference, true><<<blocks, kThreads, 0, s>>>(
    static_cast<const __nv_bfloat16 *>(x), m, rows_padded, k, nullptr, 1.0f, nullptr, swap, codes, scales_tiled);
  count_launch();
  Q35B_CUDA_TRY(cudaGetLastError(), "quantize_nvfp4_kernel(reference recipe) launch");
  return Q35B_OK;
}

int launch_quantize_weight_f32(const float * w, int n, int k, uint8_t * codes, uint8_t * scales_rowmajor,
                               float * s2_dev, void * workspace, cudaStream_t s) {
  if (w == nullptr || codes == nullptr || scales_rowmajor == nullptr || s2_dev == nullptr || workspace == nullptr) {
    return fail(Q35B_ERR_ARGUMENT, "NVFP4 weight quantisation received a null buffer.");
  }
  if (n <= 0 || k <= 0 || (k % 16) != 0) return fail(Q35B_ERR_SHAPE, "Invalid dimensions for NVFP4 weight quantisation.");
  // few blocks (every one ends with two atomics on the same pair of words), each with plenty of loads in flight
  const size_t elements = static_cast<size_t>(n) * k, per_block = static_cast<size_t>(kThreads) * 8 * 4;
  const int amax_blocks = static_cast<int>(std::min<size_t>((elements + per_block - 1) / per_block, static_cast<size_t>(sm_count()) * 4));
  const cudaError_t le = launch_pdl(amax_to_global_scale_kernel, dim3(amax_blocks), dim3(kThreads), 0, s, w, elements,
                                    static_cast<unsigned int *>(workspace), s2_dev);
  count_launch();
  Q35B_CUDA_TRY(le, "amax_to_global_scale_kernel launch");
  const size_t threads = static_cast<size_t>(n) * ((((k >> 4) + 3) >> 2) << 2);
  const unsigned blocks = static_cast<unsigned>((threads + kThreads - 1) / kThreads);
  quantize_nvfp4_kernel<float, kEngine, false><<<blocks, kThreads, 0, s>>>(w, n, n, k, s2_dev, 1.0f, nullptr, 0, codes,
                                                                          scales_rowmajor);
  count_launch();
  Q35B_CUDA_TRY(cudaGetLastError(), "quantize_nvfp4_kernel(weights) launch");
  return Q35B_OK;
}

int launch_tile_scales(const uint8_t * scales_rowmajor, int rows, int scale_cols, uint8_t * tiled,
                       unsigned int * flags, cudaStream_t s) {
  const int rows_padded = round_up_int(rows, 128);
  const size_t threads = static_cast<size_t>(rows_padded) * ((scale_cols + 3) >> 2);
  const unsigned blocks = static_cast<unsigned>((threads + kThreads - 1) / kThreads);
  tile_scales_kernel<<<blocks, kThreads, 0, s>>>(scales_rowmajor, rows, rows_padded, scale_cols, tiled, flags);
  count_launch();
  Q35B_CUDA_TRY(cudaGetLastError(), "tile_scales_kernel launch");
  return Q35B_OK;
}

}  // namespace q35b
