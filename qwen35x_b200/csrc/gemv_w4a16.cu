// W4A16 decode projection (M = 1..8 tokens) for sm_100a.
//
// y[m, r] = sum_c e2m1(w[r,c]) * e4m3(s[r,c/16]) * s2 * x[m,c], fp32 accumulation.
// Replaces the reference's scalar projection kernels
// (src/runtime/cuda_bench.cu:283-429) and the in-megakernel nvfp4_row_dot
// (src/kernels/cuda/decode_layers.cuh:200-261).
//
// HBM layout read here: codes [rows, K/2] and scales [rows, K/16], both
// row-major as in the checkpoint, so a warp that walks a row issues fully
// coalesced loads (eight codes per lane).
//
// Dequantisation: the FP4 converter of sm_100a turns a byte into two exact
// fp16 values, widened to fp32; the block scale multiplies the dot product of
// a lane's eight weights.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "engine.h"
#include "nvfp4_codec.cuh"

namespace q35b {
namespace {

constexpr int kWarpsPerBlock = 8;
constexpr int kThreads = kWarpsPerBlock * 32;

// Two E2M1 codes (nibbles j and j+4 of `w`, j = shift/4) -> float2 scaled by 2^-14.
__device__ __forceinline__ float2 e2m1_pair_to_f32(uint32_t w, int shift) {
  const uint32_t q = (w >> shift);
  const uint32_t bits = ((q & 0x00070007u) << 9) | ((q & 0x00080008u) << 12);
  const __half2 h = *reinterpret_cast<const __half2 *>(&bits);
  return __half22float2(h);
}

// E4M3 byte -> fp32 (the reference's decode, sign honoured, 0x7f = 480).
__device__ __forceinline__ float e4m3_to_f32(uint32_t b) {
  const float mag = __uint_as_float((b & 0x7fu) << 20) * 0x1p120f;
  return (b & 0x80u) ? -mag : mag;
}

__device__ __forceinline__ void store_out(__nv_bfloat16 * p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void store_out(float * p, float v) { *p = v; }

// Dot product of 16 weights (two 32-bit code words) with 16 activations.
// Code j of the block sits in nibble j%8 of word j/8.
__device__ __forceinline__ float block_dot(uint32_t w0, uint32_t w1, const float * x) {
  float acc = 0.0f;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 a = e2m1_pair_to_f32(w0, 4 * p);  // codes p and p+4
    acc = fmaf(a.x, x[p], acc);
    acc = fmaf(a.y, x[p + 4], acc);
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 a = e2m1_pair_to_f32(w1, 4 * p);
    acc = fmaf(a.x, x[8 + p], acc);
    acc = fmaf(a.y, x[8 + p + 4], acc);
  }
  return acc;
}

// Eight E2M1 codes -> four exact fp32 pairs, with the FP4 converter of sm_100a.
__device__ __forceinline__ void e2m1x8_to_f32(uint32_t w, float2 (&f)[4]) {
  uint32_t h[4];
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
#pragma unroll
  for (int p = 0; p < 4; ++p) f[p] = __half22float2(*reinterpret_cast<const __half2 *>(&h[p]));
}

// Eight consecutive activations of a lane as four fp32 pairs.
template <typename XT>
struct XLoad;
template <>
struct XLoad<__nv_bfloat16> {
  static __device__ __forceinline__ void load8(const __nv_bfloat16 * p, float, float2 (&x)[4]) {
    const uint4 q = __ldca(reinterpret_cast<const uint4 *>(p));
    x[0] = make_float2(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u));
    x[1] = make_float2(__uint_as_float(q.y << 16), __uint_as_float(q.y & 0xffff0000u));
    x[2] = make_float2(__uint_as_float(q.z << 16), __uint_as_float(q.z & 0xffff0000u));
    x[3] = make_float2(__uint_as_float(q.w << 16), __uint_as_float(q.w & 0xffff0000u));
  }
};
template <>
struct XLoad<float> {
  static __device__ __forceinline__ void load8(const float * p, float scale, float2 (&x)[4]) {
    const float4 a = __ldca(reinterpret_cast<const float4 *>(p)), b = __ldca(reinterpret_cast<const float4 *>(p) + 1);
    x[0] = make_float2(a.x * scale, a.y * scale);
    x[1] = make_float2(a.z * scale, a.w * scale);
    x[2] = make_float2(b.x * scale, b.y * scale);
    x[3] = make_float2(b.z * scale, b.w * scale);
  }
};

// Two fp32 multiply-adds in one instruction, each rounded as fmaf is.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\t"
      "mov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// One warp owns RW consecutive rows and walks K in pieces of 256 columns, eight per lane, so that the activations of a
// piece are one contiguous 16-byte load per lane and token (a lane that takes 32 columns at once, for a 16-byte code
// load, makes every activation load touch 16 or, in fp32, 32 lines).  The codes and scales of the next two or four pieces
// are in flight while the current ones are worked on; weights are constant, so the first ones are requested before the
// previous kernel of the stream has finished.  With few rows KW = 4 warps share a row's pieces, and their sums meet in
// shared memory in slice order.
// Bound by the unpacking (half a conversion and a widening per weight) and, from about four tokens on, by the
// multiply-adds.  Against the 32-columns-per-lane kernel before it, and where K was no multiple of 32 an element-wise
// one: [3584, 1024] at one token 3.2 -> 2.6 us, [17286, 6720] at one fp32 token 61 -> 27, [9162, 8240] 141 -> 18,
// [4540, 7536] at two tokens 66 -> 16, [8350, 1536] at eight 32 -> 12.5.
constexpr int kPiece = 256;
__host__ __device__ constexpr int pieces_ahead(int m) { return m <= 4 ? 4 : 2; }
template <int M, int RW, int KW, typename XT, typename OT>
__global__ void __launch_bounds__(kThreads)
gemv_w4a16_rows_kernel(const uint8_t * __restrict__ codes, const uint8_t * __restrict__ scales,
                       const XT * __restrict__ x, OT * __restrict__ y, int rows, int k, float s2,
                       float x_scale) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31;
  constexpr int kAhead = pieces_ahead(M);
  const int warp = threadIdx.x >> 5, slice = warp % KW;
  const int row0 = (blockIdx.x * (kWarpsPerBlock / KW) + warp / KW) * RW;
  const uint8_t * code_row[RW];
  const uint8_t * scale_row[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const int row = min(row0 + r, rows - 1);
    code_row[r] = codes + static_cast<size_t>(row) * (k >> 1) + lane * 4;
    scale_row[r] = scales + static_cast<size_t>(row) * (k >> 4) + (lane >> 1);
  }
  uint32_t cw[kAhead][RW], sc[kAhead][RW];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int c = k0 + u * kPiece;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        cw[u][r] = 0u;
        sc[u][r] = 0u;
        if (c + lane * 8 < k) {
          cw[u][r] = __ldcs(reinterpret_cast<const uint32_t *>(code_row[r] + (c >> 1)));
          sc[u][r] = __ldcs(scale_row[r] + (c >> 4));
        }
      }
    }
  };
  fetch(slice * kAhead * kPiece);
  asm volatile("griddepcontrol.wait;" ::: "memory");

  float2 acc[RW][M];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = make_float2(0.0f, 0.0f);

  for (int k0 = slice * kAhead * kPiece; k0 < k; k0 += KW * kAhead * kPiece) {
    uint32_t w[kAhead][RW], sb[kAhead][RW];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        w[u][r] = cw[u][r];
        sb[u][r] = sc[u][r];
      }
    if (k0 + KW * kAhead * kPiece < k) fetch(k0 + KW * kAhead * kPiece);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int col = k0 + u * kPiece + lane * 8;
      if (col < k) {
        float2 wf[RW][4];
        float s[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          e2m1x8_to_f32(w[u][r], wf[r]);
          s[r] = e4m3_to_f32(sb[u][r]);
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
          float2 xv[4];
          XLoad<XT>::load8(x + static_cast<size_t>(m) * k + col, x_scale, xv);
#pragma unroll
          for (int r = 0; r < RW; ++r) {
            float2 d = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int p = 0; p < 4; ++p) d = fma2(wf[r][p], xv[p], d);
            acc[r][m] = fma2(d, make_float2(s[r], s[r]), acc[r][m]);
          }
        }
      }
    }
  }

  __shared__ float part[KW > 1 ? kWarpsPerBlock : 1][M];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float v = acc[r][m].x + acc[r][m].y;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0) {
        if constexpr (KW > 1) {
          part[warp][m] = v;
        } else if (row0 + r < rows) {
          store_out(y + static_cast<size_t>(m) * rows + row0 + r, v * s2);
        }
      }
    }
  }
  if constexpr (KW > 1) {
    static_assert(RW == 1, "slices of one row");
    __syncthreads();
    if (slice == 0 && lane < M && row0 < rows) {
      float v = part[warp][lane];
#pragma unroll
      for (int q = 1; q < KW; ++q) v += part[warp + q][lane];
      store_out(y + static_cast<size_t>(lane) * rows + row0, v * s2);
    }
  }
}

// Activations that are not 16-byte aligned (accepted where K is no multiple of 32): one warp per row, one 16-weight
// block per lane step, element loads.
template <typename XT, typename OT>
__global__ void __launch_bounds__(kThreads)
gemv_w4a16_generic_kernel(const uint8_t * __restrict__ codes, const uint8_t * __restrict__ scales,
                          const XT * __restrict__ x, OT * __restrict__ y, int rows, int k, int m_tokens,
                          float s2_scaled, float x_scale) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int packed_cols = k >> 1;
  const int scale_cols = k >> 4;
  for (int m = 0; m < m_tokens; ++m) {
    float acc = 0.0f;
    for (int b = lane; b < scale_cols; b += 32) {
      const uint2 cw = *reinterpret_cast<const uint2 *>(codes + static_cast<size_t>(row) * packed_cols + b * 8);
      float xv[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) xv[i] = static_cast<float>(x[static_cast<size_t>(m) * k + b * 16 + i]) * x_scale;
      acc = fmaf(block_dot(cw.x, cw.y, xv), e4m3_to_f32(scales[static_cast<size_t>(row) * scale_cols + b]), acc);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) store_out(y + static_cast<size_t>(m) * rows + row, acc * s2_scaled);
  }
}

// One thread per 16-weight block: bf16(e2m1 * (e4m3 * s2)), the reference's load-time dequantisation
// (src/runtime/qwen35x_cuda_backend.cpp:742-755).  Rows of a gate/up weight take the scale of their half.
__global__ void __launch_bounds__(kThreads)
dequant_bf16_kernel(const uint8_t * __restrict__ codes, const uint8_t * __restrict__ scales, __nv_bfloat16 * __restrict__ out,
                    int rows, int k, float s2, float s2_up, int gate_up) {
  const int scale_cols = k >> 4;
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<size_t>(rows) * scale_cols) return;
  const int row = static_cast<int>(idx / scale_cols);
  const float row_s2 = (gate_up && ((row >> 3) & 1)) ? s2_up : s2;
  const float scale = e4m3_to_f32(scales[idx]) * row_s2;
  const uint2 cw = *reinterpret_cast<const uint2 *>(codes + idx * 8);
  const uint32_t w[2] = {cw.x, cw.y};
  uint32_t packed[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t c0 = (w[j >> 2] >> ((j & 3) * 8)) & 0xfu;
    const uint32_t c1 = (w[j >> 2] >> ((j & 3) * 8 + 4)) & 0xfu;
    const float v0 = __uint_as_float(((c0 & 7u) << 22) | ((c0 & 8u) << 28)) * 0x1p126f * scale;
    const float v1 = __uint_as_float(((c1 & 7u) << 22) | ((c1 & 8u) << 28)) * 0x1p126f * scale;
    const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
    packed[j] = *reinterpret_cast<const uint32_t *>(&h);
  }
  uint4 * dst = reinterpret_cast<uint4 *>(out + idx * 16);
  dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
}

template <int M, int RW, int KW, typename XT, typename OT>
int launch_rows(const q35b_weight * w, const XT * x, OT * y, float x_scale, cudaStream_t s) {
  const int warps = (w->rows + RW - 1) / RW;
  const int blocks = (warps * KW + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const cudaError_t le = launch_pdl(gemv_w4a16_rows_kernel<M, RW, KW, XT, OT>, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), 0, s,
                                    static_cast<const uint8_t *>(w->codes), static_cast<const uint8_t *>(w->scales), x, y, w->rows,
                                    w->k, w->s2, x_scale);
  count_launch();
  Q35B_CUDA_TRY(le, "gemv_w4a16_rows_kernel launch");
  return Q35B_OK;
}

template <int M, typename XT, typename OT>
int launch_simt(const q35b_weight * w, const XT * x, OT * y, float x_scale, cudaStream_t s) {
  // Fewer rows than the chip holds blocks' worth of warps: four warps per row where K has pieces for them, else one.
  // Two rows per warp share its activation loads ([5674, 7072] at four tokens: 22 us, with four rows 29).
  const int sms = sm_count();
  if (w->rows < kWarpsPerBlock * sms && w->k > pieces_ahead(M) * kPiece) return launch_rows<M, 1, 4>(w, x, y, x_scale, s);
  if (w->rows < 2 * kWarpsPerBlock * sms) return launch_rows<M, 1, 1>(w, x, y, x_scale, s);
  return launch_rows<M, 2, 1>(w, x, y, x_scale, s);
}

template <typename XT, typename OT>
int launch_any(const q35b_weight * w, const XT * x, int m, OT * y, float x_scale, int kernel, cudaStream_t s) {
  if (w == nullptr || x == nullptr || y == nullptr) return fail(Q35B_ERR_ARGUMENT, "NVFP4 projection received a null buffer.");
  if (m < 1 || m > 8) return fail(Q35B_ERR_SHAPE, "NVFP4 decode projection supports 1..8 tokens.");
  if (w->rows == 0) return Q35B_OK;
  if (w->gate_up) return fail(Q35B_ERR_ARGUMENT, "A gate/up weight runs through the projection work list (q35b_gemv_batch_*).");
  if (kernel != Q35B_GEMV_AUTO && kernel != Q35B_GEMV_SIMT && kernel != Q35B_GEMV_STREAM) {
    return fail(Q35B_ERR_ARGUMENT, "Unknown NVFP4 projection kernel id " + std::to_string(kernel) + ".");
  }
  if (const int st = check_weight_device(w)) return st;
  if ((w->k % 32) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) != 0) {
    return fail(Q35B_ERR_ARGUMENT, "Activations of the NVFP4 projection must be 16-byte aligned.");
  }
  if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) {
    const int blocks = (w->rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
    gemv_w4a16_generic_kernel<XT, OT><<<blocks, kThreads, 0, s>>>(w->codes, w->scales, x, y, w->rows, w->k, m,
                                                                 w->s2 * 16384.0f, x_scale);
    count_launch();
    Q35B_CUDA_TRY(cudaGetLastError(), "gemv_w4a16_generic_kernel launch");
    return Q35B_OK;
  }
  switch (m) {
    case 1: return launch_simt<1>(w, x, y, x_scale, s);
    case 2: return launch_simt<2>(w, x, y, x_scale, s);
    case 3: return launch_simt<3>(w, x, y, x_scale, s);
    case 4: return launch_simt<4>(w, x, y, x_scale, s);
    case 5: return launch_simt<5>(w, x, y, x_scale, s);
    case 6: return launch_simt<6>(w, x, y, x_scale, s);
    case 7: return launch_simt<7>(w, x, y, x_scale, s);
    default: return launch_simt<8>(w, x, y, x_scale, s);
  }
}

}  // namespace

int launch_dequant_bf16(const q35b_weight * w, void * w_bf16, cudaStream_t s) {
  if (w == nullptr || w_bf16 == nullptr) return fail(Q35B_ERR_ARGUMENT, "NVFP4 dequantisation received a null buffer.");
  if ((reinterpret_cast<uintptr_t>(w_bf16) & 15u) != 0) return fail(Q35B_ERR_ARGUMENT, "NVFP4 dequantisation output must be 16-byte aligned.");
  if (const int st = check_weight_device(w)) return st;
  if (w->rows == 0) return Q35B_OK;
  const size_t blocks16 = static_cast<size_t>(w->rows) * (w->k / 16);
  dequant_bf16_kernel<<<static_cast<unsigned>((blocks16 + kThreads - 1) / kThreads), kThreads, 0, s>>>(
    w->codes, w->scales, static_cast<__nv_bfloat16 *>(w_bf16), w->rows, w->k, w->s2, w->s2_up, w->gate_up ? 1 : 0);
  count_launch();
  Q35B_CUDA_TRY(cudaGetLastError(), "dequant_bf16_kernel launch");
  return Q35B_OK;
}

int launch_gemv_bf16(const q35b_weight * w, const void * x_bf16, int m, void * y_bf16, int kernel, cudaStream_t s) {
  return launch_any(w, static_cast<const __nv_bfloat16 *>(x_bf16), m, static_cast<__nv_bfloat16 *>(y_bf16), 1.0f,
                    kernel, s);
}

// The rows kernel, from fits to graph replays: so much per 256 columns for every turn of the warps that the SMs hold, and from five tokens
// on no less than so much for every block that an SM has to run (either is at most a quarter off for nine calls in ten; [6072, 4352] eight
// tokens, whose blocks go round twice, 28.0 us, 17.3 by the first, 26.0 by the second; with few tokens the second is too much for blocks that just
// overflow: [6208, 2560] two 6.1, 6.6 and 7.1).  Where four warps
// share a row, which is rarely slower than what it is compared with, 0: [112, 8192] seven tokens 5.3 us, [1064, 6912] four 5.4, [888, 5056] six
// 6.3, where the resident kernel takes 8.2, 8.4 and 7.5; except with many tokens, rows and columns: [408, 10112] five to eight 10.0 to 11.4 / 7.8 to 10.0,
// [744, 9600] 10.1 to 11.9 / 7.9 to 9.8, [488, 8448] five to seven 8.7 / 8.1, 8.9 / 9.4, 9.8 / 9.3.
double gemv_rows_ns(const q35b_weight * w, int m) {
  static constexpr int per_turn[9] = {0, 480, 480, 620, 720, 950, 1100, 1000, 840};
  static constexpr int per_block[9] = {0, 0, 0, 0, 0, 340, 445, 461, 471}, fixed[9] = {0, 0, 0, 0, 0, 1990, 1750, 1710, 2020};
  const int sms = sm_count(), pieces = (w->k + kPiece - 1) / kPiece;
  if (w->rows < kWarpsPerBlock * sms && w->k > pieces_ahead(m) * kPiece) {  // as launch_simt deals them out
    if (m < 5 || w->rows < 400 || w->k < 8400) return 0.0;
    return 1000.0 + per_turn[m] * (pieces / 4.0) * std::max(1.0, 4.0 * w->rows / (sms * 18.0));
  }
  const int warps = w->rows < 2 * kWarpsPerBlock * sms ? w->rows : (w->rows + 1) / 2;
  const int blocks = ((warps + kWarpsPerBlock - 1) / kWarpsPerBlock + sms - 1) / sms;
  return std::max(1000.0 + per_turn[m] * pieces * std::max(1.0, warps / (sms * (m == 1 ? 32.0 : 18.0))),
                  fixed[m] + static_cast<double>(per_block[m]) * pieces * blocks);  // 0 up to four tokens
}

int launch_gemv_f32(const q35b_weight * w, const float * x, float input_scale, float * y, int kernel, cudaStream_t s) {
  return launch_any(w, x, 1, y, input_scale, kernel, s);
}

}  // namespace q35b
