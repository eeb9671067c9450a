// Small kernels around the hot path: weight re-layouts (offline), the split-K finisher and the
// reference-compatible INT4-tail ("T4") epilogues.
#include "tq_common.cuh"

namespace tq {
namespace {

// ------------------------------------------------------------------ [N,K] bf16 -> [K,N] bf16
// HBM-bound: 4 bytes per element.  A thread transposes an 8 x 8 block in registers -- eight 128-bit loads, all in flight, 32
// byte permutes, eight 128-bit stores -- and nothing goes through shared memory.  The lanes of a warp are 4 blocks along k
// x 8 along n: 64-byte pieces of the rows read, full 128-byte lines written.  24576 x 4096: 230 -> 66 us (element-wise
// through a shared tile before).  N % 8 == 0, K % 8 == 0, 16-byte aligned; 128 x 128 elements per CTA.
__global__ void __launch_bounds__(256) transpose_bf16_8x8_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out,
                                                                 int N, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 128 + ((warp & 3) * 4 + (lane & 3)) * 8;
  const int n = blockIdx.y * 128 + ((warp >> 2) * 8 + (lane >> 2)) * 8;
  if (n >= N || k >= K) return;
  uint32_t a[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint4 v = ldg_nc_128(in + (size_t)(n + i) * K + k);
    a[i][0] = v.x, a[i][1] = v.y, a[i][2] = v.z, a[i][3] = v.w;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t sel = (c & 1) ? 0x7632u : 0x5410u;
    uint32_t o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = __byte_perm(a[2 * q][c >> 1], a[2 * q + 1][c >> 1], sel);
    *reinterpret_cast<uint4*>(out + (size_t)(k + c) * N + n) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// (any even N)
__global__ void transpose_bf16_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int N, int K) {
  __shared__ uint16_t tile[64][66];
  const int k0 = blockIdx.x * 64, n0 = blockIdx.y * 64;
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const int n = n0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const int k = k0 + j;
      tile[i][j] = (n < N && k < K) ? in[(size_t)n * K + k] : (uint16_t)0;
    }
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const int k = k0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const int n = n0 + j;
      if (n < N && k < K) out[(size_t)k * N + n] = tile[j][i];
    }
  }
}

// ------------------------------------------------------------------ b_col [N,K/2] -> b_row [K,N/2]
// low nibble of b_row[k][n/2] = code (n even), high nibble = code (n odd)
// (layout read by tools/fused_sparse_epilogue_ext_v58.py:63-71).
// A thread takes 8 output x 32 input channels: eight 128-bit loads, four 8 x 8 nibble transposes in registers (swaps of 16, 8
// and 4 bits), 32 stores of one word.  Conditions as above with K % 32 == 0.
__global__ void __launch_bounds__(256) col_to_row_s4_8x32_kernel(const uint8_t* __restrict__ b_col, uint8_t* __restrict__ b_row,
                                                                 int N, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 512 + ((warp & 3) * 4 + (lane & 3)) * 32;
  const int n = blockIdx.y * 128 + ((warp >> 2) * 8 + (lane >> 2)) * 8;
  if (n >= N || k >= K) return;
  uint32_t a[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint4 v = ldg_nc_128(b_col + ((size_t)(n + i) * K + k) / 2);
    a[i][0] = v.x, a[i][1] = v.y, a[i][2] = v.z, a[i][3] = v.w;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t r[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = __byte_perm(a[i][c], a[i + 4][c], 0x5410u);
      r[i + 4] = __byte_perm(a[i][c], a[i + 4][c], 0x7632u);
    }
#pragma unroll
    for (int h = 0; h < 8; h += 4)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t x = r[h + i], y = r[h + i + 2];
        r[h + i] = __byte_perm(x, y, 0x6240u);
        r[h + i + 2] = __byte_perm(x, y, 0x7351u);
      }
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t x = r[i], y = r[i + 1];
      r[i] = (x & 0x0f0f0f0fu) | ((y & 0x0f0f0f0fu) << 4);
      r[i + 1] = ((x >> 4) & 0x0f0f0f0fu) | (y & 0xf0f0f0f0u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<uint32_t*>(b_row + ((size_t)(k + 8 * c + i) * N + n) / 2) = r[i];
  }
}

__global__ void col_to_row_s4_kernel(const uint8_t* __restrict__ b_col, uint8_t* __restrict__ b_row, int N, int K) {
  const int n2 = blockIdx.x * blockDim.x + threadIdx.x;  // pair of output channels
  const int k2 = blockIdx.y;                             // pair of input channels
  if (n2 >= N / 2) return;
  const uint8_t a = b_col[(size_t)(2 * n2) * (K / 2) + k2];      // codes (n, 2k2), (n, 2k2+1)
  const uint8_t b = b_col[(size_t)(2 * n2 + 1) * (K / 2) + k2];  // codes (n+1, ..)
  b_row[(size_t)(2 * k2) * (N / 2) + n2] = (uint8_t)((a & 0x0f) | ((b & 0x0f) << 4));
  b_row[(size_t)(2 * k2 + 1) * (N / 2) + n2] = (uint8_t)((a >> 4) | (b & 0xf0));
}

// ------------------------------------------------------------------ split-K finisher
__global__ void dequant_finish_kernel(const int32_t* __restrict__ C, const float* __restrict__ sx,
                                      const float* __restrict__ sw, const float* __restrict__ tail,
                                      const float* __restrict__ bias, uint16_t* __restrict__ out, int M, int N) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)M * N) return;
  const int m = (int)(i / N), n = (int)(i % N);
  float d = __fmul_rn(__fmul_rn((float)C[i], sx[m]), sw[n]);
  if (tail) d = __fadd_rn(d, tail[i]);
  if (bias) d = __fadd_rn(d, bias[n]);
  out[i] = (uint16_t)f32_to_bf16_bits(d);
}

// the same with the accumulators still split over `splits` K ranges ([splits, M, N]): summed here, exactly.
// act = 1: SwiGLU over interleaved (gate, up) channel pairs, out [M, N/2]; one thread per output either way.
__global__ void dequant_finish_partials_kernel(const int32_t* __restrict__ P, int splits, const float* __restrict__ sx,
                                               const float* __restrict__ sw, const float* __restrict__ tail,
                                               const float* __restrict__ bias, uint16_t* __restrict__ out, int M, int N,
                                               int act) {
  const size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t total = (size_t)M * N;
  const int per = act ? 2 : 1;  // accumulators per output
  if (o * per >= total) return;
  float d[2];
  for (int e = 0; e < per; ++e) {
    const size_t i = o * per + e;
    const int m = (int)(i / N), n = (int)(i % N);
    int acc = 0;
    for (int s = 0; s < splits; ++s) acc += P[(size_t)s * total + i];
    float v = __fmul_rn(__fmul_rn((float)acc, sx[m]), sw[n]);
    if (tail) v = __fadd_rn(v, tail[i]);
    if (bias) v = __fadd_rn(v, bias[n]);
    d[e] = v;
  }
  out[o] = (uint16_t)(act ? swiglu_bf16_bits(d[0], d[1]) : f32_to_bf16_bits(d[0]));
}

// ------------------------------------------------------------------ T4 sparse term
// sum_r tq[r] * q_w[idx[r], n0 .. n0 + 7], exact.  What bounds it is the integer work, so two channels share a 32-bit
// multiply-add: the nibbles are biased to u = q + 8 (0 .. 15), the words (u_i | u_{i+4} << 16) are multiplied by tq, and the
// bias comes off with 8 sum(tq).  16 entries of any int8 fit the 16-bit halves (16 * 128 * 15 < 2^15) before they are spread.
constexpr int T4_CHUNK = 1024;   // entries staged at a time

__device__ __forceinline__ void sparse_add(const uint2* __restrict__ list, int cnt, const uint8_t* __restrict__ b_row, int N,
                                           int n0, int (&acc)[8]) {
  for (int r0 = 0; r0 < cnt; r0 += 16) {
    const int r1 = min(cnt, r0 + 16);
    int p[4] = {0, 0, 0, 0}, bias = 0;
#pragma unroll 8
    for (int r = r0; r < r1; ++r) {
      const uint2 e = list[r];
      const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(b_row + ((size_t)e.x * N + n0) / 2));
      const int a = (int)e.y;
      bias += a;
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] += a * (int)(((w >> (4 * i)) & 0x000f000fu) ^ 0x00080008u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int lo = (int)(short)p[i];
      acc[i] += lo - 8 * bias;
      acc[i + 4] += ((p[i] - lo) >> 16) - 8 * bias;
    }
  }
}

__device__ __forceinline__ float load16(const void* p, size_t i, int dtype) {
  return dtype == TQ_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i])
                          : __half2float(reinterpret_cast<const __half*>(p)[i]);
}

// mode 0: out = f16(float(C)*bs*ws + float(sum)*ts*ws)      (tools/fused_sparse_epilogue_ext_v58.py:76-86)
// mode 1: out = f16(float(out) + float(sum)*ts*ws)          (tools/sparse_correction_add_ext_v1.py:64-123)
// mode 2: out = f16(float(sum)*ts*ws)                       (tools/split_sparse_idx16_ext_v1.py:50-109)
template <typename IdxT>
__global__ void __launch_bounds__(128) t4_epilogue_kernel(int mode, const int32_t* __restrict__ C, const float* __restrict__ bs,
                                                          const int8_t* __restrict__ top_q, const IdxT* __restrict__ idx,
                                                          const uint8_t* __restrict__ b_row, const float* __restrict__ ts,
                                                          const void* __restrict__ ws, int ws_bf16, void* out, int out_dtype,
                                                          int vec, int N, int R) {
  __shared__ uint2 list[T4_CHUNK];   // (index, code) of the row's entries
  const int m = blockIdx.y;
  const int n0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const bool on = n0 < N;
  int acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int c0 = 0; c0 < R; c0 += T4_CHUNK) {
    const int cnt = min(R - c0, T4_CHUNK);
    if (c0) __syncthreads();
    for (int r = threadIdx.x; r < cnt; r += blockDim.x)
      list[r] = make_uint2((uint32_t)idx[(size_t)m * R + c0 + r], (uint32_t)(int)top_q[(size_t)m * R + c0 + r]);
    __syncthreads();
    if (on) sparse_add(list, cnt, b_row, N, n0, acc);
  }
  if (!on) return;
  const float tsm = ts[m];
  const float bsm = (mode == 0) ? bs[m] : 0.0f;
  const size_t o = (size_t)m * N + n0;
  uint32_t r16[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float w = ws_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ws)[n0 + i])
                            : reinterpret_cast<const float*>(ws)[n0 + i];
    const float sparse = __fmul_rn(__fmul_rn((float)acc[i], tsm), w);
    float d = sparse;
    if (mode == 0) d = __fadd_rn(__fmul_rn(__fmul_rn((float)C[o + i], bsm), w), sparse);
    if (mode == 1) d = __fadd_rn(load16(out, o + i, out_dtype), sparse);
    r16[i] = out_dtype == TQ_BF16 ? f32_to_bf16_bits(d) : (uint32_t)__half_as_ushort(__float2half_rn(d));
  }
  if (vec) {
    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + o) =
        make_uint4(r16[0] | (r16[1] << 16), r16[2] | (r16[3] << 16), r16[4] | (r16[5] << 16), r16[6] | (r16[7] << 16));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) reinterpret_cast<uint16_t*>(out)[o + i] = (uint16_t)r16[i];
  }
}

__global__ void idx_i32_to_u16_kernel(const int32_t* __restrict__ in, uint16_t* __restrict__ out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (uint16_t)in[i];
}

int t4_launch(int mode, const int32_t* C, const float* bs, const int8_t* top_q, const void* idx, int idx_u16,
              const uint8_t* b_row, const float* ts, const void* ws, int ws_bf16, void* out, int out_dtype, int M,
              int N, int K, int R, cudaStream_t st) {
  if (!top_q || !idx || !b_row || !ts || !ws || !out || M < 0 || N <= 0 || K <= 0 || R <= 0) return TQ_ERR_BAD_ARG;
  if (mode == 0 && (!C || !bs)) return TQ_ERR_BAD_ARG;
  if (N % 8 != 0) return TQ_ERR_UNSUPPORTED;
  if (out_dtype != TQ_BF16 && out_dtype != TQ_FP16) return TQ_ERR_BAD_ARG;
  if (M == 0) return TQ_OK;
  const int vec = aligned16(out) ? 1 : 0;
  const dim3 block(128), grid((N / 8 + 127) / 128, M);
  if (idx_u16)
    t4_epilogue_kernel<uint16_t><<<grid, block, 0, st>>>(mode, C, bs, top_q, reinterpret_cast<const uint16_t*>(idx), b_row, ts,
                                                         ws, ws_bf16, out, out_dtype, vec, N, R);
  else
    t4_epilogue_kernel<int32_t><<<grid, block, 0, st>>>(mode, C, bs, top_q, reinterpret_cast<const int32_t*>(idx), b_row, ts,
                                                        ws, ws_bf16, out, out_dtype, vec, N, R);
  return check_launch();
}

__global__ void swiglu_quotients_kernel(float* __restrict__ quotient, float* __restrict__ divided) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;   // < 2^16
  const float g = bf16_bits_to_f32(i);
  quotient[i] = swiglu_quotient(g);
  divided[i] = __fdiv_rn(g, __fadd_rn(1.0f, expf(-g)));
}

}  // namespace

int run_transpose_bf16(const void* in, void* out, int N, int K, cudaStream_t st) {
  if (N % 8 == 0 && K % 8 == 0 && aligned16(in) && aligned16(out)) {
    transpose_bf16_8x8_kernel<<<dim3((K + 127) / 128, (N + 127) / 128), 256, 0, st>>>(
        reinterpret_cast<const uint16_t*>(in), reinterpret_cast<uint16_t*>(out), N, K);
    return check_launch();
  }
  dim3 block(32, 8), grid((K + 63) / 64, (N + 63) / 64);
  transpose_bf16_kernel<<<grid, block, 0, st>>>(reinterpret_cast<const uint16_t*>(in),
                                                reinterpret_cast<uint16_t*>(out), N, K);
  return check_launch();
}

int run_col_to_row_s4(const uint8_t* b_col, uint8_t* b_row, int N, int K, cudaStream_t st) {
  if (N % 8 == 0 && K % 32 == 0 && aligned16(b_col) && aligned16(b_row)) {
    col_to_row_s4_8x32_kernel<<<dim3((K + 511) / 512, (N + 127) / 128), 256, 0, st>>>(b_col, b_row, N, K);
    return check_launch();
  }
  dim3 block(128), grid((N / 2 + 127) / 128, K / 2);
  col_to_row_s4_kernel<<<grid, block, 0, st>>>(b_col, b_row, N, K);
  return check_launch();
}

}  // namespace tq

extern "C" int tq_transpose_bf16(const void* in, void* out, int N, int K, void* stream) {
  if (!in || !out || N < 0 || K < 0) return TQ_ERR_BAD_ARG;
  if (N == 0 || K == 0) return TQ_OK;
  return tq::run_transpose_bf16(in, out, N, K, (cudaStream_t)stream);
}

extern "C" int tq_swiglu_quotients(float* quotient, float* divided, void* stream) {
  if (!quotient || !divided) return TQ_ERR_BAD_ARG;
  tq::swiglu_quotients_kernel<<<256, 256, 0, (cudaStream_t)stream>>>(quotient, divided);
  return tq::check_launch();
}

extern "C" int tq_dequant_finish(const int32_t* C, const float* body_scale, const float* w_scale, const float* tail,
                                 const float* bias, void* out_bf16, int M, int N, void* stream) {
  if (!C || !body_scale || !w_scale || !out_bf16 || M < 0 || N <= 0) return TQ_ERR_BAD_ARG;
  if (M == 0) return TQ_OK;
  const size_t total = (size_t)M * N;
  tq::dequant_finish_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      C, body_scale, w_scale, tail, bias, reinterpret_cast<uint16_t*>(out_bf16), M, N);
  return tq::check_launch();
}

extern "C" int tq_dequant_finish_partials(const int32_t* partials, int splits, const float* body_scale,
                                          const float* w_scale, const float* tail, const float* bias, void* out_bf16,
                                          int M, int N, int act, void* stream) {
  if (!partials || splits < 1 || !body_scale || !w_scale || !out_bf16 || M < 0 || N <= 0 || act < 0 || act > 1)
    return TQ_ERR_BAD_ARG;
  if (act && (N & 1)) return TQ_ERR_UNSUPPORTED;
  if (M == 0) return TQ_OK;
  const size_t outputs = (size_t)M * N / (act ? 2 : 1);
  tq::dequant_finish_partials_kernel<<<(unsigned)((outputs + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      partials, splits, body_scale, w_scale, tail, bias, reinterpret_cast<uint16_t*>(out_bf16), M, N, act);
  return tq::check_launch();
}

extern "C" int tq_scale_sparse_epilogue(const int32_t* C, const float* body_scale, const int8_t* top_q,
                                        const int32_t* idx, const uint8_t* b_row, const float* top_scale,
                                        const float* w_scale, void* out, int out_dtype, int M, int N, int K, int R,
                                        void* stream) {
  return tq::t4_launch(0, C, body_scale, top_q, idx, 0, b_row, top_scale, w_scale, 0, out, out_dtype, M, N, K, R,
                       (cudaStream_t)stream);
}

extern "C" int tq_sparse_correction_add(void* out, int out_dtype, const int8_t* top_q, const int32_t* idx,
                                        const uint8_t* b_row, const float* top_scale, const void* w_scale,
                                        int w_scale_bf16, int M, int N, int K, int R, void* stream) {
  return tq::t4_launch(1, nullptr, nullptr, top_q, idx, 0, b_row, top_scale, w_scale, w_scale_bf16, out, out_dtype, M,
                       N, K, R, (cudaStream_t)stream);
}

extern "C" int tq_sparse_top_write(void* out, int out_dtype, const int8_t* top_q, const void* idx, int idx_u16,
                                   const uint8_t* b_row, const float* top_scale, const float* w_scale, int M, int N,
                                   int K, int R, void* stream) {
  return tq::t4_launch(2, nullptr, nullptr, top_q, idx, idx_u16, b_row, top_scale, w_scale, 0, out, out_dtype, M, N, K,
                       R, (cudaStream_t)stream);
}

extern "C" int tq_idx_i32_to_u16(const int32_t* idx, uint16_t* out, long long n, void* stream) {
  if (!idx || !out || n < 0) return TQ_ERR_BAD_ARG;
  if (n == 0) return TQ_OK;
  tq::idx_i32_to_u16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(idx, out, n);
  return tq::check_launch();
}
