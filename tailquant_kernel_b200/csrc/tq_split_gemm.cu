// Split GEMM with the tail on the tensor cores: entry points and the choice of the kernel.
//   out[m,n] = bf16( (float(sum_k qx[m,k] qw[n,k]) * s_x[m]) * s_w[n]  +  sum_r x_tail[m,r] W_rot[n, idx[m,r]]  + bias[n] )
// with the dense part on tcgen05 kind::i8 (int32 accumulator in tensor memory) and the tail on tcgen05 kind::f16 (bf16 x
// bf16, fp32 accumulator in tensor memory) over the zero-filled tail matrix.
//
// Why not gather: after the rotation the tail positions are spread uniformly over K, so the gathered form is M*R*N
// scalar multiply-adds with no operand reuse; on this GPU the dense bf16 MMA over a K-wide, 95 %-zero operand is several
// times faster than that at ratio 0.05.  The exact-order gather kernel (tq_tail.cu) stays available as the bit-exact mode.
//
// The activation codes arrive as INT8 with the two nibble planes of each 8-element group de-interleaved
// ([0,2,4,6,1,3,5,7]), which is the order the widening of the weights produces, so both operands see the same permutation
// of K and the dot product is unchanged.  Weights carry a factor 16 (the nibble is kept in the top half of the byte,
// which makes it sign-correct without an extension), removed by an exact >> 4 of the accumulator.
//
// Reference behaviour covered: GEMM + dequant + sparse correction in one kernel, i.e. what the reference prototypes in
// tools/quarot_split_fused_epilogue_ext_v1.py:283-432 and tools/qfactory_split_fused_epilogue_v1.py:153-233 (there with an
// INT4 tail and R fixed at compile time).
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace tq {
namespace {

// Diagnostic build (-DTQ_GEMM_PROFILE): cycles each role spends in its barrier waits, summed over CTAs, in
// g_wait_cycles[code]; read back with tq_gemm_wait_cycles().  Compiled out otherwise.
#ifdef TQ_GEMM_PROFILE
__device__ unsigned long long g_wait_cycles[16];
#define TQ_WAIT(slot, call)                                                        \
  [&]() -> bool {                                                                  \
    const long long t0_ = clock64();                                               \
    const bool r_ = (call);                                                        \
    atomicAdd(&g_wait_cycles[slot], (unsigned long long)(clock64() - t0_));        \
    return r_;                                                                     \
  }()
#else
#define TQ_WAIT(slot, call) (call)
#endif

// Diagnostic build (-DTQ_GEMM_TRACE): clock64 stamps of CTA 0's roles in the pair kernel for slot uses [TQ_TRACE_Q0, +128),
// in g_trace[role][use][event]; read back with tq_gemm_trace().  Compiled out otherwise.
//   role 0 MMA issuer, 1 INT8 activations, 2 bf16 weight rows, 6 packed weights: 0 = wait begun, 1 = wait over, 2 = issued
//   role 3 wideners: 0 / 1 / 2 = before and after the wait for the staging buffer, after that for the slot, 3 = done
//   role 4 builders: 0 / 1 = before and after the wait for the slot, 3 = records scattered, 2 = arrived; role 5: 2 = zeroed,
//   0 / 1 = before and after the proxy fence
#ifdef TQ_GEMM_TRACE
#ifndef TQ_TRACE_Q0
#define TQ_TRACE_Q0 30
#endif
__device__ unsigned long long g_trace[8][128][4];
#define TQ_TRACE(role, q, ev)                                                              \
  do {                                                                                     \
    if (blockIdx.x == 0 && (q) >= TQ_TRACE_Q0 && (q) < TQ_TRACE_Q0 + 128)                  \
      g_trace[role][(q) - TQ_TRACE_Q0][ev] = (unsigned long long)clock64();                \
  } while (0)
#define TQ_TRACE_ONLY(...) __VA_ARGS__
#else
#define TQ_TRACE(role, q, ev) do { } while (0)
#define TQ_TRACE_ONLY(...)
#endif

}  // namespace

// -1 = choose by shape, 0 = the kernel for few and medium row counts wherever it can run, 1 = CTA pairs (set by
// tq_set_gemm_pair_mode only)
static int g_gemm_pair_mode = -1;
int run_pair_gemm(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col, const float* w_scale,
                  const void* w_rot, const uint16_t* tail_idx16, const void* tail_val, int tail_ld,
                  const uint16_t* tail_ptr, int ptr_ld, const uint32_t* tail_rec, const uint16_t* tail_cnt,
                  const void* tail_dense, int R, const float* bias, void* out_bf16, int32_t* dbg_acc, float* dbg_tail,
                  int M, int N, int K, int act, cudaStream_t st);
int run_sparse_gemm(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col, const float* w_scale, const void* w_rot,
                    const void* w_t, const SparseTail& sp, const float* bias, void* out_bf16, int32_t* dbg_acc, float* dbg_tail,
                    int M, int N, int K, int act, bool early, cudaStream_t st);
}  // namespace tq

#ifdef TQ_GEMM_PROFILE
extern "C" int tq_gemm_wait_cycles(unsigned long long* out16, int reset) {
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(out16, tq::g_wait_cycles, sizeof(unsigned long long) * 16);
  if (reset) {
    unsigned long long z[16] = {};
    cudaMemcpyToSymbol(tq::g_wait_cycles, z, sizeof(z));
  }
  return 0;
}
#endif

#ifdef TQ_GEMM_TRACE
extern "C" int tq_gemm_trace(unsigned long long* out, int reset) {
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(out, tq::g_trace, sizeof(unsigned long long) * 8 * 128 * 4);
  if (reset) {
    static unsigned long long z[8 * 128 * 4] = {};
    cudaMemcpyToSymbol(tq::g_trace, z, sizeof(z));
  }
  return 0;
}
#endif

extern "C" int tq_set_gemm_pair_mode(int mode) {
  if (mode < -1 || mode > 1) return TQ_ERR_BAD_ARG;
  tq::g_gemm_pair_mode = mode;
  return TQ_OK;
}

namespace tq {

// The zero-filled tail matrix (2 M K bytes) is worth its memory up to this many rows, and beyond them for narrow layers
// only, up to this many outputs: 1174 x 1200 x 14336 takes 63 us instead of 120.
constexpr int DENSE_ROWS = 1024;
constexpr long DENSE_OUTPUTS = 1 << 21;

// Which kernel a call takes: true = tq_gemm_stream.cu (128 channels x up to 176 rows per tile, 256 without a tail, K
// split over a cluster),
// false = tq_gemm_pair.cu (256 x 256 tiles on CTA pairs).  Both estimates are fits to timings on the layer shapes; the
// pair kernel goes through ceil(tiles / 74) rounds of 1.02 us per K slice and 5 us with a tail (0.34 and 3.5 without), and
// takes about 5 us for the launch and ring fill.  At N = K = 4096 the line lies between 700 and 1000 rows, at
// N = 28672 between 100 and 176.
static float pair_us(int M, int N, int K, int R) {
  const int tiles = ((M + 255) / 256) * ((N + 255) / 256), rounds = (tiles + 73) / 74;
  return R > 0 ? rounds * ((K / 128) * 1.02f + 5.0f) + 5.0f : rounds * ((K / 128) * 0.34f + 3.5f) + 6.0f;
}
static bool stream_can(int M, int N, int R) { return M <= DENSE_ROWS || R == 0 || (long)M * N <= DENSE_OUTPUTS; }
static bool stream_is_faster(int M, int N, int K, int R) {
  if (g_gemm_pair_mode >= 0) return g_gemm_pair_mode == 0;
  if (M <= 64) return true;
  return stream_can(M, N, R) && plan_stream(M, N, K, R > 0 ? ST_TAIL : ST_INT8).us < pair_us(M, N, K, R);
}

// The kernel with the 2:4-sparse tail (tq_gemm_sparse.cu): ceil(tiles / 74) rounds of 0.55 us per K slice and 3.7 us (narrow last
// tiles take as long as full ones), a share of the weight stream, and 0.08 us for each left-over entry among four rows of a
// tile; 5.5 us around it, 1.5 of them in the prologue.  `e`: left-over entries of a row whose R entries lie independently.  Fit
// to 200 shapes (80..2048 rows, N = 1024..28672, K = 1024, 4096, 12288, R = 0.05 K): 5 % off on average, 0.4 % lost by the
// choice.  300 x 24576 x 4096: 88 us, 118 and 122 on the other two; 2048 x 4096 x 4096: 68 against 81 on pairs.  At the ends, whole
// linears on 13 shapes (128..4096 rows, K = 512..12288) each at R = 0.001, 0.01, 0.05, 0.069 K: 0.9 % lost on average, nearly all
// of it by staying with the pairs where many entries make few rounds look long (1500 x 28672 x 512, 0.069 K: 124 us, 101
// here; 4096 x 2048 x 1024 62 and 54); where the rule takes this kernel the best of the others is at most 2.4 % ahead (520 x 4096 x
// 8192, 0.05 K: 85 against 83), and without left-over entries (0.001 K) 2048 x 6144 x 4096 takes 120 against 144.
static float sparse_us(int M, int N, int K, int R) {
  const int rounds = (((M + 255) / 256) * ((N + 223) / 224) + 73) / 74;
  const float q = (float)R / (float)K, e = (float)K * q * q * q * (1.0f - 0.5f * q);
  return rounds * ((K / 128) * 0.55f + 3.7f + 5.2f * e) + 5.5f + 1.25e-7f * (float)N * (float)K;
}
static bool sparse_is_faster(int M, int N, int K, int R) {
  if (g_gemm_pair_mode >= 0 || M <= 64) return false;
  const float us = sparse_us(M, N, K, R);
  return us < pair_us(M, N, K, R) && (!stream_can(M, N, R) || us < plan_stream(M, N, K, ST_TAIL).us);
}

static int run_split_gemm_mma(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col,
                              const float* w_scale, const void* w_rot, const uint16_t* tail_idx16,
                              const void* tail_val, int tail_ld, const uint16_t* tail_ptr, int ptr_ld,
                              const uint32_t* tail_rec, const uint16_t* tail_cnt, const void* tail_dense, int R,
                              const float* bias, void* out_bf16, int32_t* dbg_acc, float* dbg_tail, int M, int N, int K,
                              int act, bool early, void* stream) {
  if (!a_q8 || !body_scale || !b_col || !w_scale || !out_bf16 || M < 0 || N <= 0 || K <= 0 || R < 0 || R >= K)
    return TQ_ERR_BAD_ARG;
  const bool records = tail_idx16 && tail_val && tail_ld >= R && tail_ptr && ptr_ld >= K / 128 + 1 && tail_rec && tail_cnt;
  if (R > 0 && (!w_rot || (!records && !tail_dense))) return TQ_ERR_BAD_ARG;
  if (K % 128 != 0 || N % 8 != 0 || K > 65536) return TQ_ERR_UNSUPPORTED;
  if (!aligned16(a_q8) || !aligned16(b_col) || !aligned16(out_bf16) || !aligned16(w_scale) ||
      (R > 0 && !aligned16(w_rot)) || (bias && !aligned16(bias)) || (dbg_acc && !aligned16(dbg_acc)) ||
      (dbg_tail && !aligned16(dbg_tail)) || (tail_dense && !aligned16(tail_dense)))
    return TQ_ERR_MISALIGNED;
  if (M == 0) return TQ_OK;
  // (the stream kernel reads the tail from the zero-filled matrix, the pair kernel from the records)
  if (R > 0 ? (tail_dense && (!records || stream_is_faster(M, N, K, R))) : stream_is_faster(M, N, K, R))
    return run_stream_gemm(a_q8, body_scale, b_col, w_scale, w_rot, tail_dense, R, bias, out_bf16, dbg_acc, dbg_tail, M, N,
                           K, act, early, (cudaStream_t)stream);
  return run_pair_gemm(a_q8, body_scale, b_col, w_scale, w_rot, tail_idx16, tail_val, tail_ld, tail_ptr, ptr_ld, tail_rec,
                       tail_cnt, tail_dense, R, bias, out_bf16, dbg_acc, dbg_tail, M, N, K, act, (cudaStream_t)stream);
}
}  // namespace tq

extern "C" int tq_split_gemm_mma(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col,
                                 const float* w_scale, const void* w_rot, const uint16_t* tail_idx16,
                                 const void* tail_val, int tail_ld, const uint16_t* tail_ptr, int ptr_ld,
                                 const uint32_t* tail_rec, const uint16_t* tail_cnt, const void* tail_dense, int R,
                                 const float* bias, void* out_bf16,
                                 int32_t* dbg_acc, float* dbg_tail, int M, int N, int K, void* stream) {
  return tq::run_split_gemm_mma(a_q8, body_scale, b_col, w_scale, w_rot, tail_idx16, tail_val, tail_ld, tail_ptr,
                                ptr_ld, tail_rec, tail_cnt, tail_dense, R, bias, out_bf16, dbg_acc, dbg_tail, M, N, K, 0,
                                false, stream);
}

extern "C" int tq_split_gemm_mma_swiglu(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col,
                                        const float* w_scale, const void* w_rot, const uint16_t* tail_idx16,
                                        const void* tail_val, int tail_ld, const uint16_t* tail_ptr, int ptr_ld,
                                        const uint32_t* tail_rec, const uint16_t* tail_cnt, const void* tail_dense,
                                        int R, const float* bias, void* out_bf16, int M, int N, int K, void* stream) {
  return tq::run_split_gemm_mma(a_q8, body_scale, b_col, w_scale, w_rot, tail_idx16, tail_val, tail_ld, tail_ptr,
                                ptr_ld, tail_rec, tail_cnt, tail_dense, R, bias, out_bf16, nullptr, nullptr, M, N, K, 1,
                                false, stream);
}
