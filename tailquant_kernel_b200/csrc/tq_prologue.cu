// Prologue of the split W4A4 + tail linear: entry points, argument checks and the choice between the two kernels
// (tq_prologue_wide.cu: 16 elements per thread, every built width; tq_prologue_fast.cu: 64 elements per thread).
#include <cmath>

#include "tq_common.cuh"
#include "tq_prologue.cuh"

namespace tq {
namespace {

float had_scale(int kind, int K) {
  if (kind == TQ_HAD_NONE) return 1.0f;
  const double n = (kind == TQ_HAD_BLOCK128) ? 128.0 : (double)K;
  return (float)(1.0 / sqrt(n));
}

}  // namespace

static int g_prologue_mode = -1;  // -1: by width and row count; 0: 16 elements per thread always

int run_prologue(const void* x, int M, int K, int had_kind, int R, int dr, float eps, int scale_mode,
                 uint8_t* a_pack, int8_t* a_q8, float* body_scale, float* top_scale, uint16_t* tail_idx16,
                 void* tail_val, int tail_ld, uint16_t* tail_ptr, int ptr_ld, uint32_t* tail_rec, uint16_t* tail_cnt,
                 int32_t* idx32, int8_t* top_q, void* x_rot, const void* gamma, float rms_eps, cudaStream_t st,
                 int dtype, void* tail_dense, const SparseTail* sparse) {
  if ((tail_idx16 || tail_val) && tail_ld < R) return TQ_ERR_BAD_ARG;
  if (gamma && !aligned16(gamma)) return TQ_ERR_MISALIGNED;
  if (tail_ptr && (ptr_ld < K / 128 + 1 || K % 128 != 0)) return TQ_ERR_BAD_ARG;
  if ((tail_rec != nullptr) != (tail_cnt != nullptr) || (tail_rec && K % 128 != 0)) return TQ_ERR_BAD_ARG;
  if (!x || (!a_pack && !a_q8) || !body_scale || M < 0 || K <= 0 || R < 0 || R >= K) return TQ_ERR_BAD_ARG;
  if (dr < 1 || dr > K) return TQ_ERR_BAD_ARG;
  if (!aligned16(x) || (a_pack && !aligned16(a_pack)) || (a_q8 && !aligned16(a_q8)) || (x_rot && !aligned16(x_rot)) ||
      (tail_dense && !aligned16(tail_dense)) ||
      (sparse && !(aligned16(sparse->val) && aligned16(sparse->meta))))
    return TQ_ERR_MISALIGNED;
  if (M == 0) return TQ_OK;
  PrologueParams p;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x);
  p.M = M;
  p.R = R;
  p.dr = dr;
  p.tail_ld = tail_ld;
  p.ptr_ld = ptr_ld;
  p.tail_ptr = tail_ptr;
  p.tail_rec = tail_rec;
  p.tail_cnt = tail_cnt;
  p.eps = eps;
  p.hscale = had_scale(had_kind, K);
  p.scale_mode = scale_mode;
  p.a_pack = a_pack;
  p.a_q8 = a_q8;
  p.body_scale = body_scale;
  p.top_scale = top_scale;
  p.tail_idx16 = tail_idx16;
  p.tail_val = reinterpret_cast<uint16_t*>(tail_val);
  p.idx32 = idx32;
  p.top_q = top_q;
  p.x_rot = reinterpret_cast<uint16_t*>(x_rot);
  p.tail_dense = reinterpret_cast<uint16_t*>(tail_dense);
  p.gamma = reinterpret_cast<const uint16_t*>(gamma);
  p.rms_eps = rms_eps;
  p.sp = SparseTail{};
  if (sparse && R > 0) {
    if (!sparse->val || !sparse->meta || !sparse->over_cnt || !sparse->over || sparse->over_ld < (R + 1) / 2) return TQ_ERR_BAD_ARG;
    p.sp = *sparse;
  }
  p.wide = ((reinterpret_cast<uintptr_t>(a_q8) | reinterpret_cast<uintptr_t>(x_rot) | reinterpret_cast<uintptr_t>(tail_dense) |
             reinterpret_cast<uintptr_t>(p.sp.val)) & 31) == 0;
  // 64 elements per thread issue fewer instructions per element, 16 give a row a quarter of the latency: the lines lie where
  // the rows no longer fit the chip at once (K = 4096: 9.2 against 9.8 us at 300 rows, 7.8 / 5.7 at 64; K = 12288, one
  // CTA of 768 threads per SM: 16.9 / 23.7 at 300, 10.0 / 9.2 at 61).
  if (g_prologue_mode != 0 && M > (K <= 4096 ? 256 : 128)) {
    const int rc = run_prologue_fast(had_kind, K, dtype, p, st);
    if (rc != TQ_ERR_UNSUPPORTED) return rc;
  }
  return run_prologue_wide(had_kind, K, dtype, p, st);
}

}  // namespace tq

extern "C" int tq_split_prologue(const void* x, int M, int K, int had_kind, int R, int descending_rank,
                                 float eps, uint8_t* a_pack, int8_t* a_q8, float* body_scale, float* top_scale,
                                 uint16_t* tail_idx16, void* tail_val, int tail_ld, uint16_t* tail_ptr,
                                 int ptr_ld, uint32_t* tail_rec, uint16_t* tail_cnt, void* tail_dense, int32_t* idx32,
                                 int8_t* top_q, void* x_rot, void* stream) {
  return tq::run_prologue(x, M, K, had_kind, R, descending_rank, eps, 0, a_pack, a_q8, body_scale, top_scale,
                          tail_idx16, tail_val, tail_ld, tail_ptr, ptr_ld, tail_rec, tail_cnt, idx32, top_q, x_rot,
                          nullptr, 0.0f, (cudaStream_t)stream, TQ_BF16, tail_dense);
}

extern "C" int tq_set_prologue_mode(int mode) {
  if (mode < -1 || mode > 1) return TQ_ERR_BAD_ARG;
  tq::g_prologue_mode = mode;
  return TQ_OK;
}

extern "C" int tq_split_prologue_rmsnorm(const void* x, const void* gamma, float rms_eps, int M, int K, int had_kind,
                                         int R, int descending_rank, float eps, uint8_t* a_pack, int8_t* a_q8,
                                         float* body_scale, float* top_scale, uint16_t* tail_idx16, void* tail_val,
                                         int tail_ld, uint16_t* tail_ptr, int ptr_ld, uint32_t* tail_rec,
                                         uint16_t* tail_cnt, void* tail_dense, void* x_rot, void* stream) {
  if (!gamma) return TQ_ERR_BAD_ARG;
  return tq::run_prologue(x, M, K, had_kind, R, descending_rank, eps, 0, a_pack, a_q8, body_scale, top_scale,
                          tail_idx16, tail_val, tail_ld, tail_ptr, ptr_ld, tail_rec, tail_cnt, nullptr, nullptr, x_rot,
                          gamma, rms_eps, (cudaStream_t)stream, TQ_BF16, tail_dense);
}

extern "C" int tq_topr_pack(const void* A, int dtype, int M, int K, int R, int descending_rank,
                            uint8_t* A_pack, float* body_scale, float* top_scale, int8_t* top_q,
                            int32_t* idx, float eps, void* stream) {
  if (dtype != TQ_BF16 && dtype != TQ_FP16) return TQ_ERR_BAD_ARG;
  if (R > 0 && (!top_q || !idx || !top_scale)) return TQ_ERR_BAD_ARG;
  return tq::run_prologue(A, M, K, TQ_HAD_NONE, R, descending_rank, eps, 0, A_pack, nullptr, body_scale, top_scale,
                          nullptr, nullptr, 0, nullptr, 0, nullptr, nullptr, idx, top_q, nullptr, nullptr, 0.0f,
                          (cudaStream_t)stream, dtype, nullptr);
}
