// The forward of one linear as ONE host call: prologue and fused linear enqueued back to back.  The Python layer used
// to issue every kernel, event and scratch buffer of a forward itself (about 70 us of host time per small call, five
// times the GPU's); it now fills a tq_linear_call once per (layer, row count) and passes it with the two pointers that
// change.
#include "tq_common.cuh"

namespace tq {
namespace {

// Whether the operands of the pair kernel's tail are there.
bool has_records(const tq_linear_call& c) { return c.tail_idx16 && c.tail_val && c.tail_ptr && c.tail_rec && c.tail_cnt; }

// Whether the fused engine of this call runs the stream kernel (which reads the tail from the zero-filled matrix).
bool linear_streams(const tq_linear_call& c) {
  if (c.engine != TQ_LINEAR_FUSED || c.M <= 0) return false;
  return c.R == 0 ? stream_is_faster(c.M, c.N, c.K, 0) : c.tail_dense && (!has_records(c) || stream_is_faster(c.M, c.N, c.K, c.R));
}

// Rows beyond which the zero-filled matrix is not kept whatever it would save (layers whose pair kernel reads it excepted).
constexpr int DENSE_MAX_ROWS = 4096;

// Whether the kernel is built for the sizes of the call (its stores of SwiGLU outputs are 16 bytes wide).
bool sparse_fits(const tq_linear_call& c) { return c.K % 512 == 0 && c.N % (c.act ? 16 : 8) == 0 && c.K <= 65536; }

// Whether a linear can take its tail as a 2:4-sparse operand: a full rotation, which spreads the entries over K, and few enough of
// them that a group of four rarely holds more than two.  (At R = 0.1 K the left-over entries outweigh what the sparse product
// saves, and rows with a few large channels have twice as many.)
bool tail_can_be_sparse(const tq_linear_call& c) {
  return c.engine == TQ_LINEAR_FUSED && (c.had_kind == TQ_HAD_WHT || c.had_kind == TQ_HAD_KRON12) && c.R > 0 && sparse_fits(c) &&
         (long)c.R * 100 <= 7l * c.K;
}

// Whether the sparse form is the fastest for this call.
bool linear_sparse(const tq_linear_call& c) { return tail_can_be_sparse(c) && sparse_is_faster(c.M, c.N, c.K, c.R); }

// Whether a linear of some width on the prologue of this call may take it.
bool shared_sparse(const tq_linear_call& c) { return tail_can_be_sparse(c) && g_gemm_pair_mode < 0 && c.M > 64; }

// Whether a fused call runs on the sparse form that it holds: where that is the fastest, and where nothing faster is there (the
// prologue filled what the kernel of ANOTHER width reads).
bool takes_sparse(const tq_linear_call& c) {
  if (!c.sp_val || c.M == 0 || c.R == 0) return false;
  if (linear_sparse(c)) return true;
  if (has_records(c)) return false;
  // (without w_t the left-over entries cost more than the zero-filled matrix does)
  return !c.tail_dense || (c.w_t && shared_sparse(c) && sparse_us(c.M, c.N, c.K, c.R) < plan_stream(c.M, c.N, c.K, ST_TAIL).us);
}

SparseTail linear_sparse_tail(const tq_linear_call& c) {
  return SparseTail{reinterpret_cast<uint16_t*>(c.sp_val), c.sp_meta, c.sp_over_cnt, c.sp_over, c.sp_over_ld};
}

// THE rule for the buffers of a workspace (see tailquant.h); which kernel then runs follows from what is there.
int linear_outputs(const tq_linear_call& c, bool shared) {
  const bool fused = c.engine == TQ_LINEAR_FUSED;
  int o = fused ? TQ_OUT_Q8 : TQ_OUT_PACK;
  const bool few = shared && c.engine != TQ_LINEAR_GATHER && c.M <= 64;   // decode or fused, either may come
  if (few) o = TQ_OUT_Q8 | TQ_OUT_PACK;
  if (c.R == 0) return o;
  const bool pair_dense = c.had_kind == TQ_HAD_BLOCK128;   // (the pair kernel loads long runs from it)
  if (few) return o | TQ_OUT_LISTS | TQ_OUT_DENSE;
  if (!fused) return o | TQ_OUT_LISTS;
  if (c.sp_val && !shared && linear_sparse(c)) return o | TQ_OUT_LISTS;
  // (the sparse form and the zero-filled matrix serve every width between them)
  if (c.sp_val && shared && shared_sparse(c) && c.M <= DENSE_ROWS)
    return o | TQ_OUT_LISTS | TQ_OUT_DENSE | linear_outputs(c, false);
  const bool streams = c.M <= DENSE_MAX_ROWS && stream_is_faster(c.M, c.N, c.K, c.R);
  if (shared || !streams) o |= TQ_OUT_LISTS | TQ_OUT_RECORDS;
  if (streams || pair_dense || (shared && c.M <= DENSE_ROWS)) o |= TQ_OUT_DENSE;
  return o;
}

// The part of a workspace that a forward of this call fills and reads; a prologue on its own fills every array that is there,
// since another linear, of another width and hence perhaps on another kernel, may run on it.  The sorted tail lists and the
// records cost a small call about 3 us, the zero-filled matrix a large one 2 bytes per element.
tq_linear_call linear_own_part(tq_linear_call c) {
  const bool fused = c.engine == TQ_LINEAR_FUSED;
  if (fused)
    c.a_pack = nullptr;
  else
    c.a_q8 = nullptr;
  if (fused && takes_sparse(c)) {
    c.tail_dense = nullptr;
    c.tail_ptr = nullptr;
    c.tail_rec = nullptr;
    c.tail_cnt = nullptr;
    return c;
  }
  const bool streams = linear_streams(c);
  if (streams) {
    c.tail_idx16 = nullptr;
    c.tail_val = nullptr;
  }
  c.sp_val = nullptr;
  if (!fused || streams) {
    c.tail_ptr = nullptr;
    c.tail_rec = nullptr;
    c.tail_cnt = nullptr;
  }
  if (!streams && !(fused && c.had_kind == TQ_HAD_BLOCK128)) c.tail_dense = nullptr;
  return c;
}

int linear_prologue(const tq_linear_call& c, const void* x, void* stream) {
  const SparseTail sp = linear_sparse_tail(c);
  return run_prologue(x, c.M, c.K, c.had_kind, c.R, c.descending_rank, c.eps, 0, c.a_pack, c.a_q8, c.body_scale,
                      c.top_scale, c.tail_idx16, c.tail_val, c.tail_ld, c.tail_ptr, c.ptr_ld, c.tail_rec, c.tail_cnt,
                      nullptr, nullptr, nullptr, c.rms_weight, c.rms_eps, (cudaStream_t)stream, TQ_BF16, c.tail_dense,
                      sp.val ? &sp : nullptr);
}

// `early`: the prologue of this call is the kernel in front
int linear_compute(const tq_linear_call& c, void* out, bool early, void* stream) {
  if (c.engine == TQ_LINEAR_DECODE) {
    if (!c.a_pack || !c.body_scale || !c.b_col || !c.w_scale || !out || c.M < 0 || c.M > 64 || c.R < 0 || c.R >= c.K)
      return TQ_ERR_BAD_ARG;
    if (c.R > 0 && (!c.w_t || !c.tail_idx16 || !c.tail_val || c.tail_ld < c.R)) return TQ_ERR_BAD_ARG;
    if (!aligned16(c.a_pack) || !aligned16(c.b_col) || (c.R > 0 && !aligned16(c.w_t))) return TQ_ERR_MISALIGNED;
    if (c.M == 0) return TQ_OK;
    DecodeLinearParams p = {};
    p.a_pack = c.a_pack;
    p.sx = c.body_scale;
    p.idx = c.tail_idx16;
    p.val = reinterpret_cast<const uint16_t*>(c.tail_val);
    p.b_col = c.b_col;
    p.w_t = reinterpret_cast<const uint16_t*>(c.w_t);
    p.sw = c.w_scale;
    p.bias = c.bias;
    p.out = reinterpret_cast<uint16_t*>(out);
    p.M = c.M;
    p.N = c.N;
    p.K = c.K;
    p.R = c.R;
    p.ld = c.tail_ld;
    p.act = c.act;
    p.early = early ? 1 : 0;
    return run_decode_linear(p, c.tail, (cudaStream_t)stream);
  }
  if (c.engine == TQ_LINEAR_GATHER) {
    if (c.R > 0) {
      const int rc = tq_tail_gather(c.tail_idx16, c.tail_val, c.w_t, c.tail, c.M, c.N, c.K, c.R, c.tail_ld, stream);
      if (rc != TQ_OK) return rc;
    }
    return tq_split_gemm_fused(c.a_pack, c.body_scale, c.b_col, c.w_scale, c.R > 0 ? c.tail : nullptr, c.bias, out, c.M,
                               c.N, c.K, stream);
  }
  if (c.engine != TQ_LINEAR_FUSED) return TQ_ERR_BAD_ARG;
  if (takes_sparse(c)) {
    if (!c.a_q8 || !c.body_scale || !c.b_col || !c.w_scale || !c.w_rot || !out || !c.sp_meta || !c.sp_over_cnt ||
        !c.sp_over || c.sp_over_ld < (c.R + 1) / 2 || c.N <= 0 || c.K <= 0 || c.R >= c.K)
      return TQ_ERR_BAD_ARG;
    if (!sparse_fits(c)) return TQ_ERR_UNSUPPORTED;
    if (!aligned16(c.a_q8) || !aligned16(c.b_col) || !aligned16(out) || !aligned16(c.w_scale) || !aligned16(c.w_rot) ||
        !aligned16(c.w_t) || !aligned16(c.sp_over_cnt) || !aligned16(c.sp_val) || !aligned16(c.sp_meta) ||
        (c.bias && !aligned16(c.bias)))
      return TQ_ERR_MISALIGNED;
    return run_sparse_gemm(c.a_q8, c.body_scale, c.b_col, c.w_scale, c.w_rot, c.w_t, linear_sparse_tail(c), c.bias, out, nullptr,
                           nullptr, c.M, c.N, c.K, c.act, early, (cudaStream_t)stream);
  }
  return run_split_gemm_mma(c.a_q8, c.body_scale, c.b_col, c.w_scale, c.w_rot, c.tail_idx16, c.tail_val, c.tail_ld,
                            c.tail_ptr, c.ptr_ld, c.tail_rec, c.tail_cnt, c.tail_dense, c.R, c.bias, out, nullptr, nullptr,
                            c.M, c.N, c.K, c.act, early, stream);
}

}  // namespace
}  // namespace tq

extern "C" int tq_linear_outputs(const tq_linear_call* call, int shared) {
  if (!call || call->M < 0 || call->N <= 0 || call->K <= 0 || call->R < 0 || call->R >= call->K ||
      call->engine < TQ_LINEAR_DECODE || call->engine > TQ_LINEAR_GATHER)
    return TQ_ERR_BAD_ARG;
  return tq::linear_outputs(*call, shared != 0);
}

extern "C" int tq_linear_sparse(const tq_linear_call* call, int shared) {
  if (!call || call->M < 0 || call->N <= 0 || call->K <= 0 || call->R < 0 || call->R >= call->K) return TQ_ERR_BAD_ARG;
  return (shared ? tq::shared_sparse(*call) : tq::linear_sparse(*call)) ? 1 : 0;
}

extern "C" int tq_linear_forward(const tq_linear_call* call, const void* x, void* out, void* stream) {
  if (!call) return TQ_ERR_BAD_ARG;
  const tq_linear_call own = tq::linear_own_part(*call);
  const int rc = tq::linear_prologue(own, x, stream);
  return rc != TQ_OK ? rc : tq::linear_compute(own, out, true, stream);
}

extern "C" int tq_linear_prologue(const tq_linear_call* call, const void* x, void* stream) {
  return call ? tq::linear_prologue(*call, x, stream) : TQ_ERR_BAD_ARG;
}

extern "C" int tq_linear_compute(const tq_linear_call* call, void* out, void* stream) {
  return call ? tq::linear_compute(*call, out, false, stream) : TQ_ERR_BAD_ARG;
}
