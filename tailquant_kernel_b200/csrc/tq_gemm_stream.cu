// Split GEMM for few and medium row counts (sm_100a): the computation of tq_gemm_pair.cu on tiles of 128 output channels
// x T token rows (T a multiple of 16, at most 176; 256 for INT8 codes without a tail), the K range of a tile shared by a
// CLUSTER of S CTAs.
//
// What bounds it: up to a few hundred rows every weight byte (N K / 2 packed INT4 + 2 N K bf16) is used for so few rows
// that the weight stream is the floor, and 256 x 256 or 128 x 256 tiles leave most of the chip without work (32 tiles
// for N = 4096 at 300 rows).  Hence
//   * the WEIGHTS are the 128-row operand of tcgen05.mma and the tokens the N operand, so a tile does no work for rows
//     that only pad M to 128, and the slots of the ring spend their bytes on weights;
//   * S CTAs take S ranges of K; their int32 / fp32 accumulators meet over distributed shared memory (one pass, no
//     global scratch, no atomics; the integer part stays exact) and CTA r finishes rows [r T / S, (r+1) T / S);
//   * the tail operand is loaded by TMA from the zero-filled tail matrix of the prologue like every other operand: no
//     builder warps, and the cost does not depend on how the tail entries are distributed;
//   * the kernel is a programmatic dependent of the prologue: its weight loads fill the ring while the prologue runs.
//
// Operands come in two rings.  INT8 slots hold the T x 128 B token codes of a 128-wide K slice; its weights arrive as INT4
// by TMA in a staging buffer and are widened x16 by four warps (eight without a tail) into 32 columns of tensor memory,
// where the MMA reads them.  bf16 slots hold [128 rows x 128 B weights | T rows x 128 B tail] for HB 64-wide halves of a
// slice, one tiled load per operand for all of them.
// Warp roles: 0 = producer of packed weights, 1 = MMA issuer (+ tensor memory), 2 = producer of the bf16 weight rows,
// 3 = producer of the token operands, 4.. = wideners, of which 4..7 then export the accumulators; all warps share the final
// reduction.
// (One thread that waits for a slot, announces its bytes and issues its loads takes about 400 cycles per load: with one
// producer for everything a K slice took 2700 cycles however few rows there were.)
// Every mbarrier wait is bounded (see mbar_wait).
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace tq {
namespace {

// operands of a call: INT8 codes + tail rows; INT8 codes alone; packed INT4 codes alone
enum : int { ST_TAIL = 0, ST_INT8 = 1, ST_PACKED = 2 };
// Four warps with other roles, then widening groups of four: a group takes about 700 cycles per slice whatever its size
// (wait, load, store, proxy fence, arrival one after the other), which hides behind the bf16 MMAs of a tail; without one it
// bounds the slice, so two groups take the even and the odd slices (and two more the packed token codes).
__host__ __device__ constexpr int st_threads(int mode) { return mode == ST_TAIL ? 256 : mode == ST_INT8 ? 384 : 640; }
// packed staging buffers; with two groups this and the number of INT8 slots are even: a buffer then always belongs to the
// same group, and no group can fall two phases behind a barrier it waits on by parity
__host__ __device__ constexpr int st_sp(int mode) { return mode == ST_TAIL ? 3 : 4; }
constexpr int ST_MAX_SP = 4;
constexpr int ST_STAGE = 128 * 64;    // [128 channels][128 k] INT4
constexpr int ST_MAX_SLOTS = 8;       // slots of either ring
// rows per tile: with a tail the exchange buffer (8 bytes per accumulator pair) must fit in the rings, packed tokens need
// staging buffers besides
__host__ __device__ constexpr int st_max_t(int mode) { return mode == ST_INT8 ? 256 : 176; }
constexpr int ST_MAX_T = 256;
constexpr int ST_SMEM = 222 * 1024;
constexpr int ST_BARS = 4 * ST_MAX_SP + 4 * ST_MAX_SLOTS + 1;

struct StreamParams {
  int M, N, K, T, act, tiles_n;
  int si, sb;   // INT8 slots, bf16 slots
  int early;    // the weights may be read before the kernel in front has ended (it has waited for all others itself)
  const float* sx;
  const float* sw;
  const float* bias;
  uint16_t* out;
  int32_t* dbg_acc;
  float* dbg_tail;
  const float* add;   // PK: [M, N] tail sums computed elsewhere, or NULL
  int32_t* C;         // PK: [M, N] the int32 accumulators instead of `out`, or NULL
};

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// INT4 -> INT8 (x16) of `rows` rows of 64 packed bytes by 128 threads: staging -> 128-byte-swizzled operand tile
__device__ __forceinline__ void widen_rows(const unsigned char* src, unsigned char* dst, int rows, int wtid) {
#pragma unroll 4
  for (int task = wtid; task < rows * 4; task += 128) {
    const int row = task >> 2, pc = task & 3;
    const uint4 w = *reinterpret_cast<const uint4*>(src + row * 64 + pc * 16);
    unsigned char* drow = dst + (row >> 3) * 1024 + (row & 7) * 128;
    uint4 lo, hi;
    lo.x = (w.x << 4) & 0xf0f0f0f0u;
    lo.y = w.x & 0xf0f0f0f0u;
    lo.z = (w.y << 4) & 0xf0f0f0f0u;
    lo.w = w.y & 0xf0f0f0f0u;
    hi.x = (w.z << 4) & 0xf0f0f0f0u;
    hi.y = w.z & 0xf0f0f0f0u;
    hi.z = (w.w << 4) & 0xf0f0f0f0u;
    hi.w = w.w & 0xf0f0f0f0u;
    *reinterpret_cast<uint4*>(drow + (((2 * pc) ^ (row & 7)) << 4)) = lo;
    *reinterpret_cast<uint4*>(drow + (((2 * pc + 1) ^ (row & 7)) << 4)) = hi;
  }
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// INT4 -> INT8 (x16) of one channel's 64 packed bytes (64-byte swizzle: conflict-free) into its lane of tensor memory
__device__ __forceinline__ void widen_row_tmem(const unsigned char* src, uint32_t taddr, int row) {
  uint32_t r[32];
#pragma unroll
  for (int pc = 0; pc < 4; ++pc) {
    const uint4 w = *reinterpret_cast<const uint4*>(src + row * 64 + ((pc ^ ((row >> 1) & 3)) << 4));
    const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[pc * 8 + 2 * i] = (v[i] << 4) & 0xf0f0f0f0u;
      r[pc * 8 + 2 * i + 1] = v[i] & 0xf0f0f0f0u;
    }
  }
  tmem_st32(taddr, r);
}

// HB: 64-wide halves per bf16 slot.  ST_PACKED: `tmap_a8` covers the [M, K/2] packed bytes, and further warps widen the
// token codes the way the weights are.
template <int HB, int MODE>
__global__ void __launch_bounds__(st_threads(MODE), 1)
stream_gemm_kernel(const __grid_constant__ CUtensorMap tmap_b4, const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_a8, const __grid_constant__ CUtensorMap tmap_tail,
                   const StreamParams p) {
  constexpr bool PK = MODE == ST_PACKED, has_tail = MODE == ST_TAIL;
  constexpr int ST_SP = st_sp(MODE), GROUPS = has_tail ? 1 : 2;
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* sm = smem_dyn + (base - raw);

  const int T = p.T, SI = p.si, SB = p.sb;
  const uint32_t slot_bytes = (uint32_t)(128 + T) * 128u;
  const uint32_t i8_bytes = (uint32_t)T * 128u;            // INT8 slots: tokens (the widened weights are in tensor memory)
  const uint32_t bf_off = (uint32_t)SI * i8_bytes;
  const uint32_t bf_bytes = (uint32_t)HB * slot_bytes;   // [HB][128 rows] weights, then [HB][T rows] tail
  const uint32_t stage_off = bf_off + (uint32_t)SB * bf_bytes;
  const uint32_t tok_off = stage_off + ST_SP * ST_STAGE;   // PK: token staging buffers, [T rows][64 bytes]
  const uint32_t bar_off = tok_off + (PK ? (uint32_t)(ST_SP * T * 64) : 0u);
  const uint32_t bars = base + bar_off;
  auto full_p = [&](int s) { return bars + 8u * s; };
  auto empty_p = [&](int s) { return bars + 8u * (ST_SP + s); };
  auto full_i = [&](int s) { return bars + 8u * (2 * ST_SP + s); };
  auto empty_i = [&](int s) { return bars + 8u * (2 * ST_SP + ST_MAX_SLOTS + s); };
  auto full_b = [&](int s) { return bars + 8u * (2 * ST_SP + 2 * ST_MAX_SLOTS + s); };
  auto empty_b = [&](int s) { return bars + 8u * (2 * ST_SP + 3 * ST_MAX_SLOTS + s); };
  const uint32_t acc_full = bars + 8u * (2 * ST_SP + 4 * ST_MAX_SLOTS);
  auto full_t = [&](int s) { return acc_full + 8u * (1 + s); };
  auto empty_t = [&](int s) { return acc_full + 8u * (1 + ST_SP + s); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + bar_off + 8 * ST_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_sx = reinterpret_cast<float*>(sm + bar_off + 8 * ST_BARS + 16);   // [T]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = (int)gridDim.x, rank = (int)blockIdx.x;   // the cluster spans blockIdx.x
  const int nt = (int)blockIdx.y % p.tiles_n, mt = (int)blockIdx.y / p.tiles_n;
  const int kb_total = p.K / 128;
  const int kb0 = rank * kb_total / S, kb1 = (rank + 1) * kb_total / S;
  const int w_col = has_tail ? 2 * T : T, cols = w_col + 32 * SI;   // accumulators, then the widened weights of the INT8 slots
  const uint32_t tmem_cols = cols <= 32 ? 32u : cols <= 64 ? 64u : cols <= 128 ? 128u : cols <= 256 ? 256u : 512u;

  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_b4)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_a8)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_tail)) : "memory");
    for (int s = 0; s < ST_SP; ++s) {
      mbar_init(full_p(s), 1);
      mbar_init(empty_p(s), 4);
    }
    for (int s = 0; s < SI; ++s) {
      mbar_init(full_i(s), PK ? 8 : 4 + 1);   // the widener warps of both operands, or those and the token producer
      mbar_init(empty_i(s), 1);
    }
    for (int s = 0; s < SB; ++s) {
      mbar_init(full_b(s), 2);       // the two producers
      mbar_init(empty_b(s), 1);
    }
    if (PK)
      for (int s = 0; s < ST_SP; ++s) {
        mbar_init(full_t(s), 1);
        mbar_init(empty_t(s), 4);
      }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!p.early) pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ packed weights -> staging
    if (lane == 0) {
      int sp = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(empty_p(sp), ph ^ 1u, abort_flag, 0x1000u)) break;
        mbar_arrive_expect_tx(full_p(sp), ST_STAGE);
        tma_load_2d(base + stage_off + sp * ST_STAGE, &tmap_b4, kb * 64, nt * 128, full_p(sp));
        if (++sp == ST_SP) {
          sp = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ bf16 weight rows
    if (lane == 0 && has_tail) {
      int s = 0;
      uint32_t ph = 1;   // parity of the release that a use waits for
      for (int k = kb0 * 2; k < kb1 * 2; k += HB) {
        if (!mbar_wait(empty_b(s), ph, abort_flag, 0x2000u)) break;
        mbar_arrive_expect_tx(full_b(s), (uint32_t)HB * 16384u);
        tma_load_3d(base + bf_off + s * bf_bytes, &tmap_w, 0, nt * 128, k, full_b(s));
        if (++s == SB) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (PK && warp == 3) {
    // ------------------------------------------------------------------ packed token codes -> staging
    if (lane == 0) {
      int sp = 0;
      uint32_t ph = 1;
      pdl_wait();
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(empty_t(sp), ph, abort_flag, 0x40000u)) break;
        mbar_arrive_expect_tx(full_t(sp), (uint32_t)T * 64u);
        tma_load_2d(base + tok_off + (uint32_t)(sp * T * 64), &tmap_a8, kb * 64, mt * T, full_t(sp));
        if (++sp == ST_SP) {
          sp = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ token codes and tail rows
    if (lane == 0) {
      const uint32_t tok = (uint32_t)T * 128u;
      const int m0 = mt * T;
      int si = 0, sb = 0;
      uint32_t phi = 1, phb = 1;
      bool ok = true;
      pdl_wait();   // the prologue's outputs; everything else is on its way already
      for (int k = kb0 * 128; k < kb1 * 128 && ok; k += 128) {
        if (!(ok = mbar_wait(empty_i(si), phi, abort_flag, 0x40000u))) break;
        mbar_arrive_expect_tx(full_i(si), tok);
        tma_load_2d(base + si * i8_bytes, &tmap_a8, k, m0, full_i(si));
        if (++si == SI) {
          si = 0;
          phi ^= 1u;
        }
        if (has_tail) {
          for (int h = 0; h < 2; h += HB) {
            if (!(ok = mbar_wait(empty_b(sb), phb, abort_flag, 0x80000u))) break;
            mbar_arrive_expect_tx(full_b(sb), (uint32_t)HB * tok);
            tma_load_3d(base + bf_off + sb * bf_bytes + (uint32_t)HB * 16384u, &tmap_tail, 0, m0, k / 64 + h, full_b(sb));
            if (++sb == SB) {
              sb = 0;
              phb ^= 1u;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the role that bounds tiles of few
    // rows: about 45 cycles per MMA up to T = 64, so its loop holds nothing but waits, MMAs and commits)
    if (elect_one()) {
      const uint32_t idesc_i8 = make_idesc_i8<0>() | ((uint32_t)(T >> 3) << 17);
      const uint32_t idesc_bf = make_idesc_bf16<0>() | ((uint32_t)(T >> 3) << 17);
      const uint64_t desc0 = make_smem_desc(base);            // address field: 16-byte units
      const uint64_t tok_rows = (uint64_t)(T * 128) >> 4;
      uint32_t phi = 0, phb = 0, acc = 0;
      uint32_t fi = full_i(0), fb = full_b(0);
      const uint32_t ta0 = tmem_base + (uint32_t)w_col;
      uint32_t ta = ta0;
      uint64_t di = desc0, db = desc0 + (bf_off >> 4);
      const uint32_t fi_end = full_i(SI), fb_end = full_b(SB);
      constexpr uint32_t TO_EMPTY = 8u * ST_MAX_SLOTS;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = mbar_wait(fi, phi, abort_flag, 0x4000u))) break;
        tc_fence_after();
        umma_i8_ta(tmem_base, ta, di, idesc_i8, acc);
        umma_i8_ta(tmem_base, ta + 8, di + 2, idesc_i8, 1u);   // 32 bytes of K further: + 8 columns, + 2
        umma_i8_ta(tmem_base, ta + 16, di + 4, idesc_i8, 1u);
        umma_i8_ta(tmem_base, ta + 24, di + 6, idesc_i8, 1u);
        umma_commit(fi + TO_EMPTY);
        fi += 8u;
        di += i8_bytes >> 4;
        ta += 32u;
        if (fi == fi_end) {
          fi = full_i(0);
          di = desc0;
          ta = ta0;
          phi ^= 1u;
        }
        if (has_tail) {
          uint32_t accf = acc;
#pragma unroll
          for (int h = 0; h < 2; h += HB) {
            if (!(ok = mbar_wait(fb, phb, abort_flag, 0x100000u))) break;
            tc_fence_after();
#pragma unroll
            for (int e = 0; e < HB; ++e) {
              const uint64_t ad = db + e * 1024, bd = db + HB * 1024 + e * tok_rows;
              umma_bf16(tmem_base + (uint32_t)T, ad, bd, idesc_bf, accf);
              accf = 1u;
              umma_bf16(tmem_base + (uint32_t)T, ad + 2, bd + 2, idesc_bf, 1u);
              umma_bf16(tmem_base + (uint32_t)T, ad + 4, bd + 4, idesc_bf, 1u);
              umma_bf16(tmem_base + (uint32_t)T, ad + 6, bd + 6, idesc_bf, 1u);
            }
            umma_commit(fb + TO_EMPTY);
            fb += 8u;
            db += bf_bytes >> 4;
            if (fb == fb_end) {
              fb = full_b(0);
              db = desc0 + (bf_off >> 4);
              phb ^= 1u;
            }
          }
          if (!ok) break;
        }
        acc = 1u;
      }
      if (ok) umma_commit(acc_full);
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ wideners: GROUPS groups of four warps for the
    // weights, then (ST_PACKED) as many for the token codes; group g takes the slices g, g + GROUPS, ...
    const int group = ((warp - 4) >> 2) % GROUPS;
    const bool tokens = PK && warp >= 4 + 4 * GROUPS;
    const int wtid = tid & 127;
    int sp = group, s = group;
    uint32_t php = 0, phu = 1;
    for (int kb = kb0 + group; kb < kb1; kb += GROUPS) {
      bool ok = mbar_wait(tokens ? full_t(sp) : full_p(sp), php, abort_flag, 0x8000u);
      ok = ok && mbar_wait(empty_i(s), phu, abort_flag, 0x10000u);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (tokens) {
        widen_rows(sm + tok_off + sp * T * 64, sm + s * i8_bytes, T, wtid);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      } else {
        tc_fence_after();
        widen_row_tmem(sm + stage_off + sp * ST_STAGE, tmem_base + (uint32_t)(w_col + 32 * s) + ((uint32_t)(wtid & 96) << 16), wtid);
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(full_i(s));
        mbar_arrive(tokens ? empty_t(sp) : empty_p(sp));
      }
      if ((sp += GROUPS) >= ST_SP) {
        sp -= ST_SP;
        php ^= 1u;
      }
      if ((s += GROUPS) >= SI) {
        s -= SI;
        phu ^= 1u;
      }
    }
    mbar_wait(acc_full, 0, abort_flag, 0x20000u);
    tc_fence_after();
  }
  __syncwarp();
  pdl_wait();      // (scales below; every thread, so that the kernel does not complete before its predecessor)
  pdl_trigger();
  // scales of the rows and of this thread's two channels (its column in the final loop), while the last MMAs run
  const int oc = (tid & 63) * 2, on = nt * 128 + oc;
  float2 sw = make_float2(0.0f, 0.0f), bias = make_float2(0.0f, 0.0f);
  if (on < p.N && p.sw) {
    sw = *reinterpret_cast<const float2*>(p.sw + on);
    if (p.bias) bias = *reinterpret_cast<const float2*>(p.bias + on);
  }
  if (warp < 4 && p.sx)
    for (int t = tid; t < T; t += 128) s_sx[t] = mt * T + t < p.M ? p.sx[mt * T + t] : 0.0f;
  cluster_sync_all();   // every CTA's MMAs are done: the rings are free

  // ---- accumulators -> shared memory of the CTA that finishes the row: [source][row / 4][channel][4 rows], int32 then
  // fp32 (128-bit stores of four rows of a channel: with one word per store the export took 1 us per 16 rows)
  const int TS = ((T + S - 1) / S + 3) & ~3;     // rows per CTA
  const uint32_t half = (uint32_t)(S * TS * 128) * 4u;
  if (warp >= 4 && warp < 8) {
    const int ch = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const int rows = min(T, p.M - mt * T);   // (rows beyond M are not exported)
    const uint32_t mine = base + (uint32_t)(rank * TS * 128 + ch * 4) * 4u;
    int owner = 0, left = TS;                // CTA that finishes the current rows, rows left in its share
    uint32_t off = 0, peer = map_to_cta(mine, 0u);
    for (int t0 = 0; t0 < rows; t0 += 16) {
      uint32_t ri[16], rf[16];
      tmem_ld16(lane_addr + (uint32_t)t0, ri);
      if (has_tail) tmem_ld16(lane_addr + (uint32_t)(T + t0), rf);
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        if (owner == rank) {
          st_shared_v4(mine + off, ri + i);
          if (has_tail) st_shared_v4(mine + off + half, rf + i);
        } else {
          st_cluster_v4(peer + off, ri + i);
          if (has_tail) st_cluster_v4(peer + off + half, rf + i);
        }
        off += 2048u;
        if ((left -= 4) == 0) {
          left = TS;
          off = 0;
          owner = min(owner + 1, S - 1);   // (past the last share only rows beyond T)
          peer = map_to_cta(mine, (uint32_t)owner);
        }
      }
    }
    tc_fence_before();
  }
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }

  // ---- rows [rank TS, (rank + 1) TS) of the tile: a thread takes two channels of four rows
  for (int i = tid; i < (TS / 4) * 64; i += st_threads(MODE)) {
    const int t = rank * TS + (i >> 6) * 4, row0 = mt * T + t;
    if (t >= T || row0 >= p.M || on >= p.N) continue;
    int a[2][4] = {};
    float f[2][4] = {};
    const unsigned char* src = sm + (size_t)((i >> 6) * 512 + oc * 4) * 4;
    for (int q = 0; q < S; ++q) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int4 v = *reinterpret_cast<const int4*>(src + (size_t)q * TS * 512 + e * 16);
        a[e][0] += v.x;
        a[e][1] += v.y;
        a[e][2] += v.z;
        a[e][3] += v.w;
        if (has_tail) {
          const float4 w = *reinterpret_cast<const float4*>(src + half + (size_t)q * TS * 512 + e * 16);
          f[e][0] = __fadd_rn(f[e][0], w.x);
          f[e][1] = __fadd_rn(f[e][1], w.y);
          f[e][2] = __fadd_rn(f[e][2], w.z);
          f[e][3] = __fadd_rn(f[e][3], w.w);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = row0 + r;
      if (row >= p.M) break;
      const size_t o = (size_t)row * p.N + on;
      const int a0 = a[0][r] >> (PK ? 8 : 4), a1 = a[1][r] >> (PK ? 8 : 4);   // (widened operands carry a factor 16)
      if (PK && p.C) {
        *reinterpret_cast<int2*>(p.C + o) = make_int2(a0, a1);
        continue;
      }
      const float sx = s_sx[t + r];
      float d0 = __fmul_rn(__fmul_rn((float)a0, sx), sw.x), d1 = __fmul_rn(__fmul_rn((float)a1, sx), sw.y);
      if (has_tail) {
        d0 = __fadd_rn(d0, f[0][r]);
        d1 = __fadd_rn(d1, f[1][r]);
      }
      if (PK && p.add) {
        const float2 f2 = *reinterpret_cast<const float2*>(p.add + o);
        d0 = __fadd_rn(d0, f2.x);
        d1 = __fadd_rn(d1, f2.y);
      }
      if (p.bias) {
        d0 = __fadd_rn(d0, bias.x);
        d1 = __fadd_rn(d1, bias.y);
      }
      if (p.act)
        p.out[o / 2] = (uint16_t)swiglu_bf16_bits(d0, d1);
      else
        *reinterpret_cast<uint32_t*>(p.out + o) = f32_to_bf16_bits(d0) | (f32_to_bf16_bits(d1) << 16);
      if (p.dbg_acc) *reinterpret_cast<int2*>(p.dbg_acc + o) = make_int2(a0, a1);
      if (p.dbg_tail) *reinterpret_cast<float2*>(p.dbg_tail + o) = make_float2(f[0][r], f[1][r]);
    }
  }
}

}  // namespace

// Clusters of S CTAs that can be resident at once: the SMs of a GPC that a cluster size does not divide stay empty (of
// 148 SMs, 48 clusters of three need two rounds).
static int stream_active_clusters(int S) {
  static int known[64][9] = {};
  int dev = 0;
  const int sms = current_device_sms(&dev);
  if (S <= 1) return sms;
  if (dev < 64 && known[dev][S]) return known[dev][S];
  int n = 0;
  if (cudaFuncSetAttribute(stream_gemm_kernel<2, ST_TAIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)S, 1024);
    cfg.blockDim = dim3(st_threads(ST_TAIL));
    cfg.dynamicSmemBytes = ST_SMEM;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, stream_gemm_kernel<2, ST_TAIL>, &cfg) != cudaSuccess) n = 0;
  }
  cudaGetLastError();
  if (n < 1) n = sms / S > 1 ? sms / S - 1 : 1;
  if (dev < 64) known[dev][S] = n;
  return n;
}

// Work split of a call and its estimated time.  The constants are a fit to timings at 16..4000 rows of N = 1024..28672,
// K = 4096..14336: a K slice of a tile of T rows takes 0.42 + 0.0023 T us with a tail and 0.17 + 0.0005 T without (MMA issue,
// operand loads and widening of one SM), a tile costs 2.4 + 0.042 T (2 + 0.012 T, and 0.042 for each row beyond 160) us
// around its main loop (launch, ring fill, accumulator exchange, output); packed tokens take 0.16 + 0.001 T a slice and 1.5 us
// more around it; and the weights cannot arrive faster than 5.2 TB/s.
struct StreamPlan {
  int T, tiles_m, tiles_n, S;
  float us;
};
static StreamPlan plan_stream(int M, int N, int K, int mode) {
  const bool tail = mode == ST_TAIL;
  StreamPlan best = {};
  best.us = 1e30f;
  const int tiles_n = (N + 127) / 128, kb = K / 128;
  const float hbm = (float)N * (float)K * (tail ? 2.5f : 0.5f) / 5.2e6f;
  const int tm0 = (M + st_max_t(mode) - 1) / st_max_t(mode);
  for (int tm = tm0; tm <= tm0 + 3; ++tm) {
    const int T = ((M + tm - 1) / tm + 15) / 16 * 16;
    const float slice = tail ? 0.42f + 0.0023f * T : mode == ST_PACKED ? 0.16f + 0.001f * T : 0.17f + 0.0005f * T;
    const float around = tail ? 2.4f + 0.042f * T
                              : (mode == ST_PACKED ? 3.5f : 2.0f) + 0.012f * T + (T > 160 ? 0.042f * (T - 160) : 0.0f);
    for (int S = 1; S <= 8 && S <= kb; ++S) {
      const int tiles = tm * tiles_n, fit = stream_active_clusters(S), waves = (tiles + fit - 1) / fit;
      const float one = (float)((kb + S - 1) / S) * slice + around + (S > 1 ? 0.8f : 0.0f);
      float us = waves * one;
      if (us < hbm + waves * around) us = hbm + waves * around;
      if (mode == ST_PACKED ? waves > 2 : waves > 1) us *= mode == ST_PACKED ? 1.05f : 1.1f;
      if (us < best.us) {
        best.T = T;
        best.tiles_m = tm;
        best.tiles_n = tiles_n;
        best.S = S;
        best.us = us;
      }
    }
  }
  return best;
}

template <int HB, int MODE>
static int launch_stream(const StreamPlan& pl, const StreamParams& p, const CUtensorMap& mb, const CUtensorMap& mw,
                         const CUtensorMap& ma, const CUtensorMap& mt, cudaStream_t st) {
  auto kern = stream_gemm_kernel<HB, MODE>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(dev < 64 && configured[dev])) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return TQ_ERR_CUDA;
    }
    if (dev < 64) configured[dev] = true;
  }
  return launch_pdl(kern, dim3(pl.S, pl.tiles_n * pl.tiles_m), dim3(st_threads(MODE)), (size_t)ST_SMEM, st, pl.S,
                    mb, mw, ma, mt, p);
}

// `early`: the kernel in front in the stream is the prologue of this call
int run_stream_gemm(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col, const float* w_scale,
                    const void* w_rot, const void* tail_dense, int R, const float* bias, void* out_bf16,
                    int32_t* dbg_acc, float* dbg_tail, int M, int N, int K, int act, bool early, cudaStream_t st) {
  const StreamPlan pl = plan_stream(M, N, K, R > 0 ? ST_TAIL : ST_INT8);
  StreamParams p = {};
  p.M = M;
  p.N = N;
  p.K = K;
  p.T = pl.T;
  p.act = act;
  p.tiles_n = pl.tiles_n;
  p.early = early ? 1 : 0;
  p.sx = body_scale;
  p.sw = w_scale;
  p.bias = bias;
  p.out = reinterpret_cast<uint16_t*>(out_bf16);
  p.dbg_acc = dbg_acc;
  p.dbg_tail = dbg_tail;
  // What fits beside the staging buffers.  With a tail: bf16 slots beside two INT8 slots (of tokens: the widened weights are
  // in tensor memory), two or more of a whole slice up to 160 rows (half the load instructions and waits), three of half a
  // slice beyond; what is left goes to INT8 slots.
  const int slot = (128 + pl.T) * 128;
  const int room = ST_SMEM - (st_sp(R > 0 ? ST_TAIL : ST_INT8) * ST_STAGE + 8 * ST_BARS + 16 + 4 * ST_MAX_T + 1024);
  int hb = 1;
  if (R > 0) {
    const int units = (room - 2 * pl.T * 128) / slot;   // 3 at T = 176, 10 at T = 16
    hb = units >= 4 ? 2 : 1;
    p.sb = units / hb < ST_MAX_SLOTS ? units / hb : ST_MAX_SLOTS;
    p.si = (room - p.sb * hb * slot) / (pl.T * 128);
    if (p.si > 4) p.si = 4;
  } else {
    const int units = room / (pl.T * 128);
    p.si = units < ST_MAX_SLOTS ? units & ~1 : ST_MAX_SLOTS;
    p.sb = 0;
  }
  CUtensorMap mb, mw, ma, mt;
  if (!make_tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, b_col, (uint64_t)(K / 2), (uint64_t)N, (uint64_t)(K / 2),
                          64, 128, 64) ||
      !make_tensor_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_q8, (uint64_t)K, (uint64_t)M, (uint64_t)K, 128, pl.T,
                          true))
    return TQ_ERR_CUDA;
  if (R > 0) {
    if (!make_tensor_map_kblocks(&mw, w_rot, (uint64_t)K, (uint64_t)N, 128, hb) ||
        !make_tensor_map_kblocks(&mt, tail_dense, (uint64_t)K, (uint64_t)M, pl.T, hb))
      return TQ_ERR_CUDA;
  } else {
    mw = mb;   // never read
    mt = ma;
  }
  if (R == 0) return launch_stream<1, ST_INT8>(pl, p, mb, mw, ma, mt, st);
  return hb == 2 ? launch_stream<2, ST_TAIL>(pl, p, mb, mw, ma, mt, st) : launch_stream<1, ST_TAIL>(pl, p, mb, mw, ma, mt, st);
}

// Packed activations and no tail operand: the int32 product into C, or (C == NULL) the dequantised bf16 result with the
// optional tail sums `add`.
int run_stream_packed(const uint8_t* a_pack, const uint8_t* b_col, int32_t* C, const float* body_scale, const float* w_scale,
                      const float* add, const float* bias, void* out_bf16, int M, int N, int K, cudaStream_t st) {
  const StreamPlan pl = plan_stream(M, N, K, ST_PACKED);
  StreamParams p = {};
  p.M = M;
  p.N = N;
  p.K = K;
  p.T = pl.T;
  p.tiles_n = pl.tiles_n;
  p.sx = body_scale;
  p.sw = w_scale;
  p.bias = bias;
  p.add = add;
  p.C = C;
  p.out = reinterpret_cast<uint16_t*>(out_bf16);
  const int fixed = st_sp(ST_PACKED) * (ST_STAGE + pl.T * 64) + 8 * ST_BARS + 16 + 4 * ST_MAX_T + 1024;
  const int units = (ST_SMEM - fixed) / (pl.T * 128);   // 6 at T = 176
  p.si = units < ST_MAX_SLOTS ? units & ~1 : ST_MAX_SLOTS;
  CUtensorMap mb, ma;
  if (!make_tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, b_col, (uint64_t)(K / 2), (uint64_t)N, (uint64_t)(K / 2),
                          64, 128, 64) ||
      !make_tensor_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_pack, (uint64_t)(K / 2), (uint64_t)M, (uint64_t)(K / 2),
                          64, pl.T))
    return TQ_ERR_CUDA;
  return launch_stream<1, ST_PACKED>(pl, p, mb, mb, ma, ma, st);
}

}  // namespace tq
