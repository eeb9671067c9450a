// The whole linear behind the prologue for few token rows (M <= 64), ONE launch up to eight rows: INT4 x INT4 dense part,
// exact-order tail correction, dequantisation, bias / SwiGLU, bf16 out.  Beyond that, and on wide layers before, the tail
// sums come from tail_small_kernel (see run_decode_linear).
//
// What bounds it: at one row the latency of a few dependent memory round trips, from a few rows on the weight bytes
// (N K / 2 packed + the bf16 rows that the tails name).  A CTA owns 16 CT output channels and its eight WARPS are the
// eight K ranges and the eight tail chains, so everything between the prologue's lists and the bf16 results stays in
// one CTA and no warp waits for another before the final sum:
//   * warp w streams K range w of the packed weights through a ring of its own (TMA blocks of 256 K, at most 8 KB a warp;
//     the first ones are requested before the wait for the prologue, whose programmatic dependent this kernel is) and
//     multiplies with mma.sync m16n8k32 s8, both operands widened with the same nibble order;
//   * the tail sum of an output is eight interleaved fp32 fma chains (entry r on chain r mod 8), combined as
//     ((c0+c1)+(c2+c3))+((c4+c5)+(c6+c7)): warp w evaluates chain w.  The weight-row pieces of its entries arrive by
//     cp.async in buffers of the warp's own, two or three of 2 KB, so a chain costs a memory latency per buffer
//     instead of one per batch of registers;
//   * the partials meet in shared memory once, at the end.
// A cluster of eight CTAs per 64 channels (ranges = CTAs, partials over distributed shared memory) was measured first:
// as fast at N = 4096, but 27 us against 12 for the average projection at N = 24576, where thousands of small CTAs
// each pay start-up, list and cluster barriers.
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace tq {
namespace {

constexpr int DL_WARPS = 8;     // K ranges = interleaved fp32 chains of a tail sum
constexpr int DL_THREADS = 32 * DL_WARPS;
constexpr int DL_PIECES = 2048; // bytes of a warp's buffer of weight-row pieces (two or three buffers)
constexpr int DL_BLOCK = 256;   // K elements of a weight block (one 128-byte swizzled row per channel)

struct DecodeLinearParams {
  const uint8_t* a_pack;    // [M, K/2]
  const float* sx;          // [M]
  const uint16_t* idx;      // [M, ld]
  const uint16_t* val;      // [M, ld]
  const uint8_t* b_col;     // [N, K/2]
  const uint16_t* w_t;      // [K, N] bf16
  const float* sw;          // [N]
  const float* bias;        // [N] or NULL
  const float* tail;        // [M, N] tail sums computed elsewhere, or NULL (R = 0 then)
  uint16_t* out;            // [M, N], or [M, N/2] with act
  int M, N, K, R, ld, act;
  int nst;                  // stages of a warp's ring of weight blocks
  int early;                // the weights may be read before the kernel in front has ended
};

// NT: tiles of eight token rows (M <= 8 NT).  CT: tiles of 16 output channels per CTA step.  The weights are the m16
// operand of the MMA and the tokens the n8 operand: with at most eight rows half as many MMAs as the other way round.
// VC: channels per lane in the tail sums.
template <int CT>
struct DecodeSmem {
  static constexpr int CH = 16 * CT;
  static constexpr int STAGE = CH * 128;              // weight block: [CH channels][128 bytes], 128-byte swizzle
  static constexpr int MAX_ST = 8192 / STAGE;         // stages of a warp's ring: at most 8 KB
  // [8][nst] weight blocks | [8][nbuf] piece buffers | [8][MAX_ST] mbarriers, abort flag | int32 partials [8][M][CH] |
  // chain sums [8][M][CH] | tail entries [8][M][nr] (index | value bits << 16)
  int nst, nbuf, pieces, bars, part, chain, list, total;
  __host__ __device__ static int nr_max(int R) { return (R + DL_WARPS - 1) / DL_WARPS; }
  __host__ __device__ DecodeSmem(int M, int R, int nst_) {
    nst = nst_;
    nbuf = R == 0 ? 0 : (M * nr_max(R) * CH * 2 <= DL_PIECES ? 2 : 3);
    pieces = DL_WARPS * nst * STAGE;
    bars = pieces + DL_WARPS * nbuf * DL_PIECES;
    part = bars + DL_WARPS * MAX_ST * 8 + 16;
    chain = part + DL_WARPS * M * CH * 4;
    list = chain + (R > 0 ? DL_WARPS * M * CH * 4 : 0);
    total = list + DL_WARPS * M * nr_max(R) * 4 + 1024;   // + alignment slack
  }
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int NT, int CT, int VC>
__global__ void __launch_bounds__(DL_THREADS, 2)
decode_linear_kernel(const __grid_constant__ CUtensorMap tmap_b, const DecodeLinearParams p) {
  using S = DecodeSmem<CT>;
  constexpr int CH = S::CH;
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* sm = smem_dyn + (base - raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const int M = p.M, N = p.N, K = p.K, R = p.R;
  const S L(M, R, p.nst);
  unsigned char* ring = sm + warp * L.nst * S::STAGE;
  const uint32_t ring_s = base + (uint32_t)(warp * L.nst * S::STAGE);
  const unsigned char* piece = sm + L.pieces + warp * L.nbuf * DL_PIECES;
  const uint32_t piece_s = base + (uint32_t)(L.pieces + warp * L.nbuf * DL_PIECES);
  const uint32_t bars = base + (uint32_t)(L.bars + warp * S::MAX_ST * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L.bars + DL_WARPS * S::MAX_ST * 8);
  int32_t* s_int = reinterpret_cast<int32_t*>(sm + L.part);
  float* s_chain = reinterpret_cast<float*>(sm + L.chain);
  const int nrm = S::nr_max(R);
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + L.list) + warp * M * nrm;   // this warp's chain: [M][nr]
  const int tiles = (N + CH - 1) / CH;

  // ---- the weight stream first: it depends on nothing that the prologue writes.  A warp owns the K blocks [k0, k1) and
  // fills its own ring, one tiled TMA load per (channel tile, block), running ahead across the end of a channel tile.
  const int blocks = (K + DL_BLOCK - 1) / DL_BLOCK;
  const int k0 = warp * blocks / DL_WARPS, k1 = (warp + 1) * blocks / DL_WARPS;
  if (tid == 0) *abort_flag = 0;
  if (lane == 0) {
    for (int s = 0; s < L.nst; ++s) mbar_init(bars + 8u * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  int q_tile = blockIdx.x, q_k = k0, q_s = 0;   // next block to request, its stage (lane 0)
  auto request = [&]() {
    if (q_tile < tiles && k0 < k1) {
      mbar_arrive_expect_tx(bars + 8u * q_s, S::STAGE);
      tma_load_2d(ring_s + (uint32_t)(q_s * S::STAGE), &tmap_b, q_k * (DL_BLOCK / 2), q_tile * CH, bars + 8u * q_s);
      if (++q_s == L.nst) q_s = 0;
      if (++q_k == k1) {
        q_k = k0;
        q_tile += gridDim.x;
      }
    }
  };
  if (!p.early) pdl_wait();
  if (lane == 0)
    for (int s = 0; s < L.nst; ++s) request();

  pdl_wait();      // the prologue's outputs are visible from here on
  pdl_trigger();
  __syncthreads();   // (the abort flag)

  // ---- tail entries of chain `warp`: r = warp + 8 i, i < nr, of every row
  const int nr = R > warp ? (R - warp + DL_WARPS - 1) / DL_WARPS : 0;
  for (int m = 0; m < M; ++m)
    for (int i = lane; i < nr; i += 32) {
      const size_t o = (size_t)m * p.ld + warp + DL_WARPS * i;
      list[m * nrm + i] = (uint32_t)p.idx[o] | ((uint32_t)p.val[o] << 16);
    }
  __syncwarp();
  // A chunk of pieces: entries [i0, i0 + ic) of the RPW rows of a row group.  All chunks of a channel tile (row groups,
  // then entries) and then those of the next one go through the warp's piece buffers, nbuf - 1 chunks ahead of the sums.
  constexpr int LPR = CH / VC, RPW = 32 / LPR;    // lanes per row, rows side by side
  constexpr int PPE = 2 * CT;                     // 16-byte pieces per entry
  const int rows = min(RPW, M);
  const int ic = DL_PIECES / (CH * 2) / rows;
  int t_tile = blockIdx.x, t_m = 0, t_i = 0, t_b = 0;   // next chunk to request
  auto request_pieces = [&]() {
    if (t_tile < tiles && nr > 0) {
      const uint32_t dst = piece_s + (uint32_t)(t_b * DL_PIECES);
      const int cnt = min(ic, nr - t_i), n = t_tile * CH + (lane % PPE) * 8;
      if (n < N) {
        const uint16_t* wt = p.w_t + n;
        for (int r = 0; r < rows && t_m + r < M; ++r) {
          const uint32_t* lst = list + (t_m + r) * nrm + t_i;
          for (int i = lane / PPE; i < cnt; i += 32 / PPE)
            cp_async16(dst + (uint32_t)((r * ic + i) * (CH * 2) + (lane % PPE) * 16), wt + (size_t)(lst[i] & 0xffffu) * N);
        }
      }
      if (++t_b == L.nbuf) t_b = 0;
      if ((t_i += ic) >= nr) {
        t_i = 0;
        if ((t_m += RPW) >= M) {
          t_m = 0;
          t_tile += gridDim.x;
        }
      }
    }
    cp_async_commit();
  };
  if (R > 0)
    for (int b = 0; b < L.nbuf; ++b) request_pieces();

  const uint8_t* abase = p.a_pack + (size_t)g * (K / 2) + j * 32;
  int c_s = 0, c_b = 0;
  uint32_t c_par = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    // ---- dense part over this warp's K blocks
    int acc[NT][CT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int b = 0; b < CT; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][b][i] = 0;
    for (int k = k0; k < k1; ++k) {
      uint4 av[NT][2];
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
          av[t][sl] = make_uint4(0u, 0u, 0u, 0u);
          if (8 * t + g < M && k * DL_BLOCK + j * 64 + sl * 32 < K)
            av[t][sl] = *reinterpret_cast<const uint4*>(abase + (size_t)(8 * t) * (K / 2) + (size_t)k * (DL_BLOCK / 2) + sl * 16);
        }
      mbar_wait(bars + 8u * c_s, c_par, abort_flag, 0x800000u);
      const unsigned char* st = ring + c_s * S::STAGE + g * 128;
#pragma unroll
      for (int sl = 0; sl < 2; ++sl) {
        // a lane's 32 codes: 16-byte chunk 2 j + sl of the channel's row (chunk index XOR row & 7: conflict-free)
        const uint32_t ch = (uint32_t)(((2 * j + sl) ^ g) << 4);
        uint32_t lo[CT][8], hi[CT][8];
#pragma unroll
        for (int b = 0; b < CT; ++b) {
          widen16(*reinterpret_cast<const uint4*>(st + b * 2048 + ch), lo[b]);
          widen16(*reinterpret_cast<const uint4*>(st + b * 2048 + 1024 + ch), hi[b]);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          uint32_t a[8];
          widen16(av[t][sl], a);
#pragma unroll
          for (int b = 0; b < CT; ++b)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              mma_s8(acc[t][b], lo[b][2 * q], hi[b][2 * q], lo[b][2 * q + 1], hi[b][2 * q + 1], a[2 * q], a[2 * q + 1]);
        }
      }
      __syncwarp();
      if (lane == 0) request();   // the stage is free again
      if (++c_s == L.nst) {
        c_s = 0;
        c_par ^= 1u;
      }
    }
    // accumulator fragment: channels g and g + 8 of the tile, rows 2 j and 2 j + 1 of the eight; both operands carried a
    // factor 16
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = 8 * t + 2 * j + (i & 1);
        if (m < M) {
#pragma unroll
          for (int b = 0; b < CT; ++b) s_int[(warp * M + m) * CH + b * 16 + g + 8 * (i >> 1)] = acc[t][b][i] >> 8;
        }
      }

    // ---- chain `warp` of every row: a lane owns VC channels of one row of the group
    if (R > 0) {
      const int c0 = (lane % LPR) * VC, r = lane / LPR;
      for (int m = r; m - r < M; m += RPW) {
        float v[VC];
#pragma unroll
        for (int i = 0; i < VC; ++i) v[i] = 0.0f;
        for (int i0 = 0; i0 < nr; i0 += ic) {
          if (L.nbuf == 2)
            cp_async_wait<1>();   // (one group per request, empty ones included)
          else
            cp_async_wait<2>();
          __syncwarp();
          if (m < M) {
            const uint32_t* lst = list + m * nrm + i0;
            const unsigned char* src = piece + c_b * DL_PIECES + r * ic * (CH * 2) + c0 * 2;
            const int cnt = min(ic, nr - i0);
#pragma unroll 4
            for (int i = 0; i < cnt; ++i) {
              const float x = __uint_as_float(lst[i] & 0xffff0000u);
              uint32_t ww[VC / 2];
#pragma unroll
              for (int q = 0; q < VC / 2; ++q) ww[q] = reinterpret_cast<const uint32_t*>(src + i * (CH * 2))[q];
#pragma unroll
              for (int q = 0; q < VC / 2; ++q) {
                v[2 * q] = fmaf(x, __uint_as_float(ww[q] << 16), v[2 * q]);
                v[2 * q + 1] = fmaf(x, __uint_as_float(ww[q] & 0xffff0000u), v[2 * q + 1]);
              }
            }
          }
          __syncwarp();
          if (++c_b == L.nbuf) c_b = 0;
          request_pieces();
        }
        if (m < M) {
#pragma unroll
          for (int i = 0; i < VC; ++i) s_chain[(warp * M + m) * CH + c0 + i] = v[i];
        }
      }
    }
    __syncthreads();

    // ---- the ranges and chains of every output meet (a warp's lanes hold neighbouring channels)
    const int n_base = tile * CH;
    for (int t0 = 0; t0 < M * CH; t0 += DL_THREADS) {
      const int t = t0 + tid;
      const int m = t / CH, c = t % CH, no = n_base + c;
      const bool on = t < M * CH && no < N;
      float d = 0.0f;
      if (on) {
        int sum = 0;
#pragma unroll
        for (int q = 0; q < DL_WARPS; ++q) sum += s_int[q * M * CH + t];
        d = __fmul_rn(__fmul_rn((float)sum, p.sx[m]), p.sw[no]);
        if (R > 0) {
          float ch[DL_WARPS];
#pragma unroll
          for (int q = 0; q < DL_WARPS; ++q) ch[q] = s_chain[q * M * CH + t];
          d = __fadd_rn(d, __fadd_rn(__fadd_rn(__fadd_rn(ch[0], ch[1]), __fadd_rn(ch[2], ch[3])),
                                     __fadd_rn(__fadd_rn(ch[4], ch[5]), __fadd_rn(ch[6], ch[7]))));
        }
        if (p.tail) d = __fadd_rn(d, p.tail[(size_t)m * N + no]);
        if (p.bias) d = __fadd_rn(d, p.bias[no]);
      }
      if (p.act) {
        const float u = __shfl_xor_sync(0xffffffffu, d, 1);
        if (on && !(c & 1)) p.out[((size_t)m * N + no) / 2] = (uint16_t)swiglu_bf16_bits(d, u);
      } else if (on) {
        p.out[(size_t)m * N + no] = (uint16_t)f32_to_bf16_bits(d);
      }
    }
    if (tile + (int)gridDim.x < tiles) __syncthreads();   // the next tile overwrites the partials
  }
}

template <int NT, int CT, int VC>
int launch_decode_linear(DecodeLinearParams p, cudaStream_t st) {
  using S = DecodeSmem<CT>;
  auto kern = decode_linear_kernel<NT, CT, VC>;
  static bool configured[64] = {};
  int dev = 0;
  const int sms = current_device_sms(&dev);
  if (!(dev < 64 && configured[dev])) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return TQ_ERR_CUDA;
    }
    if (dev < 64) configured[dev] = true;
  }
  // the ring takes what two CTAs per SM leave of the shared memory, two stages at least
  p.nst = S::MAX_ST;
  while (p.nst > 2 && S(p.M, p.R, p.nst).total > 112 * 1024) --p.nst;
  const int smem = S(p.M, p.R, p.nst).total;
  if (smem > 226 * 1024) return TQ_ERR_UNSUPPORTED;
  CUtensorMap mb;
  if (!make_tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.b_col, (uint64_t)(p.K / 2), (uint64_t)p.N,
                          (uint64_t)(p.K / 2), 128, 16 * CT, true))
    return TQ_ERR_CUDA;
  const int tiles = (p.N + 16 * CT - 1) / (16 * CT), cap = 2 * sms;
  return launch_pdl(kern, dim3(tiles < cap ? tiles : cap), dim3(DL_THREADS), (size_t)smem, st, 1, mb, p);
}

int run_decode_linear_rows(const DecodeLinearParams& p, cudaStream_t st) {
#define TQ_DL(NT_, CT_, VC_) return launch_decode_linear<NT_, CT_, VC_>(p, st)
  // 32 channels per CTA step at one row (half as many list passes; at N = 24576 21.7 us against 26.7), 16 beyond: twice
  // the CTAs, which is what hides the latency of the tail rows (N = K = 4096 at 4 rows: 14.6 us against 15.8)
  if (p.M == 1) TQ_DL(1, 2, 2);
  if (p.M <= 4) TQ_DL(1, 1, 2);
  if (p.M <= 8) TQ_DL(1, 1, 4);
  if (p.M <= 16) TQ_DL(2, 1, 8);
  if (p.M <= 32) TQ_DL(4, 1, 8);
  TQ_DL(8, 1, 8);
#undef TQ_DL
}

int run_decode_linear(DecodeLinearParams p, float* tail_scratch, cudaStream_t st) {
  if (p.M > 64 || p.K % 128 != 0 || p.N % 8 != 0) return TQ_ERR_UNSUPPORTED;
  // Beyond eight rows the tail sums come from their own kernel, up to eight where the caller brings the scratch: a CTA's 16
  // or 32 channels make 32- or 64-byte pieces of the weight rows, and with many rows or channels the pieces, not the
  // latency, are what takes time (512 bytes each there; N = 24576, R = 205: 64 us in this kernel at 8 rows, 36 in two; at
  // one row 19 and 25.  `SplitLinear._tail_apart` draws the line; that kernel takes 8192 entries).
  if (p.R > 0 && (p.M > 8 || (tail_scratch && p.R <= 8192))) {
    if (!tail_scratch) return TQ_ERR_BAD_ARG;
    const int rc = tq_tail_gather_small(p.idx, p.val, p.w_t, tail_scratch, p.M, p.N, p.K, p.R, p.ld, st);
    if (rc != TQ_OK) return rc;
    p.tail = tail_scratch;
    p.R = 0;
  }
  // rows per launch: all of them, unless the entry lists (4 bytes per entry) outgrow shared memory
  int rows = p.M;
  while (rows > 1 && (long)rows * p.R * 4 > 96 * 1024) rows = (rows + 1) / 2;
  const int total = p.M;
  for (int m = 0; m < total; m += rows) {
    p.M = total - m < rows ? total - m : rows;
    const int rc = run_decode_linear_rows(p, st);
    if (rc != TQ_OK) return rc;
    p.a_pack += (size_t)p.M * (p.K / 2);
    p.sx += p.M;
    if (p.R > 0) {
      p.idx += (size_t)p.M * p.ld;
      p.val += (size_t)p.M * p.ld;
    }
    if (p.tail) p.tail += (size_t)p.M * p.N;
    p.out += (size_t)p.M * (p.act ? p.N / 2 : p.N);
  }
  return TQ_OK;
}

}  // namespace
}  // namespace tq
