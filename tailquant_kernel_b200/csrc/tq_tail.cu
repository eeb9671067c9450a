// Sparse tail correction, tail mode T16 (sm_100a):
//   tail[m,n] = sum_r  x_tail[m,r] * W_t[idx[m,r], n]        (W_t = rotated weight, [K,N] bf16)
// as one fp32 fma chain per output in ascending index order.
//
// The rotation scatters the tail positions uniformly over K, so rows share nothing: the work is
// M*R*N multiply-adds that each need one bf16 weight.  A CTA owns a unit of up to 128 rows x 64
// columns and streams the 64-column strip of W_t through shared memory in 512-row chunks (plain
// 2-D TMA loads, three slots: two chunks resident, the third on its way, also across units).
// Eight lanes own a row: they read a gathered weight row segment (8 x 16 B = 128 contiguous bytes:
// bank-conflict free) and carry 8 accumulators each.  Index lists are ascending, so the entries
// of a row that fall into a chunk are a contiguous run: every quarter warp walks its cursor
// through the window of two chunks, which evens out the different run lengths of the rows
// sharing a warp.  What bounds it is the instructions per entry (widening and summing 8 columns,
// the weight read, shared memory at 512 bytes per warp and entry): so the lanes fetch eight
// entries of their row at a time, 32 ahead, and pass address and value through shared memory, the
// eight reads of a batch have no branch between them, and two columns share a multiply-add.
// One row per quarter and up to 32 warps leave fewer SMs idle at few rows than four rows per
// quarter and 16 warps.  N = K = 4096, R = 205, cold caches, before -> now: M = 16: 85 -> 26 us,
// 200: 119 -> 41, 512: 127 -> 84; M = 200, K = 14336, R = 717: 444 -> 135.
//
// Reference behaviour covered (for the bf16-tail mode): `sparse_top_add_rowmajor_quad_shared`
// (call site tools/bench_hadamard_three_schemes_quarot_dense_sharedqkv_inplace_fusedtopr_v43.py:287-295)
// and tools/sparse_correction_add_ext_v1.py:64-123.
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace tq {
namespace {

constexpr int T_ROWS = 128;                   // rows per unit: one per quarter warp
constexpr int T_COLS = 64;                    // columns per unit (128 bytes of bf16)
constexpr int T_KC = 512;                     // weight rows per chunk
constexpr int T_BUF = T_KC * T_COLS * 2;      // 64 KB per ring slot
constexpr int T_SLOTS = 3;
constexpr int T_PASS = 8 * T_ROWS * 8;         // one (address, value) pair per thread
constexpr int T_SMEM = T_SLOTS * T_BUF + 64 + T_PASS + 1024;
constexpr int T_SENT = 0x7fffffff;

struct TailParams {
  const uint16_t* idx;
  const uint16_t* val;
  float* out;
  int M, N, K, R, ld;
  int units_m, units_n, rows;  // rows per unit (<= T_ROWS, a multiple of 4): one per eight threads
};

// acc (two columns) += x * w for the two bf16 of a word, each an fp32 fma
__device__ __forceinline__ void fma_bf16x2(uint64_t& acc, uint64_t xx, uint32_t w) {
  uint64_t ww;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ww) : "r"(w << 16), "r"(w & 0xffff0000u));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(xx), "l"(ww));
}

__global__ void __launch_bounds__(8 * T_ROWS, 1)
tail_kernel(const __grid_constant__ CUtensorMap tmap_w, const TailParams p) {
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* sm = smem_dyn + (base - raw);
  const uint32_t bar0 = base + T_SLOTS * T_BUF;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + T_SLOTS * T_BUF + 32);

  uint2* pass = reinterpret_cast<uint2*>(sm + T_SLOTS * T_BUF + 64);

  const int tid = threadIdx.x;
  const int l8 = tid & 7, qw = tid >> 3;
  const unsigned char* sm_l8 = sm + l8 * 16;
  const int nch = (p.K + T_KC - 1) / T_KC;
  const int total_units = p.units_m * p.units_n;
  const int my_units = ((int)blockIdx.x < total_units) ? (total_units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_w)) : "memory");
    for (int i = 0; i < T_SLOTS; ++i) mbar_init(bar0 + 8 * i, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  // thread 0 only: the next chunk of this CTA's units (running over all of them) into the next slot of the ring
  int iu = 0, ic = 0, islot = 0;
  auto issue = [&]() {
    if (iu >= my_units) return;
    const int n0 = (((int)blockIdx.x + iu * (int)gridDim.x) % p.units_n) * T_COLS;
    const uint32_t bar = bar0 + 8u * islot, dst = base + (uint32_t)islot * T_BUF;
    mbar_arrive_expect_tx(bar, T_BUF);
    tma_load_2d(dst, &tmap_w, n0, ic * T_KC, bar);
    tma_load_2d(dst + T_BUF / 2, &tmap_w, n0, ic * T_KC + T_KC / 2, bar);
    islot = islot == T_SLOTS - 1 ? 0 : islot + 1;
    if (++ic == nch) ic = 0, ++iu;
  };
  if (tid == 0)
    for (int i = 0; i < T_SLOTS; ++i) issue();

  int slot = 0;           // ring slot and parity of the chunk being worked through
  uint32_t par = 0;
  bool ok = true;
  for (int iu_ = 0; iu_ < my_units; ++iu_) {
    const int u = (int)blockIdx.x + iu_ * (int)gridDim.x;
    const int n0 = (u % p.units_n) * T_COLS;  // neighbouring CTAs share the rows' index lists
    const int row = (u / p.units_n) * p.rows + qw;
    const bool live = row < p.M;
    const uint16_t* irow = p.idx + (size_t)row * p.ld;
    const uint16_t* vrow = p.val + (size_t)row * p.ld;
    auto fetch = [&](int i) {  // entry i as index | value bits << 16
      return live && i < p.R ? (uint32_t)__ldg(irow + i) | ((uint32_t)__ldg(vrow + i) << 16) : 0u;
    };
    uint64_t acc[4] = {0, 0, 0, 0};
    // entries i0 .. i0 + 7 of the row, one per lane of the quarter warp; `done` of the eight are summed.  32 entries are in
    // registers and the next 32 on their way (moving a register waits for its load: once in four batches is rare enough)
    uint32_t cur[4], nxt[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) cur[j] = fetch(8 * j + l8), nxt[j] = fetch(32 + 8 * j + l8);
    int i0 = 0, done = 0;
    auto add = [&](uint32_t at, uint32_t x) {
      const uint4 w = *reinterpret_cast<const uint4*>(sm_l8 + at);
      uint64_t xx;
      asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "r"(x));
      fma_bf16x2(acc[0], xx, w.x);
      fma_bf16x2(acc[1], xx, w.y);
      fma_bf16x2(acc[2], xx, w.z);
      fma_bf16x2(acc[3], xx, w.w);
    };
    ok = ok && mbar_wait(bar0 + 8u * slot, par, abort_flag, 0x100u);

    for (int c = 0; c < nch; ++c) {
      const int nslot = slot == T_SLOTS - 1 ? 0 : slot + 1;
      const uint32_t npar = nslot ? par : par ^ 1u;
      if (c + 1 < nch) ok = ok && mbar_wait(bar0 + 8u * nslot, npar, abort_flag, 0x200u);
      if (ok) {
        const int chunk_end = (c + 1) * T_KC;  // entries below this must be done in this phase
        const int win_end = (c + 2) * T_KC;    // entries below this have their weights resident
        while (true) {
          const uint32_t lo = i0 & 8 ? cur[1] : cur[0], hi = i0 & 8 ? cur[3] : cur[2];
          const uint32_t batch = i0 & 16 ? hi : lo;
          const int k = live && i0 + l8 < p.R ? (int)(batch & 0xffffu) : T_SENT;
          if (!__any_sync(0xffffffffu, k < chunk_end && l8 >= done)) break;
          const uint32_t in_win = (__ballot_sync(0xffffffffu, k < win_end) >> (tid & 24)) & 0xffu;
          pass[tid] = make_uint2((uint32_t)(k < chunk_end ? slot : nslot) * T_BUF + (((uint32_t)k * (T_COLS * 2)) & (T_BUF - 1)),
                                 batch & 0xffff0000u);
          __syncwarp();
          const uint2* mine = pass + (tid & ~7);
          if (in_win == 0xffu && done == 0) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              const uint4 e2 = *reinterpret_cast<const uint4*>(mine + j);
              add(e2.x, e2.y);
              add(e2.z, e2.w);
            }
            done = 8;
          } else {
            // the last entries of a row, and batches that reach beyond the window
            const int end = __popc(in_win);
            for (; done < end; ++done) add(mine[done].x, mine[done].y);
          }
          if (done == 8) {
            i0 += 8;
            done = 0;
            if ((i0 & 31) == 0) {
#pragma unroll
              for (int j = 0; j < 4; ++j) cur[j] = nxt[j], nxt[j] = fetch(i0 + 32 + 8 * j + l8);
            }
          }
          __syncwarp();
        }
      }
      ok = __syncthreads_and(ok) != 0;  // every thread is past chunk c: its ring slot may be refilled
      if (!ok) return;
      if (tid == 0) issue();
      slot = nslot;
      par = npar;
    }

    const int n = n0 + l8 * 8;
    if (live && n < p.N) {
      ulonglong2* o = reinterpret_cast<ulonglong2*>(p.out + (size_t)row * p.N + n);
      o[0] = make_ulonglong2(acc[0], acc[1]);
      o[1] = make_ulonglong2(acc[2], acc[3]);
    }
  }
}

}  // namespace
}  // namespace tq

extern "C" int tq_tail_gather(const uint16_t* tail_idx16, const void* tail_val, const void* w_t, float* tail,
                              int M, int N, int K, int R, int tail_ld, void* stream) {
  using namespace tq;
  if (!tail_idx16 || !tail_val || !w_t || !tail || M < 0 || N <= 0 || K <= 0 || R <= 0 || R >= K || tail_ld < R)
    return TQ_ERR_BAD_ARG;
  if (N % 8 != 0 || K > 65536) return TQ_ERR_UNSUPPORTED;
  if (!aligned16(w_t) || !aligned16(tail)) return TQ_ERR_MISALIGNED;
  if (M == 0) return TQ_OK;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(dev < 64 && configured[dev])) {
    cudaError_t e = cudaFuncSetAttribute(tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T_SMEM);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return TQ_ERR_CUDA;
    }
    if (dev < 64) configured[dev] = true;
  }
  CUtensorMap map;
  if (!make_tensor_map_2d(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_t, (uint64_t)N, (uint64_t)K,
                          (uint64_t)N * 2, T_COLS, T_KC / 2))
    return TQ_ERR_CUDA;
  TailParams p;
  p.idx = tail_idx16;
  p.val = reinterpret_cast<const uint16_t*>(tail_val);
  p.out = tail;
  p.M = M;
  p.N = N;
  p.K = K;
  p.R = R;
  p.ld = tail_ld;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  p.units_n = (N + T_COLS - 1) / T_COLS;
  // Rows per unit: the split of M with the shortest longest CTA.  A unit costs its rows and the strip of weights that it
  // streams, which weighs like the entries of some 50 rows (2048 x 6144 x 4096, R = 205: 37 us per unit of 128 rows, 0.2 us a row).
  long best = 0;
  const int um0 = (M + T_ROWS - 1) / T_ROWS;
  for (int um = um0; um <= 4 * um0 && (um == um0 || um <= (M + 15) / 16); ++um) {
    const int rows = ((M + um - 1) / um + 3) / 4 * 4;
    const long rounds = ((long)um * p.units_n + sms - 1) / sms;
    const long cost = rounds * (rows + 50);
    if (best == 0 || cost < best) best = cost, p.rows = rows;
  }
  p.units_m = (M + p.rows - 1) / p.rows;
  const int total = p.units_m * p.units_n;
  const int grid = total < sms ? total : sms;
  tail_kernel<<<grid, 8 * p.rows, T_SMEM, (cudaStream_t)stream>>>(map, p);
  return check_launch();
}
