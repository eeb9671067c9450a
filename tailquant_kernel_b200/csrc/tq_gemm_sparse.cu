// Split GEMM on CTA pairs with the tail as a 2:4-sparse operand (sm_100a): the computation of tq_gemm_pair.cu, tail product
// on tcgen05.mma.sp.
//
// The tail has a few entries in a hundred, at positions that the rotation spreads over K, so a group of four neighbours
// rarely holds more than two.  The prologue writes each row as its first two entries per group (K / 2 values) and their
// places (four bits per group), and what is left over as a list.  The tensor cores then take half the time for the tail product
// and a row's tail operand is half the bytes, loaded by TMA: no warps that build it.
//
// The entries left over (one row in two has one at R = 0.05 K, K = 4096) follow behind the K slices of a tile, 64 of them at a
// time, as one more dense slice: warp 0 collects them from the lists of the tile's 256 rows while the K slices run and builds A,
// one value per column; B are rows of w_t, gathered by TMA.  A dense slice takes about 0.8 us.  (Added in the epilogue instead,
// where nothing hides the loads, the left-over entries cost 30 % of the GEMM.)  Their number is without bound, and rows that
// consist of a few equal values have many: 2048 x 6144 x 4096 with three equal large channels, whose indices agree in the last two
// bits, (7.4 left over in every row) 203 us, with four (26) 471, where the dense product takes 125 and 130.
//
// Tile: 256 rows x up to 224 channels per pair.  The two accumulators (int32, fp32) of 224 columns leave 64 columns of tensor
// memory for the places (16 per K slice); 256 channels would leave none.  The last tile of a row of tiles is as narrow as its
// channels need (a multiple of 32).
//
// Operands come in two rings of three slots: INT8 slots (activation codes by TMA, INT4 weights loaded into registers and
// widened x16 by two groups of four warps, even and odd K slices) and bf16 slots (tail values and bf16 weight rows of a K slice
// by TMA, places by four warps from global memory into tensor memory).  Barriers, cluster protocol and epilogue as in the pair
// kernel.
//
// What bounds it: a K slice takes about 1250 cycles, its eight MMAs at the rate that dense bf16 GEMMs reach on this part; a tile
// boundary another 6000.  While it runs, a load that misses the few KB of L1 beside the rings takes 2000 cycles, so everything
// is requested two slices ahead and no thread has anything in local memory (56 bytes of spills: 327 -> 384 us at 24576
// channels).  us, R = 0.05 K, plain activations with 1 channel in 256 fifty times as large, dense pair kernel -> this one:
// 2048 x 6144 x 4096 115 -> 92, x 4096 x 4096 79 -> 69, x 24576 x 4096 413 -> 315, x 4096 x 12288 214 -> 187, R = 0.01 K
// 4096 x 28672 x 4096 966 -> 704.
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace tq {
namespace {

// warp 0: left-over entries, 1: MMA issuer, 2..5 / 6..9: wideners of even / odd K slices, 10..13: places of the tail values,
// 14: activation operands, 15: bf16 weight rows.  Warps 2..13 share the epilogue.
constexpr int SPG_THREADS = 512;
constexpr int SPG_BM = 128, SPG_BN = 224, SPG_BH = SPG_BN / 2;

struct SG {
  static constexpr int SI = 3, SB = 3;                    // INT8 slots, bf16 slots
  static constexpr int LIST = 64, LISTS = 3;              // left-over entries of a dense slice, buffers for them
  static constexpr int A = SPG_BM * 128, B = SPG_BH * 128;
  static constexpr int ISLOT = A + B;                     // codes of this CTA's rows, widened weights of its channels
  static constexpr int BSLOT = A + 2 * B;                 // tail values, bf16 weights of the two 64-wide halves
  static constexpr int B_OFF = SI * ISLOT;
  static constexpr int BAR_OFF = B_OFF + SB * BSLOT;
  static constexpr int NUM_BARS = 2 * SI + 2 * SB + 6 + 2 * LISTS;
  static constexpr int LIST_OFF = (BAR_OFF + NUM_BARS * 8 + 16 + 15) / 16 * 16;
  static constexpr int SCALE_OFF = (LIST_OFF + LISTS * LIST * 4 + 1024 + 8 + 15) / 16 * 16;   // channel scales and bias
  static constexpr int DYN = SCALE_OFF + 2 * SPG_BN * 4 + 1024;
  static constexpr uint32_t T_TAIL = SPG_BN, T_META = 2 * SPG_BN;   // tensor-memory columns
  static constexpr uint32_t T_SLOT = 16;   // of a slot's places: one of four columns (the MMA takes an aligned address) per 32 of K
};
static_assert(SG::DYN <= 232448 && SG::T_META + SG::T_SLOT * SG::SB <= 512 , "sparse pair kernel");

struct SparseGemmParams {
  int M, N, K, tiles_m, tiles_n, kbt, early;
  int over_ld;
  const uint32_t* meta;           // (SparseTail)
  const uint16_t* over_cnt;
  const uint32_t* over;           // [M, over_ld]
  const uint8_t* b_col;
  const uint16_t* w_t;            // [K, N] bf16, or NULL: the same values from w_rot
  const uint16_t* w_rot;          // [N, K] bf16
  const float* sx;
  const float* sw;
  const float* bias;
  __nv_bfloat16* out;
  int32_t* dbg_acc;
  float* dbg_tail;
};

__device__ __forceinline__ void umma_sp_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t meta, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.sp.cta_group::2.kind::f16 [%0], %1, %2, [%3], %4, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(meta), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar_cluster)
      : "memory");
}
// four words of a lane to every fourth column from `taddr` on
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr + 4u * j), "r"(r[j]) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 16 packed bytes of a channel's K slice -> 32 codes (x16) in the 128-byte-swizzled operand tile (as widen_rows)
__device__ __forceinline__ void widen_piece(unsigned char* dst, int row, int piece, uint4 w) {
  unsigned char* drow = dst + (row >> 3) * 1024 + (row & 7) * 128;
  *reinterpret_cast<uint4*>(drow + (((2 * piece) ^ (row & 7)) << 4)) =
      make_uint4((w.x << 4) & 0xf0f0f0f0u, w.x & 0xf0f0f0f0u, (w.y << 4) & 0xf0f0f0f0u, w.y & 0xf0f0f0f0u);
  *reinterpret_cast<uint4*>(drow + (((2 * piece + 1) ^ (row & 7)) << 4)) =
      make_uint4((w.z << 4) & 0xf0f0f0f0u, w.z & 0xf0f0f0f0u, (w.w << 4) & 0xf0f0f0f0u, w.w & 0xf0f0f0f0u);
}

// Barriers of a CTA (shared-window addresses)
struct SparseBars {
  uint32_t bars;
  __device__ __forceinline__ uint32_t full_i(int s) const { return bars + 8u * s; }
  __device__ __forceinline__ uint32_t empty_i(int s) const { return bars + 8u * (SG::SI + s); }
  __device__ __forceinline__ uint32_t full_b(int s) const { return bars + 8u * (2 * SG::SI + s); }
  __device__ __forceinline__ uint32_t empty_b(int s) const { return bars + 8u * (2 * SG::SI + SG::SB + s); }
  __device__ __forceinline__ uint32_t acc_full() const { return bars + 8u * (2 * SG::SI + 2 * SG::SB); }
  __device__ __forceinline__ uint32_t acc_empty() const { return acc_full() + 8u; }
  // the places of a tile's last K slice are in (by tile parity, as the next one: no role can fall two phases behind)
  __device__ __forceinline__ uint32_t last_placed(int b) const { return acc_full() + 16u + 8u * b; }
  // the number of dense slices of a tile is known
  __device__ __forceinline__ uint32_t over_known(int b) const { return acc_full() + 32u + 8u * b; }
  // the entries of a dense slice are in their buffer
  __device__ __forceinline__ uint32_t listed(int b) const { return acc_full() + 48u + 8u * b; }
  // and so is its operand A
  __device__ __forceinline__ uint32_t built(int b) const { return acc_full() + 48u + 8u * (SG::LISTS + b); }
};

// The tiles of a pair: pair, pair + npairs, ..., row tiles first
struct SparseTiles {
  int pair, npairs, count, tiles_m, N;
  __device__ __forceinline__ int tile(int i) const { return i * npairs + pair; }
  __device__ __forceinline__ int mt(int i) const { return tile(i) % tiles_m; }
  __device__ __forceinline__ int n0(int i) const { return tile(i) / tiles_m * SPG_BN; }
  __device__ __forceinline__ int width(int n0) const { return min(SPG_BN, (N - n0 + 31) & ~31); }
};

// MMA issuer (one thread of the leader CTA).  A function of its own, so that its loop keeps its registers whatever the other
// roles need: inlined, the kernel took 20 % longer whenever another role grew.
__device__ __noinline__ void sparse_issue(SparseTiles tiles, SparseBars b, uint32_t base, uint32_t tmem_base, int kbt,
                                          volatile int* extra, volatile int* abort_flag) {
  using S = SG;
  const uint64_t di0 = make_smem_desc(base), db0 = make_smem_desc(base + S::B_OFF);
  uint64_t di = di0, db = db0;
  uint32_t fi = b.full_i(0), fb = b.full_b(0), phi = 0, phb = 0, tm = tmem_base + S::T_META;
  constexpr uint64_t A = S::A >> 4, B = S::B >> 4;
  auto next_b = [&]() {
    fb += 8u;
    db += S::BSLOT >> 4;
    tm += S::T_SLOT;
    if (fb == b.full_b(S::SB)) {
      fb = b.full_b(0);
      db = db0;
      tm = tmem_base + S::T_META;
      phb ^= 1u;
    }
  };
  for (int i = 0; i < tiles.count; ++i) {
    const uint32_t n_bits = (uint32_t)(tiles.width(tiles.n0(i)) >> 3) << 17;
    const uint32_t idesc_i8 = make_idesc_i8<0, 256>() | n_bits;
    const uint32_t idesc = make_idesc_bf16<0, 256>() | n_bits, idesc_sp = idesc | 4u, idesc_bf = idesc | 1u << 16;   // sparse; B transposed
    auto sparse_slice = [&](uint32_t acc) -> bool {
      if (!mbar_wait(fb, phb, abort_flag, 0x20000u)) return false;
      tc_fence_after();
      // 32 of K: 32 bytes of values, 64 bytes of weights, one column of places
      umma_sp_bf16_pair(tmem_base + S::T_TAIL, db, db + A, tm, idesc_sp, acc);
      umma_sp_bf16_pair(tmem_base + S::T_TAIL, db + 2, db + A + 4, tm + 4, idesc_sp, 1u);
      umma_sp_bf16_pair(tmem_base + S::T_TAIL, db + 4, db + A + B, tm + 8, idesc_sp, 1u);
      umma_sp_bf16_pair(tmem_base + S::T_TAIL, db + 6, db + A + B + 4, tm + 12, idesc_sp, 1u);
      umma_commit_pair(fb + 8u * S::SB);
      next_b();
      return true;
    };
    if (!mbar_wait(b.acc_empty(), (uint32_t)(i & 1) ^ 1u, abort_flag, 0x8000u)) return;
    tc_fence_after();
    uint32_t acc = 0;
    for (int kb = 0; kb < kbt; ++kb) {
      if (!mbar_wait(fi, phi, abort_flag, 0x10000u)) return;
      tc_fence_after();
      umma_i8_pair(tmem_base, di, di + A, idesc_i8, acc);
      umma_i8_pair(tmem_base, di + 2, di + A + 2, idesc_i8, 1u);
      umma_i8_pair(tmem_base, di + 4, di + A + 4, idesc_i8, 1u);
      umma_i8_pair(tmem_base, di + 6, di + A + 6, idesc_i8, 1u);
      umma_commit_pair(fi + 8u * S::SI);
      fi += 8u;
      di += S::ISLOT >> 4;
      if (fi == b.full_i(S::SI)) {
        fi = b.full_i(0);
        di = di0;
        phi ^= 1u;
      }
      if (!sparse_slice(acc)) return;
      acc = 1u;
    }
    if (!mbar_wait(b.over_known(i & 1), (uint32_t)((i >> 1) & 1), abort_flag, 0x800000u)) return;
    const int ex = extra[i & 1];
    for (int q = 0; q < ex; ++q) {
      if (!mbar_wait(fb, phb, abort_flag, 0x20000u)) return;
      tc_fence_after();
      // left-over entries: rows of w_t, so B has its channels in a row (blocks of 64 channels 8192 bytes apart)
      const uint64_t w = (db + A) | (uint64_t)(8192u >> 4) << 16;
      umma_bf16_pair(tmem_base + S::T_TAIL, db, w, idesc_bf, 1u);
      umma_bf16_pair(tmem_base + S::T_TAIL, db + 2, w + 128, idesc_bf, 1u);
      umma_bf16_pair(tmem_base + S::T_TAIL, db + 4, w + 256, idesc_bf, 1u);
      umma_bf16_pair(tmem_base + S::T_TAIL, db + 6, w + 384, idesc_bf, 1u);
      umma_commit_pair(fb + 8u * S::SB);
      next_b();
    }
    umma_commit_pair(b.acc_full());
  }
}

// Four rows of a matrix (box: one row of 64 elements, 128-byte swizzle), one behind the other
__device__ __forceinline__ void tma_gather4_pair(uint32_t dst, const CUtensorMap* map, int x, uint32_t y0, uint32_t y1, uint32_t y2,
                                                 uint32_t y3, uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 [%0], "
      "[%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(bar_cluster)
      : "memory");
}

// two accumulators at once: one wait for both loads
__device__ __forceinline__ void tmem_ld16_pair(uint32_t ta, uint32_t (&a)[16], uint32_t tb, uint32_t (&b)[16]) {
#define TQ_LD16(addr, r)                                                                                                   \
  asm volatile(                                                                                                            \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"             \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),         \
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                            \
      : "r"(addr))
  TQ_LD16(ta, a);
  TQ_LD16(tb, b);
#undef TQ_LD16
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
template <int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SPG_THREADS, 1)
sparse_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a8, const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ CUtensorMap tmap_t,
                   const SparseGemmParams p) {
  using S = SG;
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* sm = smem_dyn + (base - raw);
  const uint32_t bars = base + S::BAR_OFF;
  const SparseBars b{bars};
  uint32_t* const list = reinterpret_cast<uint32_t*>(sm + S::LIST_OFF);   // [LISTS][LIST] left-over entries: index | bf16 << 16
  uint32_t* const starts = list + S::LISTS * S::LIST;                     // [256] places of the rows' first ones
  volatile int* const extra = reinterpret_cast<volatile int*>(starts + 256);   // [2] dense slices, by tile parity
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + S::BAR_OFF + S::NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + S::BAR_OFF + S::NUM_BARS * 8 + 4);

  float* const scales = reinterpret_cast<float*>(sm + S::SCALE_OFF);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();          // 0 = leader
  SparseTiles tiles;
  tiles.pair = blockIdx.x >> 1;
  tiles.npairs = gridDim.x >> 1;
  tiles.tiles_m = p.tiles_m;
  tiles.N = p.N;
  tiles.count = (p.tiles_m * p.tiles_n - tiles.pair + tiles.npairs - 1) / tiles.npairs;   // (no more pairs than tiles)
  const int my_tiles = tiles.count, kbt = p.kbt, G = my_tiles * kbt;   // K slices of this pair over all its tiles
  auto lead = [&](uint32_t bar) { return map_to_cta(bar, 0u); };
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_a8)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_v)) : "memory");
    for (int s = 0; s < S::SI; ++s) {
      mbar_init(b.full_i(s), 8 + 1);   // four widening warps of each CTA and the activation producer (leader's copy is used)
      mbar_init(b.empty_i(s), 1);
    }
    for (int s = 0; s < S::SB; ++s) {
      mbar_init(b.full_b(s), 8 + 2);   // four warps of each CTA with the places and the two producers
      mbar_init(b.empty_b(s), 1);
    }
    mbar_init(b.acc_full(), 1);
    mbar_init(b.acc_empty(), 2 * 12);    // the epilogue warps of both CTAs
    for (int k = 0; k < 2; ++k) {
      mbar_init(b.over_known(k), 1);
      mbar_init(b.last_placed(k), 4);
    }
    for (int k = 0; k < S::LISTS; ++k) {
      mbar_init(b.listed(k), 1);
      mbar_init(b.built(k), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  bool ok = true;
  // Epilogue of local tile i, shared by warps 2..13: y = bf16((float(acc) * s_x) * s_w + tail + bias), rows of the warp's
  // lane quadrant, every third chunk of 32 channels.  The next tile's MMAs wait for the accumulators, so everything that can
  // lies outside of the stretch in which they are read: the channel scales are fetched to shared memory before it, the
  // output is stored behind it (32 bytes of a row at a time).
  auto epilogue = [&](int i) -> bool {
    const int quad = warp & 3, third = (warp - 2) >> 2, n_tile = tiles.n0(i), chunks = tiles.width(n_tile) >> 5;
    const int row = (2 * tiles.mt(i) + rank) * SPG_BM + quad * 32 + lane;
    const bool row_ok = row < p.M;
    const float sx = row_ok ? p.sx[row] : 0.0f;
    float sc[3], bi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int n = n_tile + 32 * (third + 3 * k) + lane;
      const bool in = third + 3 * k < chunks && n < p.N;
      sc[k] = in ? p.sw[n] : 0.0f;
      bi[k] = in && p.bias ? p.bias[n] : 0.0f;
    }
    if (!__all_sync(0xffffffffu, mbar_wait(b.acc_full(), (uint32_t)(i & 1), abort_flag, 0x40000u))) return false;
    tc_fence_after();
    // (every warp is through with the former tile's scales; each of the four warps of a chunk writes the same values)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (third + 3 * k < chunks) {
        scales[32 * (third + 3 * k) + lane] = sc[k];
        scales[SPG_BN + 32 * (third + 3 * k) + lane] = bi[k];
      }
    __syncwarp();
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    __nv_bfloat16* const orow = p.out + (size_t)(row_ok ? row : 0) * (ACT ? p.N / 2 : p.N);
    const bool wide = (p.N & 15) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
#pragma unroll 1
    for (int c = 2 * third; c < 2 * chunks; c += (c & 1) ? 5 : 1) {   // 16 channels at a time
      uint32_t ri[16], rf[16], o[8];
      __syncwarp();
      tmem_ld16_pair(lane_addr + (uint32_t)(c * 16), ri, lane_addr + S::T_TAIL + (uint32_t)(c * 16), rf);
      if ((c & 1) && c + 5 >= 2 * chunks) {   // this warp's last ones
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead(b.acc_empty()));
      }
      const float4* sw4 = reinterpret_cast<const float4*>(scales + 16 * c);
      const float4* bi4 = reinterpret_cast<const float4*>(scales + SPG_BN + 16 * c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 w4 = sw4[j];
        float d0 = __fadd_rn(__fmul_rn(__fmul_rn((float)((int)ri[4 * j] >> 4), sx), w4.x), __uint_as_float(rf[4 * j]));
        float d1 = __fadd_rn(__fmul_rn(__fmul_rn((float)((int)ri[4 * j + 1] >> 4), sx), w4.y), __uint_as_float(rf[4 * j + 1]));
        float d2 = __fadd_rn(__fmul_rn(__fmul_rn((float)((int)ri[4 * j + 2] >> 4), sx), w4.z), __uint_as_float(rf[4 * j + 2]));
        float d3 = __fadd_rn(__fmul_rn(__fmul_rn((float)((int)ri[4 * j + 3] >> 4), sx), w4.w), __uint_as_float(rf[4 * j + 3]));
        if (p.bias) {
          const float4 b4 = bi4[j];
          d0 = __fadd_rn(d0, b4.x);
          d1 = __fadd_rn(d1, b4.y);
          d2 = __fadd_rn(d2, b4.z);
          d3 = __fadd_rn(d3, b4.w);
        }
        if (ACT) {
          o[j] = swiglu_bf16_bits(d0, d1) | (swiglu_bf16_bits(d2, d3) << 16);
        } else {
          o[2 * j] = pack_bf16x2(d0, d1);
          o[2 * j + 1] = pack_bf16x2(d2, d3);
        }
      }
      const int nc = n_tile + 16 * c;
      if (!row_ok || nc >= p.N) continue;
      if (ACT) {
        *reinterpret_cast<uint4*>(orow + nc / 2) = make_uint4(o[0], o[1], o[2], o[3]);   // (N % 16 == 0)
      } else if (wide) {
        st_global_v8(orow + nc, o);
      } else {   // (N is a multiple of 8)
        *reinterpret_cast<uint4*>(orow + nc) = make_uint4(o[0], o[1], o[2], o[3]);
        if (nc + 8 < p.N) *reinterpret_cast<uint4*>(orow + nc + 8) = make_uint4(o[4], o[5], o[6], o[7]);
      }
      if (p.dbg_acc || p.dbg_tail) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (nc + j < p.N && p.dbg_acc) p.dbg_acc[(size_t)row * p.N + nc + j] = (int)ri[j] >> 4;
          if (nc + j < p.N && p.dbg_tail) p.dbg_tail[(size_t)row * p.N + nc + j] = __uint_as_float(rf[j]);
        }
      }
    }
    if (third >= chunks) {   // (a narrow tile has no chunk for this warp)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead(b.acc_empty()));
    }
    return true;
  };
  int epi_done = 0;
  auto catch_up = [&](int upto) {
    while (ok && epi_done < upto) ok = epilogue(epi_done++);
  };
  // rows of w_t of dense slice `n` (counted over all tiles), the 64 channels from `ch` on, four rows per load
  auto gather = [&](int n, int ch, uint32_t dst, uint32_t bar) -> bool {
    if (!mbar_wait(b.listed(n % S::LISTS), (uint32_t)((n / S::LISTS) & 1), abort_flag, 0x4000000u)) return false;
    const uint4* l = reinterpret_cast<const uint4*>(list + n % S::LISTS * S::LIST);
#pragma unroll 4
    for (int k = 0; k < S::LIST / 4; ++k) {
      const uint4 v = l[k];
      tma_gather4_pair(dst + 512u * k, &tmap_t, ch, v.x & 0xffffu, v.y & 0xffffu, v.z & 0xffffu, v.w & 0xffffu, bar);
    }
    return true;
  };
  // what follows the K slices of local tile i (known from its first slices on)
  auto extra_of = [&](int i) -> int {
    ok = mbar_wait(b.over_known(i & 1), (uint32_t)((i >> 1) & 1), abort_flag, 0x800000u);
    return ok ? extra[i & 1] : 0;
  };

  if (!(p.early && warp == 15)) pdl_wait();   // (weights do not come from the kernel in front)

  if (warp == 0) {
    // ------------------------------------------------------------------ left-over entries
    int use = 0, slices = 0;   // uses of the bf16 ring, dense slices so far
    for (int i = 0; ok && i < my_tiles; ++i) {
      const int m0 = 256 * tiles.mt(i), n_tile = tiles.n0(i), n0 = n_tile + rank * (tiles.width(n_tile) >> 1);
      // entries of rows 8 lane .. 8 lane + 7 of the tile, places of their first ones in its list.  (Counts and indices are held
      // inside their arrays: outputs that no prologue has filled give wrong sums and no access out of range.)
      int total = 0;
      {
        const int row = m0 + 8 * lane;
        uint32_t cnt[8];
        if (row + 8 <= p.M) {
          const uint4 v = *reinterpret_cast<const uint4*>(p.over_cnt + row);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) cnt[j] = min((w[j >> 1] >> (16 * (j & 1))) & 0xffffu, (uint32_t)p.over_ld);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) cnt[j] = row + j < p.M ? min((uint32_t)p.over_cnt[row + j], (uint32_t)p.over_ld) : 0u;
        }
        uint32_t sum = 0, incl;
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += cnt[j];
        incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        total = (int)__shfl_sync(0xffffffffu, incl, 31);
        uint32_t first = incl - sum;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          starts[8 * lane + j] = first;
          first += cnt[j];
        }
        if (lane == 0) {
          extra[i & 1] = (total + 63) / 64;
          mbar_arrive(b.over_known(i & 1));
        }
        __syncwarp();
      }
      // This lane's two entries of a dense slice: place `at` of the tile's list, its row by bisection of the first places (so
      // that a row with many entries is loaded by many lanes); beyond the last one zeros of row 0.
      uint32_t v[2], r[2], nv[2], nr[2];
      auto load = [&](int at, uint32_t& value, uint32_t& row) {
        value = row = 0u;
        if (at >= total) return;
#pragma unroll
        for (int step = 128; step > 0; step >>= 1)
          if (starts[row + step] <= (uint32_t)at) row += step;
        value = p.over[(size_t)(m0 + (int)row) * p.over_ld + (at - (int)starts[row])];
      };
      load(lane, nv[0], nr[0]);
      load(lane + 32, nv[1], nr[1]);
      ok = __all_sync(0xffffffffu, mbar_wait(b.last_placed(i & 1), (uint32_t)((i >> 1) & 1), abort_flag, 0x1000000u));
      use += kbt;
      // (the slots of the uses from here on are at most one release behind what is waited for)
      for (int q = 0; ok && 64 * q < total; ++q, ++use, ++slices) {
        const int s = use % S::SB, l = slices % S::LISTS;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          v[j] = (nv[j] & 0xffffu) < (uint32_t)p.K ? nv[j] : 0u;
          r[j] = nr[j];
        }
        ok = __all_sync(0xffffffffu, mbar_wait(b.empty_b(s), (uint32_t)((use / S::SB) & 1) ^ 1u, abort_flag, 0x2000000u));
        if (!ok) break;
        tc_fence_after();
        unsigned char* const a = sm + S::B_OFF + s * S::BSLOT;
        // (the slice that used this buffer before, three ago, is through)
        list[l * S::LIST + lane] = v[0];
        list[l * S::LIST + lane + 32] = v[1];
        __syncwarp();
        if (lane == 0) mbar_arrive(b.listed(l));   // warps 14 and 15 load the rows of w_t
        // (the next slice's entries, on their way while this one is built: 26 a row 538 -> 471 us; asked for in front of the wait
        // for the slot they cost the kernel 1.2 % with plain rows)
#pragma unroll
        for (int j = 0; j < 2; ++j) load(64 * (q + 1) + lane + 32 * j, nv[j], nr[j]);
#pragma unroll 8
        for (int c = 0; c < S::A / 512; ++c) *reinterpret_cast<uint4*>(a + c * 512 + lane * 16) = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int k = lane + 32 * j, row = (int)r[j] - rank * SPG_BM;
          if (row >= 0 && row < SPG_BM)
            *reinterpret_cast<uint16_t*>(a + (row >> 3) * 1024 + (row & 7) * 128 + (((k >> 3) ^ (row & 7)) << 4) + (k & 7) * 2) =
                (uint16_t)(v[j] >> 16);
        }
        if (!p.w_t) {
          for (int item = lane; item < 64 * SPG_BH / 8; item += 32) {   // 64 entries x 14 pieces of eight channels
            const int e = item / (SPG_BH / 8), c = item - e * (SPG_BH / 8), n = n0 + 8 * c;
            const size_t k = list[l * S::LIST + e] & 0xffffu;
            uint32_t w[4] = {0u, 0u, 0u, 0u};
            if (n < p.N)
#pragma unroll
              for (int j = 0; j < 8; ++j) w[j >> 1] |= (uint32_t)p.w_rot[(size_t)(n + j) * p.K + k] << (16 * (j & 1));
            st_shared_v4(smem_u32(a) + S::A + (uint32_t)((c >> 3) * 8192 + (e >> 3) * 1024 + (e & 7) * 128 + (((c & 7) ^ (e & 7)) << 4)), w);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(b.built(l));
      }
    }
  } else if (warp == 15) {
    // ------------------------------------------------------------------ bf16 weight rows, both halves of a K slice at once
    if (elect_one()) {
      int s = 0, slices = 0;
      uint32_t ph = 1;
      for (int i = 0; ok && i < my_tiles; ++i) {
        const int n0 = tiles.n0(i), nrow = n0 + rank * (tiles.width(n0) >> 1);
        for (int kb = 0; kb < kbt; ++kb) {
          if (!(ok = mbar_wait(b.empty_b(s), ph, abort_flag, 0x4000u))) break;
          if (rank == 0) mbar_arrive_expect_tx(b.full_b(s), 4 * S::B);
          tma_load_3d_pair(base + S::B_OFF + s * S::BSLOT + S::A, &tmap_w, 0, nrow, 2 * kb, lead(b.full_b(s)));
          if (++s == S::SB) {
            s = 0;
            ph ^= 1u;
          }
        }
        const int ex = ok ? extra_of(i) : 0;
        for (int q = 0; ok && q < ex; ++q, ++slices) {   // dense slices: the first 64 channels
          if (!(ok = mbar_wait(b.empty_b(s), ph, abort_flag, 0x4000u))) break;
          if (rank == 0 && p.w_t) mbar_arrive_expect_tx(b.full_b(s), 2 * 64 * 128);
          if (rank == 0 && !p.w_t) mbar_arrive(b.full_b(s));
          if (p.w_t && !(ok = gather(slices, nrow, base + S::B_OFF + s * S::BSLOT + S::A, lead(b.full_b(s))))) break;
          if (++s == S::SB) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (warp == 14) {
    // ------------------------------------------------------------------ activation codes and tail values
    if (elect_one()) {
      int si = 0, sb = 0, slices = 0;
      uint32_t phi = 1, phb = 1;
      for (int i = 0; ok && i < my_tiles; ++i) {
        const int mrow = (2 * tiles.mt(i) + rank) * SPG_BM, n0 = tiles.n0(i), nrow = n0 + rank * (tiles.width(n0) >> 1);
        for (int kb = 0; kb < kbt; ++kb) {
          if (!(ok = mbar_wait(b.empty_i(si), phi, abort_flag, 0x2000u))) break;
          if (rank == 0) mbar_arrive_expect_tx(b.full_i(si), 2 * S::A);
          tma_load_2d_pair(base + si * S::ISLOT, &tmap_a8, kb * 128, mrow, lead(b.full_i(si)));
          if (++si == S::SI) {
            si = 0;
            phi ^= 1u;
          }
          if (!(ok = mbar_wait(b.empty_b(sb), phb, abort_flag, 0x80000u))) break;
          if (rank == 0) mbar_arrive_expect_tx(b.full_b(sb), 2 * S::A);
          tma_load_2d_pair(base + S::B_OFF + sb * S::BSLOT, &tmap_v, kb * 64, mrow, lead(b.full_b(sb)));
          if (++sb == S::SB) {
            sb = 0;
            phb ^= 1u;
          }
        }
        const int ex = ok ? extra_of(i) : 0;
        for (int q = 0; ok && q < ex; ++q, ++slices) {   // dense slices: the other 48
          if (!(ok = mbar_wait(b.empty_b(sb), phb, abort_flag, 0x80000u))) break;
          if (rank == 0 && p.w_t) mbar_arrive_expect_tx(b.full_b(sb), 2 * 64 * 128);
          if (rank == 0 && !p.w_t) mbar_arrive(b.full_b(sb));
          if (p.w_t && !(ok = gather(slices, nrow + 64, base + S::B_OFF + sb * S::BSLOT + S::A + 8192u, lead(b.full_b(sb))))) break;
          if (++sb == S::SB) {
            sb = 0;
            phb ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) sparse_issue(tiles, b, base, tmem_base, kbt, extra, abort_flag);
  } else if (warp >= 2 && warp < 10) {
    // ------------------------------------------------------------------ wideners: group 0 the even K slices, group 1 the
    // odd ones (counted over all tiles).  A thread has up to four 16-byte pieces of a slice and loads those of its next slice as
    // soon as it has stored them (two slices ahead; through staging buffers filled by TMA, which left room for two INT8 slots
    // only, 2048 x 6144 x 4096 took 8 % longer).  A tile's epilogue share follows the group's first slice of the
    // next tile.
    const int group = (warp - 2) >> 2, wtid = (threadIdx.x - 64) & 127;
    const int row0 = wtid >> 2, piece = wtid & 3;
    int tile = 0, kb = group, fetched = -1;   // tile and slice of the pieces in `w`, tile that `src` belongs to
    const uint8_t* src = nullptr;
    int rows = 0;                             // of the tile from row0 on that exist
    uint4 w[4];
    auto fetch = [&]() {
      while (kb >= kbt) {
        kb -= kbt;
        ++tile;
      }
      if (tile >= my_tiles) return;
      if (tile != fetched) {
        fetched = tile;
        const int n0 = tiles.n0(tile), n = n0 + rank * (tiles.width(n0) >> 1) + row0;
        src = p.b_col + (size_t)n * (p.K / 2) + piece * 16;
        rows = min(SPG_BH - row0, p.N - n);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        w[u] = make_uint4(0u, 0u, 0u, 0u);
        if (32 * u < rows) w[u] = ldg_na_128(src + (size_t)kb * 64 + (size_t)u * 16 * p.K);
      }
    };
    fetch();
    int s = group;
    uint32_t ph = 1;
    for (int g = group; g < G && ok; g += 2) {
      const int now = tile;
      ok = __all_sync(0xffffffffu, mbar_wait(b.empty_i(s), ph, abort_flag, 0x200000u));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (row0 + 32 * u < SPG_BH) widen_piece(sm + s * S::ISLOT + S::A, row0 + 32 * u, piece, w[u]);
      kb += 2;
      fetch();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead(b.full_i(s)));
      if ((s += 2) >= S::SI) {
        s -= S::SI;
        ph ^= 1u;
      }
      catch_up(now);
    }
    catch_up(my_tiles);
  } else if (warp >= 10) {
    // ------------------------------------------------------------------ places of the tail values.  A lane loads the 32 bytes
    // of its row and two K slices at a time, two slices or more ahead (a load takes the time of two slices here).  Tensor
    // memory wants, in lane 16 a + 8 h + b and the column of 32 of K, the places of the groups 4 h .. 4 h + 3 of rows
    // 16 a + b (low half) and 16 a + b + 8 (high half).
    const int quad = warp & 3, h = (lane >> 3) & 1, tid = quad * 32 + lane;   // lane of tensor memory, row of this CTA
    const uint32_t taddr = tmem_base + S::T_META + ((uint32_t)(quad * 32) << 16);
    const uint32_t sel = h ? 0x7632u : 0x5410u;
    const size_t meta_ld = (size_t)(p.K / 32);
    int s = 0, slices = 0;   // bf16 slot and the parity of the release that its next use waits for; dense slices so far
    uint32_t ph = 1;
    auto next_slot = [&]() {
      if (++s == S::SB) {
        s = 0;
        ph ^= 1u;
      }
    };
    auto wait_slot = [&]() -> bool {
      ok = __all_sync(0xffffffffu, mbar_wait(b.empty_b(s), ph, abort_flag, 0x400000u));
      tc_fence_after();
      return ok;
    };
    auto place = [&](uint4 v) -> bool {
      if (!ok) return false;
      const uint32_t own[4] = {v.x, v.y, v.z, v.w};
      uint32_t r[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, own[j], 8);
        r[j] = __byte_perm(h ? other : own[j], h ? own[j] : other, sel);
      }
      if (!wait_slot()) return false;
      tmem_st4(taddr + S::T_SLOT * s, r);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead(b.full_b(s)));
      next_slot();
      return true;
    };
    auto row_meta = [&](int i) -> const uint32_t* {   // this lane's row of tile i, NULL beyond M
      const int row = (2 * tiles.mt(i) + rank) * SPG_BM + tid;
      return row < p.M ? p.meta + (size_t)row * meta_ld : nullptr;
    };
    auto load2 = [&](const uint32_t* m, int kb, uint4& x, uint4& y) {
      x = y = make_uint4(0x44444444u, 0x44444444u, 0x44444444u, 0x44444444u);
      if (m) {
        x = *reinterpret_cast<const uint4*>(m + 4 * kb);
        y = *reinterpret_cast<const uint4*>(m + 4 * kb + 4);
      }
    };
    const uint32_t* cur = my_tiles > 0 ? row_meta(0) : nullptr;
    uint4 a0, a1, b0, b1;
    load2(cur, 0, a0, a1);
    load2(cur, 2, b0, b1);

    for (int i = 0; ok && i < my_tiles; ++i) {
      const uint32_t* nxt = i + 1 < my_tiles ? row_meta(i + 1) : nullptr;
#pragma unroll 1
      for (int kb = 0; ok && kb < kbt; kb += 4) {
        place(a0);
        place(a1);
        load2(kb + 4 < kbt ? cur : nxt, kb + 4 < kbt ? kb + 4 : 0, a0, a1);
        place(b0);
        if (kb == 0) catch_up(i);
        place(b1);
        load2(kb + 4 < kbt ? cur : nxt, kb + 4 < kbt ? kb + 6 : 2, b0, b1);
      }
      cur = nxt;
      if (!ok) break;
      if (lane == 0) mbar_arrive(b.last_placed(i & 1));
      const int ex = extra_of(i);
      if (!(ok = __all_sync(0xffffffffu, ok))) break;
      // dense slices: these warps pass on that warp 0 has built A.  (Every role takes part in every use of a slot: one that only
      // watched could find the slot released twice and wait, by parity, for a release that needs it.)
      for (int q = 0; q < ex && wait_slot(); ++q, ++slices) {
        ok = __all_sync(0xffffffffu, mbar_wait(b.built(slices % S::LISTS), (uint32_t)((slices / S::LISTS) & 1), abort_flag, 0x8000000u));
        if (!ok) break;
        if (lane == 0) mbar_arrive_cluster(lead(b.full_b(s)));
        next_slot();
      }
    }
    catch_up(my_tiles);
  }

  __syncwarp();
  pdl_wait();
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <int ACT>
int launch_sparse_gemm(const CUtensorMap& ma, const CUtensorMap& mw, const CUtensorMap& mv,
                       const CUtensorMap& mt, const SparseGemmParams& p, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  const int sms = current_device_sms(&dev);
  if (!(dev < 64 && configured[dev])) {
    cudaError_t e = cudaFuncSetAttribute(sparse_gemm_kernel<ACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SG::DYN);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return TQ_ERR_CUDA;
    }
    if (dev < 64) configured[dev] = true;
  }
  const int total = p.tiles_m * p.tiles_n, pairs = total < sms / 2 ? total : sms / 2;
  return launch_pdl(sparse_gemm_kernel<ACT>, dim3(2 * pairs), dim3(SPG_THREADS), (size_t)SG::DYN, st, 1, ma, mw, mv, mt, p);
}

}  // namespace

// `early`: the kernel in front in the stream is the prologue of this call
int run_sparse_gemm(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col, const float* w_scale, const void* w_rot,
                    const void* w_t, const SparseTail& sp,
                    const float* bias, void* out_bf16, int32_t* dbg_acc, float* dbg_tail, int M, int N, int K, int act, bool early, cudaStream_t st) {
  SparseGemmParams p = {};
  p.M = M;
  p.N = N;
  p.K = K;
  p.tiles_m = (M + 2 * SPG_BM - 1) / (2 * SPG_BM);
  p.tiles_n = (N + SPG_BN - 1) / SPG_BN;
  p.kbt = K / 128;
  p.early = early ? 1 : 0;
  p.b_col = b_col;
  p.meta = sp.meta;
  p.over_cnt = sp.over_cnt;
  p.over = sp.over;
  p.over_ld = sp.over_ld;
  p.w_t = reinterpret_cast<const uint16_t*>(w_t);
  p.w_rot = reinterpret_cast<const uint16_t*>(w_rot);
  p.sx = body_scale;
  p.sw = w_scale;
  p.bias = bias;
  p.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  p.dbg_acc = dbg_acc;
  p.dbg_tail = dbg_tail;
  CUtensorMap ma, mw, mv, mt;
  if (!make_tensor_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_q8, (uint64_t)K, (uint64_t)M, (uint64_t)K, 128, SPG_BM, true) ||
      !make_tensor_map_2d(&mv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, sp.val, (uint64_t)(K / 2), (uint64_t)M, (uint64_t)K, 64, SPG_BM, true) ||
      !make_tensor_map_2d(&mt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_t ? w_t : w_rot, (uint64_t)(w_t ? N : K), (uint64_t)(w_t ? K : N),
                          (uint64_t)(w_t ? N : K) * 2, 64, 1, true) ||   // (not read without w_t)
      !make_tensor_map_kblocks(&mw, w_rot, (uint64_t)K, (uint64_t)N, SPG_BH, 2))
    return TQ_ERR_CUDA;
  return act ? launch_sparse_gemm<1>(ma, mw, mv, mt, p, st) : launch_sparse_gemm<0>(ma, mw, mv, mt, p, st);
}

}  // namespace tq

extern "C" int tq_split_gemm_sparse(const int8_t* a_q8, const float* body_scale, const uint8_t* b_col, const float* w_scale,
                                    const void* w_rot, const void* w_t, int R, void* sp_val, uint32_t* sp_meta,
                                    uint16_t* sp_over_cnt, uint32_t* sp_over, int sp_over_ld, const float* bias,
                                    void* out_bf16, int32_t* dbg_acc, float* dbg_tail, int M, int N, int K, int act,
                                    void* stream) {
  using namespace tq;
  if (!a_q8 || !body_scale || !b_col || !w_scale || !w_rot || R <= 0 || R >= K || sp_over_ld < (R + 1) / 2 ||
      !sp_val || !sp_meta || !sp_over_cnt || !sp_over || !out_bf16 || M < 0 || N <= 0 || K <= 0 || (act & ~1))
    return TQ_ERR_BAD_ARG;
  if (K % 512 != 0 || N % (act ? 16 : 8) != 0 || K > 65536) return TQ_ERR_UNSUPPORTED;
  if (!aligned16(a_q8) || !aligned16(b_col) || !aligned16(out_bf16) || !aligned16(w_scale) || !aligned16(w_rot) ||
      (w_t && !aligned16(w_t)) || !aligned16(sp_over_cnt) || !aligned16(sp_val) || !aligned16(sp_meta) ||
      (bias && !aligned16(bias)))
    return TQ_ERR_MISALIGNED;
  if (M == 0) return TQ_OK;
  const SparseTail sp = {reinterpret_cast<uint16_t*>(sp_val), sp_meta, sp_over_cnt, sp_over, sp_over_ld};
  return run_sparse_gemm(a_q8, body_scale, b_col, w_scale, w_rot, w_t, sp, bias, out_bf16,
                         dbg_acc, dbg_tail, M, N, K, act, false,
                         (cudaStream_t)stream);
}
