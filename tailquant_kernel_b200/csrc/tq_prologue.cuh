// Types and small helpers shared by the two prologue kernels (tq_prologue_wide.cu, tq_prologue_fast.cu).
#pragma once

#include "tq_common.cuh"

namespace tq {
namespace {

// 12x12 Paley-I Hadamard over GF(11): bit j of row a2 set <=> H[a2][j] = -1.
__device__ constexpr unsigned short H12_NEG[12] = {0x000, 0x475, 0x8e9, 0x1d3, 0x3a5, 0x749,
                                                   0xe91, 0xd23, 0xa47, 0x48f, 0x91d, 0x23b};

struct PrologueParams {
  const __nv_bfloat16* x;
  int M, R, dr, tail_ld, ptr_ld;
  float eps, hscale;
  int scale_mode;  // 0: max(t, eps) / 7 (activations); 1: max(t / 7, eps) (weights)
  uint8_t* a_pack;
  int8_t* a_q8;
  float* body_scale;
  float* top_scale;
  uint16_t* tail_idx16;
  uint16_t* tail_val;
  uint16_t* tail_ptr;  // [M, ptr_ld]: entries with index < 128 * j, j = 0 .. K/128
  uint32_t* tail_rec;  // [2 ceil(M/256)][K/64][128][TQ_TAIL_REC_CAP]: tile position | bf16 << 16
  uint16_t* tail_cnt;  // [2 ceil(M/256)][K/64][128]: entries per 64-wide half slice
  int32_t* idx32;
  int8_t* top_q;
  uint16_t* x_rot;
  uint16_t* tail_dense;   // [M, K] bf16: the rotated row with every element outside the tail set to zero (R > 0), or NULL
  const uint16_t* gamma;  // [K] bf16 RMSNorm weight, or NULL: x is used as it is
  float rms_eps;
  SparseTail sp;          // (val == NULL: not asked for)
  bool wide;              // a_q8, x_rot, tail_dense, sp.val are 32-byte aligned
};

// What to do with a group of four, by which of its elements are tail entries (bit 0 = element 0, 1 = element 2, 2 = element 1,
// 3 = element 3, the order in which the membership masks have them).  x: byte selector that picks the first two entries (or as
// many as there are, completed by other elements), their places << 16; y: the halves of the pair that are entries.
struct GroupTable {
  uint2 e[16];
  constexpr GroupTable() : e{} {
    for (int i = 0; i < 16; ++i) {
      const int in[4] = {i & 1, (i >> 2) & 1, (i >> 1) & 1, (i >> 3) & 1};
      int a = -1, b = -1;
      for (int k = 0; k < 4; ++k)
        if (in[k]) {
          if (a < 0) a = k;
          else if (b < 0) b = k;
        }
      if (a < 0) a = 0;
      if (b < 0) b = a == 3 ? 2 : a + 1;
      if (a > b) {
        const int t = a;
        a = b;
        b = t;
      }
      e[i].x = (unsigned)(2 * a | (2 * a + 1) << 4 | 2 * b << 8 | (2 * b + 1) << 12 | (a | b << 2) << 16);
      e[i].y = (in[a] ? 0xffffu : 0u) | (in[b] ? 0xffff0000u : 0u);
    }
  }
};
__device__ const GroupTable GROUP_TABLE = GroupTable();

// Entry of the table for the group whose elements are words j, j + 1 of a mask half (see the kernels: bit j = element 2 j,
// bit 16 + j = element 2 j + 1).
__device__ __forceinline__ uint32_t group_index(uint32_t tm, int j) {
  const uint32_t t = (tm >> j) & 0x00030003u;
  return (t | (t >> 14)) & 15u;
}

// Groups with more than two entries, bit 2 g of the result for group g of the mask; `extra`: their entries beyond two.
__device__ __forceinline__ uint32_t over_groups(uint32_t tm, int& extra) {
  const uint32_t lo = tm & 0xffffu, hi = tm >> 16;   // elements 0 and 2, elements 1 and 3 in neighbouring bits
  const uint32_t both = lo & (lo >> 1), any = lo | (lo >> 1), hboth = hi & (hi >> 1), hany = hi | (hi >> 1);
  const uint32_t om = ((both & hany) | (any & hboth)) & 0x5555u;
  extra = __popc(om) + __popc(both & hboth & 0x5555u);
  return om;
}

// The entries beyond the first two of each of these groups, in ascending order: f(element offset inside the mask).
template <typename F>
__device__ __forceinline__ void for_each_over(uint32_t tm, uint32_t om, F&& f) {
  for (; om; om &= om - 1u) {
    const int j = __ffs(om) - 1;
    const uint32_t t = tm >> j;
    int seen = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if ((t >> ((e >> 1) + 16 * (e & 1))) & 1u)
        if (++seen > 2) f(2 * j + e);
  }
}

__device__ __forceinline__ float make_scale(float t, float eps, int mode) {
  return mode == 0 ? __fdiv_rn(fmaxf(t, eps), 7.0f) : fmaxf(__fdiv_rn(t, 7.0f), eps);
}

}  // namespace

// Kernels of tq_prologue_wide.cu and tq_prologue_fast.cu for the (rotation, K, dtype) combinations they are built for;
// TQ_ERR_UNSUPPORTED otherwise.
int run_prologue_wide(int kind, int K, int dtype, const PrologueParams& p, cudaStream_t st);
int run_prologue_fast(int kind, int K, int dtype, const PrologueParams& p, cudaStream_t st);

}  // namespace tq
