// Fused prologue of the split W4A4 + tail linear, 16 elements per thread: every built width (sm_100a).
//
// One CTA of K / 16 threads works on one row at a time (grid-stride, the next row prefetched):
//   1. a thread loads its 16 contiguous elements with two 128-bit loads; optional RMSNorm;
//   2. rotation in fp32 with ascending butterfly strides: 1..8 in registers, 16..256 by shuffles across the warp, what is
//      left (strides 512.. of the full transform, stride 512 and the 12-point mix of 12 (x) 2^n) through ONE exchange in
//      shared memory; block-128 needs none;
//   3. one fp32 multiply by the normalisation and one rounding to bf16; from there on thread t owns elements
//      [16 t, 16 t + 16);
//   4. exact rank selection on the 15-bit magnitude key: distances from the row maximum in a 256-bin shared histogram, window
//      after window until the rank is reached (the first one for any Gaussian-like row); every warp reads the histogram
//      itself, so a window costs two barriers;
//   5. tail membership with ties broken by lowest index: per-thread masks and one scan over the CTA; the four threads of a
//      64-wide half slice sit in one warp, so records and boundaries are shuffles;
//   6. INT4 codes of the body with true-division semantics, stored straight to global memory.
//
// What bounds it: for few rows the latency of one row, i.e. the instructions a thread issues one after the other, which is
// why a thread has so few elements (one row of K = 4096, R = 205, with RMSNorm: 5.9 us; 9.5 with 64 elements per thread,
// 7.4 without norm in the 256-thread kernel with three exchanges that this one replaces); with many rows the
// instructions per element, where the 64-element kernel of tq_prologue_fast.cu (K = 4096, 12288, 14336) is ahead: 25 against 30 us at 2048 rows.
//
// Reference behaviour covered: tools/fused_threshold_topr_pack_ext_v57.py:96-194 (select, scales, pack),
// tools/fused_topr_pack_ext_v55.py:21-26,73-109 (clamp_s4, scale = max(key, eps)/7, body nibble 0 at tail positions, nibble
// order; fp16 input as there), plus the online rotation that the reference runs as a separate kernel.
#include "tq_common.cuh"
#include "tq_ptx.cuh"
#include "tq_prologue.cuh"

namespace tq {
namespace {

template <int KIND, int K>
struct WS {
  static constexpr int NT = K / 16, NW = NT / 32;
  static constexpr bool XBUF = (KIND == TQ_HAD_WHT && K > 512) || KIND == TQ_HAD_KRON12;
  static constexpr int X_OFF = 0;                               // [K] fp32 exchange buffer
  static constexpr int ROW_OFF = XBUF ? K * 4 : 0;              // [K] 16-bit rotated row
  static constexpr int HIST_OFF = ROW_OFF + K * 2;              // [256]
  static constexpr int RED_OFF = HIST_OFF + 1024;               // [32] warp maxima
  static constexpr int SCAN_OFF = RED_OFF + 128;                // [32] warp totals
  static constexpr int SUM_OFF = SCAN_OFF + 128;                // [256] sums of squares
  static constexpr int OVER_OFF = SUM_OFF + 1024;               // [32] entries beyond two of a group, by warp
  static constexpr int TAB_OFF = OVER_OFF + 128;                // group table
  static constexpr int BYTES = TAB_OFF + 128;
};

// rank is 1-based in (key descending) order; dd[j] holds the distances kmax - key of elements 2j (low half) and 2j + 1 (high
// half).  Uniform over the CTA.  `hist` (256 words) is zero on entry, and a barrier has passed since it was cleared.
template <int NT, int W>
__device__ __forceinline__ Sel select_rank_wide(const uint32_t (&dd)[W], int rank, uint32_t* hist, int tid) {
  const uint32_t hist_s = smem_u32(hist);
  const int lane = tid & 31;
  int below = 0;
  Sel out;
  out.kp = 32767;
  out.cnt_lt = 0;
  out.cnt_eq = 0;
  out.next_kp = -1;
  for (int base = 0; base < 32768; base += 256) {
    const uint32_t b4 = (uint32_t)base << 2;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const uint32_t lo = ((dd[j] << 2) & 0x3fffcu) - b4;
      const uint32_t hi = ((dd[j] >> 14) & 0x3fffcu) - b4;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.lt.u32 p, %1, 1024;\n\t"
          "setp.lt.u32 q, %2, 1024;\n\t"
          "@p red.shared.add.u32 [%0], 1;\n\t"
          "@q red.shared.add.u32 [%3], 1;\n\t}"
          ::"r"(hist_s + lo), "r"(lo), "r"(hi), "r"(hist_s + hi)
          : "memory");
    }
    __syncthreads();
    const uint4 ha = *reinterpret_cast<const uint4*>(hist + 8 * lane);
    const uint4 hb = *reinterpret_cast<const uint4*>(hist + 8 * lane + 4);
    const uint32_t h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += h[i];
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(FM, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t r2 = (uint32_t)(rank - below);
    const unsigned hit = __ballot_sync(FM, incl >= r2);
    if (hit) {
      const int fl = __ffs(hit) - 1;
      // in the lane of the hit: its first bin that reaches the rank; in later lanes the first bin that is not empty
      uint32_t acc = incl - s, lt = 0, eq = 0;
      int f = -1, nx = -1;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (f < 0 && acc + h[i] >= r2) {
          f = i;
          lt = acc;
          eq = h[i];
        }
        acc += h[i];
      }
      const int start = lane == fl ? f + 1 : 0;
#pragma unroll
      for (int i = 7; i >= 0; --i)
        if (i >= start && h[i] > 0) nx = i;
      const unsigned later = __ballot_sync(FM, lane >= fl && nx >= 0);
      out.kp = base + 8 * fl + __shfl_sync(FM, f, fl);
      out.cnt_lt = below + (int)__shfl_sync(FM, lt, fl);
      out.cnt_eq = (int)__shfl_sync(FM, eq, fl);
      const int ln = later ? __ffs(later) - 1 : 0;
      const int nb = __shfl_sync(FM, nx, ln);
      out.next_kp = later ? base + 8 * ln + nb : -1;
      return out;
    }
    below += (int)__shfl_sync(FM, incl, 31);
    __syncthreads();   // every warp has read the histogram
    for (int i = tid; i < 256; i += NT) hist[i] = 0u;
    __syncthreads();
  }
  out.cnt_lt = below;
  return out;
}

// register budgets: 64 up to 4096 and at 8192, 72 .. 85 for the others
constexpr int wide_min_ctas(int K) { return K <= 1024 ? 16 : K == 2048 ? 8 : K == 4096 ? 4 : K <= 8192 ? 2 : 1; }

// SP: the tail in its 2:4-sparse form too (p.sp)
template <int KIND, int K, int DT, bool NORM, bool SP>
__global__ void __launch_bounds__(K / 16, wide_min_ctas(K)) prologue_wide_kernel(const PrologueParams p) {
  using S = WS<KIND, K>;
  constexpr int NT = S::NT, NW = S::NW;
  static_assert(NT % 32 == 0 && NW <= 32, "row width");
  extern __shared__ __align__(16) unsigned char sm[];
  float* const xbuf = reinterpret_cast<float*>(sm + S::X_OFF);
  const smp rowbuf = sm + S::ROW_OFF;
  uint32_t* const hist = reinterpret_cast<uint32_t*>(sm + S::HIST_OFF);
  uint32_t* const red = reinterpret_cast<uint32_t*>(sm + S::RED_OFF);
  uint32_t* const scanw = reinterpret_cast<uint32_t*>(sm + S::SCAN_OFF);
  float* const sums = reinterpret_cast<float*>(sm + S::SUM_OFF);
  uint32_t* const overw = reinterpret_cast<uint32_t*>(sm + S::OVER_OFF);
  uint2* const table = reinterpret_cast<uint2*>(sm + S::TAB_OFF);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = p.R;
  const smp my_row = rowbuf + tid * 32;
  if (SP && tid < 16) table[tid] = GROUP_TABLE.e[tid];   // (read behind the barriers of the selection)

  pdl_wait();   // the rows may come from the kernel in front
  pdl_trigger();
  uint4 ga, gb;
  if (NORM) {
    ga = *reinterpret_cast<const uint4*>(p.gamma + 16 * tid);
    gb = *reinterpret_cast<const uint4*>(p.gamma + 16 * tid + 8);
  }
  const uint4* xrow = reinterpret_cast<const uint4*>(p.x + (size_t)blockIdx.x * K + 16 * tid);
  uint4 xa = make_uint4(0u, 0u, 0u, 0u), xb = xa;
  if ((int)blockIdx.x < p.M) {
    xa = ldg_na_128(xrow);
    xb = ldg_na_128(xrow + 1);
  }

  for (int m = blockIdx.x; m < p.M; m += gridDim.x) {
    uint32_t w[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
    if (m + (int)gridDim.x < p.M) {   // the next row, while this one is worked on
      xrow += (size_t)gridDim.x * (K / 8);
      xa = ldg_na_128(xrow);
      xb = ldg_na_128(xrow + 1);
    }
    for (int i = tid; i < 256; i += NT) hist[i] = 0u;

    if (KIND != TQ_HAD_NONE || NORM) {
      u64 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float lo, hi;
        unpack_word<TQ_BF16>(w[j], lo, hi);
        v[j] = pk2(lo, hi);
      }
      if (NORM) {
        // fixed sum order.  Widths of the 64-element kernel: 64 contiguous elements one after the other (here four lanes,
        // each continuing its predecessor's sum); other widths: a "thread" of 256 adds its 16-element chunks t, t + 256.
        // Then a butterfly over 32 such sums, and those in order.
        constexpr bool BY64 = K == 4096 || K == 12288 || K == 14336;
        constexpr int GROUPS = BY64 ? K / 2048 : (NT < 256 ? NT : 256) / 32;
        float sq[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float lo, hi;
          up2(v[j], lo, hi);
          sq[2 * j] = __fmul_rn(lo, lo);
          sq[2 * j + 1] = __fmul_rn(hi, hi);
        }
        float ss = 0.0f;
        if (BY64) {
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            float acc = __shfl_up_sync(FM, ss, 1);
            if (s == 0) acc = 0.0f;
#pragma unroll
            for (int e = 0; e < 16; ++e) acc = __fadd_rn(acc, sq[e]);
            if ((lane & 3) == s) ss = acc;
          }
          if ((lane & 3) == 3) sums[tid >> 2] = ss;
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) ss = __fadd_rn(ss, sq[e]);
          if (tid < 256) sums[tid] = ss;
          if (NT > 256) {
            __syncthreads();
            if (tid >= 256) {
              ss = sums[tid - 256];
#pragma unroll
              for (int e = 0; e < 16; ++e) ss = __fadd_rn(ss, sq[e]);
              sums[tid - 256] = ss;
            }
          }
        }
        __syncthreads();
        float tot = 0.0f;
#pragma unroll
        for (int q = 0; q < GROUPS; ++q) {
          float t = sums[32 * q + lane];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(FM, t, o));
          tot = q == 0 ? t : __fadd_rn(tot, t);
        }
        const float rms_inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)K), p.rms_eps)));
        const uint32_t gw[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float lo, hi, gl, gh;
          up2(v[j], lo, hi);
          unpack_word<TQ_BF16>(gw[j], gl, gh);
          uint32_t r = cvt_bf16x2(__fmul_rn(lo, rms_inv), __fmul_rn(hi, rms_inv));
          unpack_word<TQ_BF16>(r, lo, hi);
          r = cvt_bf16x2(__fmul_rn(lo, gl), __fmul_rn(hi, gh));
          w[j] = r;
          unpack_word<TQ_BF16>(r, lo, hi);
          v[j] = pk2(lo, hi);
        }
      }
      if (KIND != TQ_HAD_NONE) {
        // strides 1 .. 8 in registers
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float a, b;
          up2(v[j], a, b);
          v[j] = pk2(__fadd_rn(a, b), __fsub_rn(a, b));
        }
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if ((j & s) == 0) {
              const u64 a = v[j], b = v[j + s];
              v[j] = add2(a, b);
              v[j + s] = sub2(a, b);
            }
          }
        }
        // strides 16 .. 64 (block-128) or 16 .. 256 across the lanes: even lane v + partner, odd lane partner - v
        constexpr int TOP = KIND == TQ_HAD_BLOCK128 ? 8 : 32;
#pragma unroll
        for (int o = 1; o < TOP; o <<= 1) {
          const float sg = (lane & o) ? -1.0f : 1.0f;
          const u64 sg2 = pk2(sg, sg);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float lo, hi;
            up2(v[j], lo, hi);
            v[j] = fma2(sg2, v[j], pk2(__shfl_xor_sync(FM, lo, o), __shfl_xor_sync(FM, hi, o)));
          }
        }
        const u64 hs2 = pk2(p.hscale, p.hscale);
        if (!S::XBUF) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float lo, hi;
            up2(mul2(v[j], hs2), lo, hi);
            w[j] = cvt_bf16x2(lo, hi);
          }
        } else {
          // ---- own 16 values -> buffer; the 16-byte chunks of a thread's 64 bytes are permuted with the lane so that
          // eight lanes hit eight different bank groups
          {
            float* const dst = xbuf + 16 * tid;
            const int sw = (lane >> 1) & 3;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              float a0, a1, a2, a3;
              up2(v[2 * c], a0, a1);
              up2(v[2 * c + 1], a2, a3);
              *reinterpret_cast<float4*>(dst + 4 * (c ^ sw)) = make_float4(a0, a1, a2, a3);
            }
          }
          __syncthreads();
          // position q of a 512-element warp block -> word of the buffer
          auto place = [](int q) { return (q & ~15) + 4 * (((q >> 2) & 3) ^ ((q >> 5) & 3)) + (q & 3); };
          if (KIND == TQ_HAD_WHT) {
            // strides 512 .. K / 2: thread t takes positions PP t .. of the NB warp blocks
            constexpr int NB = K / 512, PP = NB > 16 ? 1 : 16 / NB;
            static_assert(KIND != TQ_HAD_WHT || K <= 512 || (NB * PP == 16 && NT * PP == 512), "full transform: K = 2^n <= 8192");
            float f[NB][PP];
#pragma unroll
            for (int q = 0; q < NB; ++q) {
              if (PP >= 4) {
#pragma unroll
                for (int c = 0; c < PP / 4; ++c) {
                  const float4 t = *reinterpret_cast<const float4*>(xbuf + 512 * q + place(PP * tid + 4 * c));
                  f[q][(4 * c) % PP] = t.x, f[q][(4 * c + 1) % PP] = t.y, f[q][(4 * c + 2) % PP] = t.z, f[q][(4 * c + 3) % PP] = t.w;
                }
              } else if (PP == 2) {
                const float2 t = *reinterpret_cast<const float2*>(xbuf + 512 * q + place(2 * tid));
                f[q][0] = t.x, f[q][1 % PP] = t.y;
              } else {
                f[q][0] = xbuf[512 * q + place(tid)];
              }
            }
#pragma unroll
            for (int s = 1; s < NB; s <<= 1) {
#pragma unroll
              for (int q = 0; q < NB; ++q) {
                if ((q & s) == 0) {
#pragma unroll
                  for (int e = 0; e < PP; ++e) {
                    const float x0 = f[q][e], x1 = f[q + s][e];
                    f[q][e] = __fadd_rn(x0, x1);
                    f[q + s][e] = __fsub_rn(x0, x1);
                  }
                }
              }
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) {
              const smp dst = rowbuf + (512 * q + PP * tid) * 2;
              if (PP == 1) {
                sts16(dst, f32_to_bf16_bits(__fmul_rn(f[q][0], p.hscale)));
              } else {
#pragma unroll
                for (int e = 0; e < PP; e += 2)
                  sts32(dst + 2 * e, cvt_bf16x2(__fmul_rn(f[q][e], p.hscale), __fmul_rn(f[q][(e + 1) % PP], p.hscale)));
              }
            }
          } else {
            // the 12-point mix, sums in the fixed order a = 0 .. 11.  K = 12288: threads 0 .. 511 take one position of the 24
            // warp blocks, stride 512 first; K = 6144: threads 0 .. 255 take two positions of the 12 warp blocks.
            static_assert(KIND != TQ_HAD_KRON12 || K == 12288 || K == 6144, "12 (x) 2^n: K = 6144, 12288");
            constexpr bool TWO = K == 12288;
            if (tid < (TWO ? 512 : 256)) {
              u64 c[12];
#pragma unroll
              for (int a = 0; a < 12; ++a) {
                if (TWO) {
                  const float* src = xbuf + place(tid) + 1024 * a;
                  const float x0 = src[0], x1 = src[512];
                  c[a] = pk2(__fadd_rn(x0, x1), __fsub_rn(x0, x1));
                } else {
                  const float2 t = *reinterpret_cast<const float2*>(xbuf + place(2 * tid) + 512 * a);
                  c[a] = pk2(t.x, t.y);
                }
              }
              float n0, n1;
              up2(c[0], n0, n1);
              const u64 neg0 = pk2(-n0, -n1);
#pragma unroll
              for (int a2 = 0; a2 < 12; ++a2) {
                u64 acc = (H12_NEG[a2] & 1) ? neg0 : c[0];
#pragma unroll
                for (int a = 1; a < 12; ++a) acc = ((H12_NEG[a2] >> a) & 1) ? sub2(acc, c[a]) : add2(acc, c[a]);
                float lo, hi;
                up2(mul2(acc, hs2), lo, hi);
                const uint32_t b2 = cvt_bf16x2(lo, hi);
                if (TWO) {
                  sts16(rowbuf + (1024 * a2 + tid) * 2, b2);
                  sts16(rowbuf + (1024 * a2 + 512 + tid) * 2, b2 >> 16);
                } else {
                  sts32(rowbuf + (512 * a2 + 2 * tid) * 2, b2);
                }
              }
            }
          }
          __syncthreads();
          const uint4 qa = lds128(my_row), qb = lds128(my_row + 16);
          w[0] = qa.x, w[1] = qa.y, w[2] = qa.z, w[3] = qa.w, w[4] = qb.x, w[5] = qb.y, w[6] = qb.z, w[7] = qb.w;
        }
      }
    }
    if (!S::XBUF) {   // (single values are picked from the row buffer below, each thread its own)
      sts128(my_row, make_uint4(w[0], w[1], w[2], w[3]));
      sts128(my_row + 16, make_uint4(w[4], w[5], w[6], w[7]));
    }

    // =============================================================== thread t owns elements [16 t, 16 t + 16)
    if (p.x_rot) {
      uint4* dst = reinterpret_cast<uint4*>(p.x_rot + (size_t)m * K + 16 * tid);
      dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
      dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    // ---- row maximum of the 15-bit magnitude keys
    uint32_t kmax;
    {
      uint32_t mx = 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = max_u16x2(mx, w[j] & 0x7fff7fffu);
      mx = max(mx & 0xffffu, mx >> 16);
      mx = __reduce_max_sync(FM, mx);
      if (lane == 0) red[warp] = mx;
      __syncthreads();
      kmax = __reduce_max_sync(FM, lane < NW ? red[lane] : 0u);
    }
    uint32_t dd[8];   // distances from the maximum, two per word
    {
      const uint32_t km2 = kmax | (kmax << 16);
#pragma unroll
      for (int j = 0; j < 8; ++j) dd[j] = km2 - (w[j] & 0x7fff7fffu);
    }

    // ---- rank selection: first the tail rank, then, if it does not follow from that result, the body rank
    int Tkp = -1, cnt_lt = 0, body_kp = 0;
    {
      int want = R > 0 ? R : (p.dr > 1 ? p.dr : 0);
      bool tail_pass = R > 0;
      while (want) {   // uniform over the CTA
        const Sel s = select_rank_wide<NT, 8>(dd, want, hist, tid);
        want = 0;
        if (tail_pass) {
          tail_pass = false;
          Tkp = s.kp;
          cnt_lt = s.cnt_lt;
          if (p.dr > s.cnt_lt && p.dr <= s.cnt_lt + s.cnt_eq) {
            body_kp = s.kp;
          } else if (p.dr == s.cnt_lt + s.cnt_eq + 1 && s.next_kp >= 0) {
            body_kp = s.next_kp;
          } else {
            want = p.dr;
            __syncthreads();   // the second selection starts from a cleared histogram
            for (int i = tid; i < 256; i += NT) hist[i] = 0u;
            __syncthreads();
          }
        } else {
          body_kp = s.kp;
        }
      }
    }
    const int need = R - cnt_lt;   // keys equal to the threshold that still belong to the tail (lowest indices)
    const float tscale = make_scale(key_to_f32<DT>(kmax), p.eps, p.scale_mode);
    const float bscale = make_scale(key_to_f32<DT>(kmax - (uint32_t)body_kp), p.eps, p.scale_mode);
    const float brinv = __fdiv_rn(1.0f, bscale);

    // ---- tail membership.  Mask layout: bit i = element 2 i (low half of word i), bit 16 + i = element 2 i + 1.
    uint32_t tm = 0u;
    int n_over = 0;   // this thread's entries beyond two of a group of four
    if (R > 0) {
      const uint32_t T2 = (uint32_t)Tkp | ((uint32_t)Tkp << 16);
      const uint32_t c_le = 0x80008000u + T2, c_lt = 0x7fff7fffu + T2;   // per half: top bit set <=> d <= T, d < T
      uint32_t le = 0u, lt = 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        le |= ((c_le - dd[j]) >> (15 - j)) & (0x00010001u << j);
        lt |= ((c_lt - dd[j]) >> (15 - j)) & (0x00010001u << j);
      }
      const uint32_t eq = le ^ lt;
      const uint32_t cnt = (uint32_t)__popc(lt) | ((uint32_t)__popc(eq) << 16);
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FM, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) scanw[warp] = incl;
      __syncthreads();
      uint32_t wt = lane < NW ? scanw[lane] : 0u;   // totals of the warps in front, summed by every warp
      wt = lane < warp ? wt : 0u;
      const uint32_t pre = incl - cnt + __reduce_add_sync(FM, wt);
      const int gt_before = (int)(pre & 0xffffu), eq_before = (int)(pre >> 16);
      const int tail_before = gt_before + min(eq_before, need);
      tm = lt;
      int take = need - eq_before;   // ties of this thread that join the tail: its first `take` in index order
      if (take > 0 && eq) {
        if (take >= (int)(cnt >> 16)) {
          tm |= eq;
        } else {
          uint32_t ev = eq & 0xffffu, od = eq >> 16;
          while ((ev | od) && take > 0) {
            const int a = ev ? __ffs(ev) - 1 : 32, b = od ? __ffs(od) - 1 : 32;
            if (a <= b) {
              tm |= 1u << a;
              ev &= ev - 1u;
            } else {
              tm |= 0x10000u << b;
              od &= od - 1u;
            }
            --take;
          }
        }
      }
      const int ntail = __popc(tm);
      if (p.tail_dense) {
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = w[j] & (((tm >> j) & 0x00010001u) * 0xffffu);
        uint4* dst = reinterpret_cast<uint4*>(p.tail_dense + (size_t)m * K + 16 * tid);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
      }
      // list position of the half slice's first entry and its entry count (four lanes per half slice)
      const int hs = tid >> 2;
      const int hs_first = __shfl_sync(FM, tail_before, lane & ~3);
      if (p.tail_ptr) {   // run boundaries of the row's ascending index list at multiples of 128
        if ((tid & 7) == 0) p.tail_ptr[(size_t)m * p.ptr_ld + (tid >> 3)] = (uint16_t)tail_before;
        if (tid == 0) p.tail_ptr[(size_t)m * p.ptr_ld + K / 128] = (uint16_t)R;
      }
      if (p.tail_cnt) {
        int c = ntail;
        c += __shfl_xor_sync(FM, c, 1);
        c += __shfl_xor_sync(FM, c, 2);
        if ((lane & 3) == 0) {
          p.tail_cnt[((size_t)(m >> 7) * (K / 64) + hs) * 128 + (m & 127)] = (uint16_t)c;
          // the rows that pad M to a multiple of 256 (the CTA-pair GEMM's tile height) have no entries; they are shared
          // out over the rows
          for (int r = p.M + m; r < (p.M + 255) / 256 * 256; r += p.M)
            p.tail_cnt[((size_t)(r >> 7) * (K / 64) + hs) * 128 + (r & 127)] = 0;
        }
      }
      if (p.tail_idx16 || p.tail_val || p.idx32 || p.top_q || p.tail_rec) {
        // ---- tail entries in ascending index order
        const size_t rl = (size_t)m * p.tail_ld, rb = (size_t)m * R;
        uint32_t ev = tm & 0xffffu, od = tm >> 16;
        int r = tail_before;
        while (ev | od) {
          const int a = ev ? __ffs(ev) - 1 : 32, b = od ? __ffs(od) - 1 : 32;
          int e;
          if (a <= b) {
            e = 2 * a;
            ev &= ev - 1u;
          } else {
            e = 2 * b + 1;
            od &= od - 1u;
          }
          const uint32_t i = (uint32_t)(16 * tid + e);
          const uint32_t vb = lds16(my_row + 2 * e);
          if (p.tail_idx16) p.tail_idx16[rl + r] = (uint16_t)i;
          if (p.tail_val) p.tail_val[rl + r] = (uint16_t)vb;
          if (p.idx32) p.idx32[rb + r] = (int32_t)i;
          if (p.top_q) {
            float xv, dummy;
            unpack_word<DT>(vb, xv, dummy);
            p.top_q[rb + r] = (int8_t)(int)fminf(fmaxf(rintf(__fdiv_rn(xv, tscale)), -8.0f), 7.0f);
          }
          if (p.tail_rec) {
            const int jr = r - hs_first;
            const uint32_t e6 = i & 63u;
            if (jr < TQ_TAIL_REC_CAP)
              // half the byte offset of the value inside its 128-byte row of the swizzled operand tile; the bf16 value
              p.tail_rec[(((size_t)(m >> 7) * (K / 64) + hs) * 128 + (m & 127)) * TQ_TAIL_REC_CAP + jr] =
                  ((((e6 >> 3) ^ ((uint32_t)m & 7u)) << 3) | (e6 & 7u)) | (vb << 16);
          }
          ++r;
        }
      }
      if (SP) {   // 2:4-sparse operand (see the 64-element kernel)
        if ((uint32_t)Tkp == kmax) {   // the threshold is zero: entries that are add nothing
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (!(w[j] & 0x7fffu)) tm &= ~(1u << j);
            if (!(w[j] & 0x7fff0000u)) tm &= ~(0x10000u << j);
          }
        }
        uint32_t v[4], places = 0u;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint2 e = table[group_index(tm, 2 * g)];
          v[g] = prmt(w[2 * g], w[2 * g + 1], e.x) & e.y;
          places |= (e.x >> 16) << (4 * g);
        }
        *reinterpret_cast<uint4*>(p.sp.val + (size_t)m * (K / 2) + 8 * tid) = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint16_t*>(p.sp.meta)[(size_t)m * (K / 16) + tid] = (uint16_t)places;
        over_groups(tm, n_over);
        const int w_over = __reduce_add_sync(FM, n_over);
        if (lane == 0) overw[warp] = (uint32_t)w_over;
      }
    }

    // ---- INT4 codes of the body (see the 64-element kernel): reciprocal product, magic-number rounding, IEEE division
    // for the elements on a rounding boundary
    const bool clampq = p.dr != R + 1;   // (body scale below the body maximum: codes can leave [-8, 7])
    uint32_t fm = 0u;
    uint32_t ev[2], od[2];   // byte k of ev[s] / od[s] = code of element 2 k / 2 k + 1 of 8-group s
    {
      const u64 rinv2 = pk2(brinv, brinv);
      const u64 magic2 = pk2(12582912.0f, 12582912.0f), nmagic2 = pk2(-12582912.0f, -12582912.0f);
      uint32_t ul[8], uh[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float lo, hi;
        unpack_word<DT>(w[j], lo, hi);
        u64 t2 = mul2(pk2(lo, hi), rinv2);
        if (clampq) {
          float a, b;
          up2(t2, a, b);
          t2 = pk2(fminf(fmaxf(a, -8.0f), 7.0f), fminf(fmaxf(b, -8.0f), 7.0f));
        }
        const u64 u2 = add2(t2, magic2);
        const u64 e2 = sub2(t2, add2(u2, nmagic2));
        float el, eh, fl, fh;
        up2(e2, el, eh);
        if (fabsf(el) >= 0.499998f) fm |= 1u << j;
        if (fabsf(eh) >= 0.499998f) fm |= 0x10000u << j;
        up2(u2, fl, fh);
        ul[j] = __float_as_uint(fl);
        uh[j] = __float_as_uint(fh);
      }
      auto bytemask = [](uint32_t nib) -> uint32_t { return (((nib & 0xfu) * 0x00204081u) & 0x01010101u) * 0xffu; };
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int j0 = 4 * s;
        ev[s] = prmt(prmt(ul[j0], ul[j0 + 1], 0x0040u), prmt(ul[j0 + 2], ul[j0 + 3], 0x0040u), 0x5410u) & ~bytemask(tm >> j0);
        od[s] = prmt(prmt(uh[j0], uh[j0 + 1], 0x0040u), prmt(uh[j0 + 2], uh[j0 + 3], 0x0040u), 0x5410u) & ~bytemask(tm >> (16 + j0));
      }
    }
    for (uint32_t mk = fm & ~tm; mk; mk &= mk - 1u) {
      const int b = __ffs(mk) - 1, jw = b & 15;   // word of the element
      const uint32_t vb = lds16(my_row + 2 * (b < 16 ? 2 * b : 2 * jw + 1));
      float xv, dummy;
      unpack_word<DT>(vb, xv, dummy);
      const uint32_t code = (uint32_t)(int)fminf(fmaxf(rintf(__fdiv_rn(xv, bscale)), -8.0f), 7.0f) & 0xffu;
      const uint32_t keep = ~(0xffu << (8 * (jw & 3))), put = code << (8 * (jw & 3));
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if ((jw >> 2) == s) {
          if (b < 16)
            ev[s] = (ev[s] & keep) | put;
          else
            od[s] = (od[s] & keep) | put;
        }
      }
    }
    if (p.a_q8)
      *reinterpret_cast<uint4*>(p.a_q8 + (size_t)m * K + 16 * tid) = make_uint4(ev[0], od[0], ev[1], od[1]);
    if (p.a_pack)
      *reinterpret_cast<uint2*>(p.a_pack + (size_t)m * (K / 2) + 8 * tid) =
          make_uint2((ev[0] & 0x0f0f0f0fu) | ((od[0] & 0x0f0f0f0fu) << 4), (ev[1] & 0x0f0f0f0fu) | ((od[1] & 0x0f0f0f0fu) << 4));
    if (tid == 0) {
      p.body_scale[m] = bscale;
      if (p.top_scale) p.top_scale[m] = tscale;
    }
    if (SP) {   // (R > 0) the list of the entries beyond two of a group, in index order
      __syncthreads();
      const int cw = lane < NW ? (int)overw[lane] : 0;
      const int total = __reduce_add_sync(FM, cw);
      int pos = __reduce_add_sync(FM, lane < warp ? cw : 0);
      if (tid == 0) p.sp.over_cnt[m] = (uint16_t)total;
      if (overw[warp]) {   // (uniform over the warp)
        int incl = n_over;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(FM, incl, o);
          if (lane >= o) incl += t;
        }
        pos += incl - n_over;
        if (n_over)
          for_each_over(tm, over_groups(tm, incl), [&](int e) {
            p.sp.over[(size_t)m * p.sp.over_ld + pos] = (uint32_t)(16 * tid + e) | (lds16(my_row + 2 * e) << 16);
            ++pos;
          });
      }
    }
    if (m + (int)gridDim.x < p.M) __syncthreads();   // the next row starts over on all buffers
  }
}

template <int KIND, int K, int DT, bool NORM, bool SP = false>
int launch_wide(const PrologueParams& p, cudaStream_t st) {
  using S = WS<KIND, K>;
  auto kern = prologue_wide_kernel<KIND, K, DT, NORM, SP>;
  static int grid_per_dev[64] = {};
  int dev = 0;
  const int sms = current_device_sms(&dev);
  int cap = dev < 64 ? grid_per_dev[dev] : 0;
  if (!cap) {
    int per_sm = 1;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, S::NT, S::BYTES);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return TQ_ERR_CUDA;
    }
    cap = sms * (per_sm < 1 ? 1 : per_sm);
    if (dev < 64) grid_per_dev[dev] = cap;
  }
  return launch_pdl(kern, dim3(p.M < cap ? p.M : cap), dim3(S::NT), (size_t)S::BYTES, st, 1, p);
}

}  // namespace

// TQ_ERR_UNSUPPORTED for a (rotation, width, type) that is not built.
int run_prologue_wide(int kind, int K, int dtype, const PrologueParams& p, cudaStream_t st) {
  const bool norm = p.gamma != nullptr;
  if (dtype == TQ_FP16) {
    if (kind != TQ_HAD_NONE || norm) return TQ_ERR_UNSUPPORTED;
    if (K == 4096) return launch_wide<TQ_HAD_NONE, 4096, TQ_FP16, false>(p, st);
    if (K == 12288) return launch_wide<TQ_HAD_NONE, 12288, TQ_FP16, false>(p, st);
    return TQ_ERR_UNSUPPORTED;
  }
  if (p.sp.val) {   // (full rotations only)
#define TQ_WIDE_SP(KIND, KK)                     \
  if (kind == KIND && K == KK)                   \
    return norm ? launch_wide<KIND, KK, TQ_BF16, true, true>(p, st) : launch_wide<KIND, KK, TQ_BF16, false, true>(p, st);
    TQ_WIDE_SP(TQ_HAD_WHT, 512)
    TQ_WIDE_SP(TQ_HAD_WHT, 1024)
    TQ_WIDE_SP(TQ_HAD_WHT, 2048)
    TQ_WIDE_SP(TQ_HAD_WHT, 4096)
    TQ_WIDE_SP(TQ_HAD_WHT, 8192)
    TQ_WIDE_SP(TQ_HAD_KRON12, 6144)
    TQ_WIDE_SP(TQ_HAD_KRON12, 12288)
#undef TQ_WIDE_SP
    return TQ_ERR_UNSUPPORTED;
  }
#define TQ_WIDE(KIND, KK)                        \
  if (kind == KIND && K == KK)                   \
    return norm ? launch_wide<KIND, KK, TQ_BF16, true>(p, st) : launch_wide<KIND, KK, TQ_BF16, false>(p, st);
  TQ_WIDE(TQ_HAD_WHT, 512)
  TQ_WIDE(TQ_HAD_WHT, 1024)
  TQ_WIDE(TQ_HAD_WHT, 2048)
  TQ_WIDE(TQ_HAD_WHT, 4096)
  TQ_WIDE(TQ_HAD_WHT, 8192)
  TQ_WIDE(TQ_HAD_KRON12, 6144)
  TQ_WIDE(TQ_HAD_KRON12, 12288)
  TQ_WIDE(TQ_HAD_BLOCK128, 2048)
  TQ_WIDE(TQ_HAD_BLOCK128, 14336)
  TQ_WIDE(TQ_HAD_NONE, 512)
  TQ_WIDE(TQ_HAD_NONE, 1024)
  TQ_WIDE(TQ_HAD_NONE, 2048)
  TQ_WIDE(TQ_HAD_NONE, 4096)
  TQ_WIDE(TQ_HAD_NONE, 6144)
  TQ_WIDE(TQ_HAD_NONE, 8192)
  TQ_WIDE(TQ_HAD_NONE, 12288)
  TQ_WIDE(TQ_HAD_NONE, 14336)
#undef TQ_WIDE
  return TQ_ERR_UNSUPPORTED;
}

}  // namespace tq
