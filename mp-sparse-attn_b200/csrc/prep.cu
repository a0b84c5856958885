// Operand preparation in one launch: up to two operands (Q and K) to MXFP8 / MXFP4 along the depth, and V for P.V - transposed
// to fp16, or quantised along the sequence.  16-bit input whose depth is 64 or a multiple of 128; every other case has a
// kernel of its own in quant.cu / attn.cu.  Results are those of the reference's quantizers, bit for bit
// (ours/quant_mxint8.py:164-221, :276-351).
//
// What bounds it: memory, once the E2M1 rule of the reference stays under ~8 ALU instructions an element (ALU 64 lanes per
// clock and SM against 7 elements per clock and SM at 6.2 TB/s, one code per byte).  The rule - keep the exponent, set the
// mantissa bit iff the mantissa exceeds .25 (:315-331) - does not agree with the hardware's round-to-nearest conversion; done
// on fp32 values it took 10 instructions an element.  bf16 values are therefore classified in pairs on their 16-bit patterns:
// for x > 0 the pattern is a piecewise linear logarithm, the softmax scale folded into Q only moves the class boundaries, and
// a boundary is an integer (found on the host by trying the 128 mantissas).  5.5 instructions an element.
#include "api_internal.h"
#include "common.cuh"
#include "quant_math.h"
#include "prep.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <type_traits>

namespace mpsa {
namespace {

constexpr int PREP_THREADS = 256;
constexpr int PREP_V_SMEM = 128 * 256;                // 128 keys x 128 depth elements of 16 bits

template <typename T> __device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi);
template <> __device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& lo, float& hi) {
  lo = __uint_as_float(w << 16);
  hi = __uint_as_float(w & 0xffff0000u);
}
template <> __device__ __forceinline__ void unpack2<__half>(uint32_t w, float& lo, float& hi) {
  const float2 f = __half22float2(*reinterpret_cast<__half2*>(&w));
  lo = f.x;
  hi = f.y;
}
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ float pattern_to_float(uint32_t h);
template <> __device__ __forceinline__ float pattern_to_float<__nv_bfloat16>(uint32_t h) { return __uint_as_float(h << 16); }
template <> __device__ __forceinline__ float pattern_to_float<__half>(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

__device__ __forceinline__ void mul2(float& a, float& b, float c) {      // (a, b) *= c, one instruction for the pair
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(c));
}
template <bool E4M3>
__device__ __forceinline__ uint32_t cvt_fp8x4(float y0, float y1, float y2, float y3) {
  uint32_t r;
  if (E4M3) {
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\t"
        "mov.b32 %0, {lo, hi};\n\t}" : "=r"(r) : "f"(y0), "f"(y1), "f"(y2), "f"(y3));
  } else {
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e5m2x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e5m2x2.f32 hi, %4, %3;\n\t"
        "mov.b32 %0, {lo, hi};\n\t}" : "=r"(r) : "f"(y0), "f"(y1), "f"(y2), "f"(y3));
  }
  return r;
}
__device__ __forceinline__ uint32_t cvt_e2m1x8(const float* y) {
  uint32_t r;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(r)
      : "f"(y[0]), "f"(y[1]), "f"(y[2]), "f"(y[3]), "f"(y[4]), "f"(y[5]), "f"(y[6]), "f"(y[7]));
  return r;
}
// The reference's E2M1 rule as a value the hardware conversion rounds to the right code (see fp4_snap_ref for the rule):
// from 1 up the conversion agrees except where it would round up into the next binade (mantissa of .75 and more), so that
// mantissa bit is dropped; below 1 the answer is .5 iff |y| > .125.
__device__ __forceinline__ float fp4_snap_fast(float y) {
  const uint32_t u = __float_as_uint(y);
  const float z = __uint_as_float(u & ~((u >> 1) & 0x00200000u));
  const float h = __uint_as_float((u & 0x80000000u) | (fabsf(y) > 0.125f ? 0x3f000000u : 0u));
  return fabsf(y) >= 1.0f ? z : h;
}

// E2M1 codes of 16 elements from their packed patterns, one code per byte in element order; kb: exponent field of the x whose scaled
// value lies in [1, 2).  Position of |x| above y = .5 in pattern steps, bits 7.. counting binades: a class is a binade and
// whether the position inside it reaches `upper`.  Positions up to there collapse into 0 and, where y > .125, get `upper`
// added back: everything in (.125, 1) is one class.
__device__ __forceinline__ void e2m1_patterns(const uint32_t* w, int kb, const PrepThresholds& thr, uint32_t* q) {
  const int k1 = thr.k1 - (kb << 7), kn = k1 + thr.kd;
  const uint32_t c1 = __byte_perm(k1, 0, 0x1010), cn = __byte_perm(kn, 0, 0x1010);
  uint32_t u[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t t = w[j] & 0x7fff7fffu;
    const uint32_t pos = __viaddmin_s16x2_relu(t, c1, thr.cmax);
    const uint32_t n = __viaddmin_s16x2_relu(t, cn, 0x00010001u);      // 1 iff y > .125
    const uint32_t q0 = pos * 4 + n * thr.ck;
    u[j] = __viaddmin_u16x2(q0, thr.ca, q0 | 0x01fc01fcu);             // class in bits 8..10, never carried into the next binade
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t cd = __byte_perm(u[2 * j], u[2 * j + 1], 0x7531), sn = __byte_perm(w[2 * j], w[2 * j + 1], 0x7531);
    q[j] = cd | ((sn >> 4) & 0x08080808u);
  }
}
__device__ __forceinline__ void e2m1_no_minus_zero(const uint32_t* w, uint32_t* q) {      // -0 counts as positive
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if ((w[j] & 0xffffu) == 0x8000u) q[j >> 1] &= ~(0x08u << ((j & 1) * 16));
    if ((w[j] >> 16) == 0x8000u) q[j >> 1] &= ~(0x0800u << ((j & 1) * 16));
  }
}
template <typename T>
__device__ __forceinline__ void e2m1_arithmetic(const uint32_t* w, float s, float inv_scale, uint32_t* q) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    float y[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float x0, x1;
      unpack2<T>(w[4 * j + k], x0, x1);
      y[2 * k] = fp4_snap_fast(__fmaf_rn(__fmul_rn(x0, s), inv_scale, 0.0f));
      y[2 * k + 1] = fp4_snap_fast(__fmaf_rn(__fmul_rn(x1, s), inv_scale, 0.0f));
    }
    const uint32_t e = cvt_e2m1x8(y), ev = e & 0x0f0f0f0fu, od = (e >> 4) & 0x0f0f0f0fu;
    q[2 * j] = __byte_perm(ev, od, 0x5140);
    q[2 * j + 1] = __byte_perm(ev, od, 0x7362);
  }
}
// n / d for n below the bound the host checked (see div_magic), one multiplication; magic 0: an ordinary division, d = 1 apart
__device__ __forceinline__ int div_by(int n, int d, uint32_t magic) {
  return d == 1 ? n : (magic ? (int)__umulhi((uint32_t)n, magic) : n / d);
}

// Mean over the rows of a head, every column, rounded to T, in the order of col_sum_kernel: eight rows, 16 apart, of every 128 a thread,
// then the threads, then the groups of 128.  mean: 128 floats, and 16 x 128 more behind them.
template <typename T>
__device__ __forceinline__ void own_column_mean(const T* x, long long xs_l, int L, int D, float* mean) {
  float* const acc_s = mean + 128;
  const int tid = threadIdx.x, c8 = tid & 15, rg = tid >> 4;
  x += c8 * 8;
  float total = 0.0f;
  _Pragma("unroll 1") for (int first = 0; first < L; first += 128) {
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int r = first + rg + 16 * k;
      v[k] = r < L && c8 * 8 < D ? *reinterpret_cast<const uint4*>(x + (long long)r * xs_l) : make_uint4(0, 0, 0, 0);
    }
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const T* e = reinterpret_cast<const T*>(&v[k]);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += (float)e[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) acc_s[rg * 128 + c8 * 8 + j] = acc[j];
    __syncthreads();
    if (tid < 128) {
      float t = 0.0f;
#pragma unroll
      for (int g = 0; g < 16; ++g) t += acc_s[g * 128 + tid];
      total += t;
    }
  }
  if (tid < 128) {
    float lo, hi;
    unpack2<T>(pack2<T>(__fdiv_rn(total, (float)L), 0.0f), lo, hi);
    mean[tid] = lo;
  }
}

// One tile of 128 rows (depth 128 and more) or 256 rows (depth 64) of one (batch, head).  A thread owns runs of 16 elements, two
// neighbouring lanes one 32-element block.  All loads of the CTA go out before any arithmetic, held as they arrived;
// scale codes are gathered with shuffles and stored a row at a time, so that no thread waits for another.  (Persistent
// CTAs that copy their next tile to shared memory under the present one were slower: 172 against 141 us for 167M elements.)
// What bounds it is instruction issue, so the loop over the runs is straight-line code for blocks in the middle of the
// exponent range (24 -> 18 instructions an element with both formats, most of the difference branches; 67M elements 56.7 ->
// 46.7 us, MXFP4 alone to one code a byte 5.7 TB/s, MXFP8 alone 6.9); a warp that meets another block - all zero, near an end
// of the range, or whose maximum is so close below a power of two that log2 rounds up - fetches the run again after the
// loop and takes the general code.  MXFP4 needs more registers than four CTAs an SM leave it (spills): three.
template <typename T, bool W8, bool W4, bool E4M3, bool D64, bool OWN>
__device__ __forceinline__ void quant_rows(const PrepOperand& p, int tile, int D, float* mean) {
  constexpr bool PATTERNS = W4 && std::is_same<T, __nv_bfloat16>::value;
  constexpr int LPR = D64 ? 4 : 8;                      // 16-element runs of a row inside the tile
  constexpr int ROWS = D64 ? 256 : 128;
  constexpr int RSTEP = PREP_THREADS / LPR;             // a thread's four runs are this many rows apart
  constexpr int EMAX8 = E4M3 ? 8 : 7, EMAX4 = 3;
  const int tid = threadIdx.x;
  const int cl = (tid & (LPR - 1)) * 16, rl0 = tid / LPR;
  const int ntd = D64 ? 1 : D >> 7;
  const int ntl = (p.L + ROWS - 1) / ROWS;
  const int v0 = ntd == 1 ? tile : tile / ntd, tile_d = tile - v0 * ntd;
  const int bh = div_by(v0, ntl, p.ntl_magic), tile_l = v0 - bh * ntl;
  const int b = div_by(bh, p.H, p.h_magic), h = bh - b * p.H, c = tile_d * 128 + cl;
  const int r0 = tile_l * ROWS + rl0, n_live = p.L - r0;     // run i is inside the operand iff i * RSTEP < n_live
  const T* const x0 = reinterpret_cast<const T*>(p.x) + (long long)b * p.xs_b + (long long)h * p.xs_h + (long long)r0 * p.xs_l + c;
  const long long xstep = p.xs_l * RSTEP;
  if (OWN && p.own_sums) own_column_mean<T>(reinterpret_cast<const T*>(p.x) + (long long)b * p.xs_b + (long long)h * p.xs_h, p.xs_l, p.L, D, mean);
  uint4 raw[4][2];
  {
    const T* x = x0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      raw[i][0] = raw[i][1] = make_uint4(0, 0, 0, 0);
      if (i * RSTEP < n_live) {
        raw[i][0] = reinterpret_cast<const uint4*>(x)[0];
        raw[i][1] = reinterpret_cast<const uint4*>(x)[1];
      }
      x += xstep;
    }
  }
  const bool centred = p.part || p.mean || (OWN && p.own_sums);
  if (centred) {
    // "smooth K": k - mean over the sequence (ours/mxfp_attn_kernel.py:33-34), an elementwise op in the input dtype.  The
    // mean is assembled here from the partial column sums, in their order.
    if (!(OWN && p.own_sums) && tid < 128 && tid < D) {
      const long long col = tile_d * 128 + tid;
      if (p.mean) {
        mean[tid] = p.mean[(long long)bh * D + col];
      } else {
        // only this waits for the column sums: everything else a launch reads or writes was ready, and free, before them
        grid_dependency_wait();
        float t = 0.0f;
        const float* part = p.part + (long long)bh * p.nchunk * D + col;
        for (int ch = 0; ch < p.nchunk; ++ch) t += __ldcg(part + (long long)ch * D);
        float lo, hi;
        unpack2<T>(pack2<T>(__fdiv_rn(t, (float)p.L), 0.0f), lo, hi);
        mean[tid] = lo;
      }
    }
    __syncthreads();
  }
  // output addresses of run 0; later runs step from there
  const long long row0 = (long long)bh * p.L + r0;
  uint8_t* o8 = W8 && p.fp8_codes ? p.fp8_codes + (long long)b * p.o8_b + (long long)h * p.o8_h + (long long)r0 * p.o8_l + c : nullptr;
  uint8_t* o4 = W4 && p.fp4_unpacked ? p.fp4_unpacked + (long long)b * p.o4_b + (long long)h * p.o4_h + (long long)r0 * p.o4_l + c : nullptr;
  uint8_t* op = W4 && p.fp4_packed ? p.fp4_packed + row0 * p.p4_row + (c >> 1) : nullptr;
  const long long s8 = p.o8_l * RSTEP, s4 = p.o4_l * RSTEP, sp = p.p4_row * RSTEP;
  constexpr bool AMAX = W8 && !W4;                      // NVFP4 next to MXFP8: this pass finds the tensor's maximum for it
  [[maybe_unused]] float amax_all = 0.0f;
  const int nblk = D >> 5;
  const long long rm0 = row0 * nblk + tile_d * 4;
  // 512-byte scale tiles: row r, block k at byte (r % 32) * 16 + (r / 32) * 4 + k
  const int ntr = (p.L + 127) >> 7, tr0 = tile_l * (ROWS >> 7);
  const long long tl0 = (((long long)bh * ntr + tr0) * ntd + tile_d) * 512 + (rl0 & 31) * 16 + (rl0 >> 5) * 4;
  auto centre = [&](uint32_t* w) {
    if (centred) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float a, d;
        unpack2<T>(w[j], a, d);
        w[j] = pack2<T>(a - mean[cl + 2 * j], d - mean[cl + 2 * j + 1]);
      }
    }
  };
  // Block maximum on the patterns: without the sign their order as integers is the order of the magnitudes, and the maximum of
  // the rounded products |x| * s is the rounded product of the maximum (s > 0).  The smallest pattern as a signed number is
  // 0x8000 iff there is a -0.
  auto block_amax = [&](const uint32_t* w, uint32_t& lowest) {
    uint32_t m = 0;
    lowest = 0;
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      m = __vimax3_s16x2(m, w[j] & 0x7fff7fffu, w[j + 1] & 0x7fff7fffu);
      if (PATTERNS) lowest = __vimin3_s16x2(lowest, w[j], w[j + 1]);
    }
    m = max(m & 0xffffu, m >> 16);
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    return __fmul_rn(pattern_to_float<T>(m), p.s);
  };
  auto store_fp4 = [&](int i, const uint32_t* q) {
    if (o4) *reinterpret_cast<uint4*>(o4 + i * s4) = make_uint4(q[0], q[1], q[2], q[3]);
    if (op) {
      uint32_t pk[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {                     // bytes -> nibbles
        const uint32_t a = q[2 * k] | (q[2 * k] >> 4), d = q[2 * k + 1] | (q[2 * k + 1] >> 4);        // bytes 0 and 2 hold two codes each
        pk[k] = __byte_perm(a, d, 0x6420);
      }
      *reinterpret_cast<uint2*>(op + i * sp) = make_uint2(pk[0], pk[1]);
    }
  };
  // a row's scale codes in one word, one store per row and layout; rows beyond L and blocks beyond D hold 1.0
  auto gather = [&](uint32_t code) {
    uint32_t v = code << (((tid >> 1) & (LPR / 2 - 1)) * 8);
    v |= __shfl_xor_sync(0xffffffffu, v, 2);
    if (!D64) v |= __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
  };
  auto store_scale = [&](int i, bool live, uint8_t* st, uint8_t* rm, uint32_t v) {
    if (st && (D64 ? tr0 + (i >> 1) : tr0) < ntr) *reinterpret_cast<uint32_t*>(st + tl0 + (D64 ? (i >> 1) * 512 + (i & 1) * 8 : i * 4)) = D64 ? v | 0x7f7f0000u : v;
    if (rm && live) {
      if (D64) *reinterpret_cast<uint16_t*>(rm + rm0 + i * (RSTEP * 2)) = (uint16_t)v;
      else *reinterpret_cast<uint32_t*>(rm + rm0 + (long long)i * RSTEP * nblk) = v;
    }
  };
  // With |es| <= 16 (mild) and the exponent field of the block's maximum in 48 .. 230 no scale code is clamped, s / scale and the
  // products that matter are normal, and every code boundary is the pattern of a normal number.
  const bool fast_operand = p.thr.mild && (!PATTERNS || p.thr.valid);
  uint32_t todo = 0, exps[4];                           // runs that need the general code; exponent fields of a row's blocks
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool live = i * RSTEP < n_live;
    uint32_t w[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
    centre(w);
    uint32_t lowest;
    const float amax = block_amax(w, lowest);
    if (AMAX) amax_all = fmaxf(amax_all, live ? amax : 0.0f);
    const uint32_t ab = __float_as_uint(amax), ef = ab >> 23;
    const bool plain = !live || (fast_operand && ef - 48u <= 182u && (ab & 0x007fffffu) < 0x007fff00u);
    if (!__all_sync(0xffffffffu, plain)) {
      todo |= 1u << i;
      exps[i] = 0;
      continue;
    }
    if (W8) {
      const float f = p.s * __uint_as_float((254u + EMAX8 - ef) << 23);      // s / scale
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a0, a1, a2, a3;
        unpack2<T>(w[2 * j], a0, a1);
        unpack2<T>(w[2 * j + 1], a2, a3);
        mul2(a0, a1, f);
        mul2(a2, a3, f);
        o[j] = cvt_fp8x4<E4M3>(a0, a1, a2, a3);
      }
      if (o8 && live) *reinterpret_cast<uint4*>(o8 + i * s8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    if (W4) {
      uint32_t q[4];
      if (PATTERNS) {
        e2m1_patterns(w, (int)ef - EMAX4 - p.thr.es, p.thr, q);
        if ((lowest & 0xffffu) == 0x8000u || (lowest >> 16) == 0x8000u) e2m1_no_minus_zero(w, q);
      } else {
        e2m1_arithmetic<T>(w, p.s, __uint_as_float((254u + EMAX4 - ef) << 23), q);
      }
      if (live) store_fp4(i, q);
    }
    exps[i] = gather(live ? ef : 0u);
  }
  // scale code = exponent field - emax: no byte borrows from the next (rows whose run is still to do are written again below)
  if ((tid & (LPR - 1)) == 0) {
    constexpr uint32_t ONES = D64 ? 0x0101u : 0x01010101u;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (!(f ? W4 : W8)) continue;
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = i * RSTEP < n_live ? exps[i] - ONES * (f ? EMAX4 : EMAX8) : 0x7f7f7f7fu;
      uint8_t* st = f ? p.sf4_tiled : p.sf8_tiled;
      uint8_t* rm = f ? p.sc4_rows : p.sc8_rows;
      if (st && !D64) *reinterpret_cast<uint4*>(st + tl0) = make_uint4(v[0], v[1], v[2], v[3]);      // rows 32 apart lie side by side
      if (rm || D64) {
#pragma unroll
        for (int i = 0; i < 4; ++i) store_scale(i, i * RSTEP < n_live, D64 ? st : nullptr, rm, v[i]);
      }
    }
  }
#pragma unroll 1
  for (; todo; todo &= todo - 1) {
    const int i = __ffs(todo) - 1;
    const bool live = i * RSTEP < n_live;
    uint4 r[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    if (live) {
      r[0] = reinterpret_cast<const uint4*>(x0 + i * xstep)[0];
      r[1] = reinterpret_cast<const uint4*>(x0 + i * xstep)[1];
    }
    uint32_t w[8] = {r[0].x, r[0].y, r[0].z, r[0].w, r[1].x, r[1].y, r[1].z, r[1].w};
    centre(w);
    uint32_t lowest;
    const float amax = block_amax(w, lowest);
    uint32_t code8 = 127, code4 = 127;
    if (live) {
      if (W8) {
        const BlockScale b8 = mx_block_scale(amax, EMAX8);
        code8 = b8.code;
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float a0, a1, a2, a3;
          unpack2<T>(w[2 * j], a0, a1);
          unpack2<T>(w[2 * j + 1], a2, a3);
          mul2(a0, a1, p.s);
          mul2(a2, a3, p.s);
          mul2(a0, a1, b8.inv_scale);
          mul2(a2, a3, b8.inv_scale);
          o[j] = b8.zero ? 0u : cvt_fp8x4<E4M3>(a0, a1, a2, a3);      // the reference stores the NaN pattern of 0/0 there
        }
        if (o8) *reinterpret_cast<uint4*>(o8 + i * s8) = make_uint4(o[0], o[1], o[2], o[3]);
      }
      if (W4) {
        const BlockScale b4 = mx_block_scale(amax, EMAX4);
        code4 = b4.code;
        uint32_t q[4];
        const int base = (int)b4.code - p.thr.es;
        if (b4.zero) {
          q[0] = q[1] = q[2] = q[3] = 0x08080808u;      // 0/0 in the reference: sign 1, exponent 0, mantissa 0
        } else if (PATTERNS && p.thr.valid && base >= 4 && base <= 253) {
          e2m1_patterns(w, base, p.thr, q);
          e2m1_no_minus_zero(w, q);
        } else {
          e2m1_arithmetic<T>(w, p.s, b4.inv_scale, q);
        }
        store_fp4(i, q);
      }
    }
    const uint32_t v8 = W8 ? gather(code8) : 0u, v4 = W4 ? gather(code4) : 0u;
    if ((tid & (LPR - 1)) == 0) {
      if (W8) store_scale(i, live, p.sf8_tiled, p.sc8_rows, v8);
      if (W4) store_scale(i, live, p.sf4_tiled, p.sc4_rows, v4);
    }
  }
  if (AMAX && p.amax) {                                 // few warps find a new maximum: the others only look at the word
    const unsigned a = __reduce_max_sync(0xffffffffu, __float_as_uint(amax_all));
    if ((tid & 31) == 0 && a > __ldcg(p.amax)) atomicMax(p.amax, a);
  }
}

// 128 keys of one (batch, head) of V [keys, D], transposed through shared memory: fp16 V^T, or MXFP8 / MXFP4 V^T with 32-key
// blocks along the sequence (round to nearest even, shared exponent floor(log2(amax)) - emax).  ldmatrix.trans hands a lane two
// keys of one depth element; its row addresses are chosen so that four neighbouring lanes hold 16 consecutive keys each of
// the same depth element.  16-byte pieces of a key's row are swizzled by the key bits those addresses differ in: no
// bank conflicts on either side.
template <typename T, bool E4M3>
__device__ __forceinline__ void v_tile(const PrepV& p, int cta, int D, uint8_t* smem) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int ntk = p.pitch >> 7;
  const int bh = cta / ntk, kt = cta - bh * ntk;
  const int b = bh / p.H, h = bh - b * p.H;
  const int key0 = kt * 128;
  const uint8_t* src = reinterpret_cast<const uint8_t*>(p.v) + ((long long)b * p.vs_b + (long long)h * p.vs_h) * 2;
  const int vlog = D == 64 ? 3 : 4;                     // 16-byte pieces of a key's row: 8 or 16
  uint4 ld[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int i = tid + j * PREP_THREADS, key = i >> vlog, vc = i & ((1 << vlog) - 1);
    ld[j] = make_uint4(0, 0, 0, 0);
    if (key < 128 && key0 + key < p.Skv) ld[j] = reinterpret_cast<const uint4*>(src + (long long)(key0 + key) * p.vs_l * 2)[vc];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int i = tid + j * PREP_THREADS, key = i >> vlog, vc = i & ((1 << vlog) - 1);
    const int sw = (key & 1) | (((key >> 4) & 3) << 1);
    if (key < 128) *reinterpret_cast<uint4*>(smem + (key << (vlog + 4)) + ((vc ^ sw) << 4)) = ld[j];
  }
  __shared__ __align__(16) uint8_t sf[2][512];
  for (int i = tid; i < 256; i += PREP_THREADS) reinterpret_cast<uint32_t*>(&sf[0][0])[i] = 0x7f7f7f7fu;
  __syncthreads();
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int units = D >> 2;                             // (group of 8 depth elements) x (64 keys)
  for (int u = tid >> 5; u < units; u += PREP_THREADS / 32) {
    const int half = u & 1, dg = u >> 1;
    uint32_t w[8];                                      // keys half * 64 + (lane & 3) * 16 + 0..15 of depth element d
#pragma unroll
    for (int x4 = 0; x4 < 2; ++x4) {
      const int mtx = x4 * 4 + (lane >> 3), r = lane & 7;       // this lane's address: row r of matrix mtx
      const int key = half * 64 + 16 * (r >> 1) + 2 * mtx + (r & 1);
      const int sw = (key & 1) | (((key >> 4) & 3) << 1);
      const uint32_t a = sbase + (key << (vlog + 4)) + ((dg ^ sw) << 4);
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(w[4 * x4]), "=r"(w[4 * x4 + 1]), "=r"(w[4 * x4 + 2]), "=r"(w[4 * x4 + 3]) : "r"(a));
    }
    const int d = dg * 8 + (lane >> 2);
    const long long row = (long long)bh * D + d;
    const int key = key0 + half * 64 + (lane & 3) * 16;
    if (p.vt16) {
      if (!std::is_same<T, __half>::value) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float lo, hi;
          unpack2<T>(w[k], lo, hi);
          w[k] = pack2<__half>(lo, hi);
        }
      }
      uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.vt16) + row * p.pitch + key);
      o[0] = make_uint4(w[0], w[1], w[2], w[3]);
      o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    } else {
      uint32_t m = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) m = __vmaxu2(m, w[k] & 0x7fff7fffu);
      m = max(m & 0xffffu, m >> 16);
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));           // two lanes share a 32-key block
      const float amax = pattern_to_float<T>(m);
      const int sf_off = (d & 31) * 16 + (d >> 5) * 4 + half * 2 + ((lane >> 1) & 1);
      float y[16];
#pragma unroll
      for (int k = 0; k < 8; ++k) unpack2<T>(w[k], y[2 * k], y[2 * k + 1]);
      if (p.vt8) {
        const BlockScale bs = mx_block_scale(amax, E4M3 ? 8 : 7);
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          o[k] = bs.zero ? 0u : cvt_fp8x4<E4M3>(y[4 * k] * bs.inv_scale, y[4 * k + 1] * bs.inv_scale, y[4 * k + 2] * bs.inv_scale, y[4 * k + 3] * bs.inv_scale);
        *reinterpret_cast<uint4*>(p.vt8 + row * p.pitch + key) = make_uint4(o[0], o[1], o[2], o[3]);
        if ((lane & 1) == 0) sf[0][sf_off] = bs.code;
      }
      if (p.vt4) {
        const BlockScale bs = mx_block_scale(amax, 2);
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] = bs.zero ? 0.0f : y[k] * bs.inv_scale;
        *reinterpret_cast<uint2*>(p.vt4 + row * (p.pitch >> 1) + (key >> 1)) = make_uint2(cvt_e2m1x8(y), cvt_e2m1x8(y + 8));
        if ((lane & 1) == 0) sf[1][sf_off] = bs.code;
      }
    }
  }
  if (p.vt16) return;
  __syncthreads();
  const long long tile = (long long)bh * ntk + kt;
  if (tid < 32) {
    if (p.vt8) reinterpret_cast<uint4*>(p.v8_sf + tile * 512)[tid] = reinterpret_cast<const uint4*>(sf[0])[tid];
  } else if (tid < 64) {
    if (p.vt4) reinterpret_cast<uint4*>(p.v4_sf + tile * 512)[tid - 32] = reinterpret_cast<const uint4*>(sf[1])[tid - 32];
  }
}

// OWN: K's CTAs may add up the columns themselves; an instance of its own, because it costs the others 1 - 2 %
template <typename T, bool W8, bool W4, bool E4M3, bool D64, bool OWN>
__global__ void __launch_bounds__(PREP_THREADS, W4 ? 3 : 4) prep_kernel(const __grid_constant__ PrepCall p) {
  extern __shared__ __align__(128) uint8_t prep_smem[];
  int cta = blockIdx.x;
  // Behind the column sums only what reads them waits: this kernel starts once they have seen the end of everything before them, and
  // some CTA of K waits for them in any case, so that what follows finds them complete.
  if (!p.after_sums) grid_dependency_wait();
  grid_dependents_go();
  if (cta == 0 && threadIdx.x < 2) {
    // words the launches behind this one expect to find zero
    int* z = threadIdx.x ? p.zero1 : p.zero0;
    if (z) *z = 0;
  }
  if (cta < p.v.ctas) {
    v_tile<T, E4M3>(p.v, cta, p.D, prep_smem);
    return;
  }
  cta -= p.v.ctas;
  const int which = cta >= p.op[0].ctas;
  if (which) cta -= p.op[0].ctas;
  quant_rows<T, W8, W4, E4M3, D64, OWN>(p.op[which], cta, p.D, reinterpret_cast<float*>(prep_smem));
}

template <typename T>
int launch_prep(const PrepCall& p, bool w8, bool w4, bool e4m3, int grid, size_t smem, cudaStream_t st) {
  const bool dep = p.after_sums || overlaps_previous(st);
#define MPSA_PREP(A, B, C)                                                                                                    \
  do {                                                                                                      \
    if (!C && (p.op[0].own_sums || p.op[1].own_sums)) {                                                                   \
      if (p.D == 64) launch_dependent(prep_kernel<T, A, B, false, true, true>, dim3(grid), PREP_THREADS, smem, st, dep, p);  \
      else launch_dependent(prep_kernel<T, A, B, false, false, true>, dim3(grid), PREP_THREADS, smem, st, dep, p);         \
    } else if (p.D == 64) launch_dependent(prep_kernel<T, A, B, C, true, false>, dim3(grid), PREP_THREADS, smem, st, dep, p);  \
    else launch_dependent(prep_kernel<T, A, B, C, false, false>, dim3(grid), PREP_THREADS, smem, st, dep, p);         \
  } while (0)
  if (w8 && w4) { if (e4m3) MPSA_PREP(true, true, true); else MPSA_PREP(true, true, false); }
  else if (w4) { if (e4m3) MPSA_PREP(false, true, true); else MPSA_PREP(false, true, false); }
  else { if (e4m3) MPSA_PREP(true, false, true); else MPSA_PREP(true, false, false); }
#undef MPSA_PREP
  return check_launch("prep");
}

}  // namespace

PrepThresholds prep_thresholds(float s) {
  PrepThresholds t;
  if (!(s > 0.0f) || !std::isfinite(s)) return t;
  int e;
  const float ms = 2.0f * std::frexp(s, &e);            // s = ms * 2^(e - 1), ms in [1, 2)
  t.es = e - 1;
  t.mild = t.es >= -16 && t.es <= 16;
  // y = fl(x * s): the first of the 128 mantissas whose product reaches the next binade
  // (products of neighbouring mantissas differ by ms / 128, far more than a rounding: everything here is strictly monotone)
  auto lowest = [](int n, auto reached) {               // smallest i in [0, n] with reached(i), n if none
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (reached(mid)) hi = mid; else lo = mid + 1;
    }
    return lo;
  };
  const int first = lowest(128, [&](int m) { return (1.0f + (float)m / 128.0f) * ms >= 2.0f; });
  // y's mantissa at position k = 0 .. 127 of its own binade
  auto mant = [&](int k) {
    const int m = first + k;                            // x mantissas first .. 127, then 0 .. first - 1 of the next binade
    return m < 128 ? (1.0f + (float)m / 128.0f) * ms * 0.5f : (1.0f + (float)(m - 128) / 128.0f) * ms;
  };
  const int shift = 128 - first;                        // added to a pattern, bits 7.. count the binades of y
  const int strict = mant(0) == 1.0f;                   // position 0 of a binade is a power of two exactly
  t.upper = lowest(128, [&](int k) { return mant(k) > 1.25f; });
  t.valid = t.upper <= 64;
  t.k1 = shift + 0x80 - t.upper;
  t.kd = t.upper - 0x80 + 0x180 - strict + 1;
  auto lanes = [](int v) { return (uint32_t)(v & 0xffff) * 0x10001u; };
  t.cmax = lanes(0x1ff - t.upper);
  t.ca = lanes((0x40 - t.upper) * 4);
  t.ck = (uint32_t)t.upper * 4;
  return t;
}

bool prep_operand_ok(const PrepOperand& p, int D) {
  auto al = [](const void* q, int n) { return (uintptr_t)q % n == 0; };
  return (D == 64 || (D > 0 && D % 128 == 0)) && p.s > 0.0f && std::isfinite(p.s) && al(p.x, 16) && (p.xs_b * 2) % 16 == 0 &&
         (p.xs_h * 2) % 16 == 0 && (p.xs_l * 2) % 16 == 0;
}

// n / d == mulhi(n, magic) for 0 <= n < bound: magic = ceil(2^32 / d) is too large by less than d / 2^32 of a unit, which
// does no harm while n d < 2^32 (d = 1 has no such magic); 0 otherwise
static uint32_t div_magic(int d, long long bound) {
  return d > 1 && bound * d < (1ll << 32) ? (uint32_t)(((1ull << 32) + d - 1) / d) : 0;
}

int prep_launch(PrepCall& p, int in_dtype, bool w8, bool w4, int fp8_fmt, cudaStream_t st) {
  long long ctas = 0;
  const int rows_cta = p.D == 64 ? 256 : 128, ntd = p.D == 64 ? 1 : p.D / 128;
  for (PrepOperand& o : p.op) {
    o.ctas = 0;
    if (!o.x) continue;
    o.thr = prep_thresholds(o.s);
    o.ntl_magic = div_magic((o.L + rows_cta - 1) / rows_cta, (long long)o.B * o.H * ((o.L + rows_cta - 1) / rows_cta));
    o.h_magic = div_magic(o.H, (long long)o.B * o.H);
    const long long n = (long long)o.B * o.H * ((o.L + rows_cta - 1) / rows_cta) * ntd;
    ctas += n;
    if (ctas > 0x3fffffff) return set_error(MPSA_ERR_UNSUPPORTED, "prep: operand too large");
    o.ctas = (int)n;
  }
  p.v.ctas = 0;
  size_t smem = p.op[0].own_sums || p.op[1].own_sums ? 512 + 16 * 128 * 4 : 512;
  if (p.v.v) {
    const long long n = (long long)p.v.B * p.v.H * (p.v.pitch >> 7);
    ctas += n;
    p.v.ctas = (int)n;
    smem = PREP_V_SMEM;
  }
  if (ctas <= 0 || ctas > 0x7fffffff) return set_error(MPSA_ERR_UNSUPPORTED, "prep: bad number of tiles");
  const bool e4m3 = fp8_fmt == FMT_FP8_E4M3;
  if (in_dtype == 0) return launch_prep<__nv_bfloat16>(p, w8, w4, e4m3, (int)ctas, smem, st);
  return launch_prep<__half>(p, w8, w4, e4m3, (int)ctas, smem, st);
}

}  // namespace mpsa
