// Operand preparation in one launch (prep.cu): the parameter blocks its callers fill in.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mpsa {

// How the E2M1 classes of y = x * s lie on the 16-bit patterns of bf16 x > 0 (see prep.cu).
struct PrepThresholds {
  bool valid = false;
  bool mild = false;      // s is far from the ends of the exponent range
  int es = 0;             // s = ms * 2^es
  int upper = 0;          // first position of a binade whose y exceeds 1.25
  int k1 = 0, kd = 0;     // offsets of the class positions and of the .125 boundary
  uint32_t cmax = 0, ca = 0, ck = 0;   // packed constants of the classification
};

// One operand [B,H,L,D] quantised along D; a null output is not produced.
struct PrepOperand {
  const void* x = nullptr;                             // null: no operand
  int B = 0, H = 0, L = 0;
  long long xs_b = 0, xs_h = 0, xs_l = 0;              // input strides in elements
  float s = 1.0f;                                      // multiplied in before quantisation
  const float* part = nullptr; int nchunk = 0;         // partial column sums [B*H, nchunk, D] of the mean to subtract,
  const float* mean = nullptr;                         // or that mean itself [B*H, D],
  bool own_sums = false;                               // or every CTA adds up its head's columns itself (prep_own_sums; D <= 128, E5M2)
  uint8_t* fp8_codes = nullptr; long long o8_b = 0, o8_h = 0, o8_l = 0;
  uint8_t* fp4_unpacked = nullptr; long long o4_b = 0, o4_h = 0, o4_l = 0;
  uint8_t* fp4_packed = nullptr; long long p4_row = 0; // [B,H,L] rows of p4_row bytes
  uint8_t* sc8_rows = nullptr; uint8_t* sc4_rows = nullptr;       // [B,H,L,D/32]
  uint8_t* sf8_tiled = nullptr; uint8_t* sf4_tiled = nullptr;     // [B,H,ceil(L/128),ceil(D/128),512]
  unsigned* amax = nullptr;                            // optional word, zero before: bits of the largest |x * s|
  PrepThresholds thr;                                  // filled in by prep_launch, like what follows
  uint32_t ntl_magic = 0, h_magic = 0;                 // division by row tiles and by heads
  int ctas = 0;
};

// V [B,H,Skv,D] transposed: vt16, or vt8 / vt4 with their scale tiles.
struct PrepV {
  const void* v = nullptr;                             // null: no V
  int B = 0, H = 0, Skv = 0, pitch = 0;                // pitch: keys per V^T row, a multiple of 128
  long long vs_b = 0, vs_h = 0, vs_l = 0;
  void* vt16 = nullptr;
  uint8_t *vt8 = nullptr, *v8_sf = nullptr, *vt4 = nullptr, *v4_sf = nullptr;
  int ctas = 0;
};

struct PrepCall {
  PrepOperand op[2];
  PrepV v;
  int D = 0;
  int *zero0 = nullptr, *zero1 = nullptr;              // words set to zero on the way
  bool after_sums = false;                             // the kernel before this one on the stream is col_sums'
};

// Whether the CTAs of K add up the columns of their head themselves, each the whole head (up to PREP_OWN_SUMS rows), instead of waiting
// for a launch that does it once.  That saves the launch; it costs every CTA of K a pass over its head, in a second round of CTAs where
// the chip does not hold all of them at once.  GPU time of a call, MXFP4 scores, depth 128, launch -> own: 16 heads of 333 rows 16.8 ->
// 14.6 us, 64 heads of 333 (192 CTAs of K) 26.2 -> 25.1, 48 heads of 512 (192) 27.3 -> 26.9; against it 64 heads of 512 (256) 29.0 -> 31.0,
// 128 of 512 51.3 -> 55.1, 96 of 333 (288) 30.4 -> 31.5.  Up to two tiles it pays whatever the heads (256 heads of 256 49.0 -> 45.4; depth
// 64, where a tile has 256 rows, 64 heads of 512 23.7 -> 23.1), but for 96 heads of 333 - 384 rows of depth 64 (25.2 -> 25.9).
constexpr int PREP_OWN_SUMS = 512, PREP_OWN_CTAS = 200;
inline bool prep_own_sums(long long heads, int L, int D) {
  const int rows = D == 64 ? 256 : 128, tiles = (L + rows - 1) / rows;
  return L <= PREP_OWN_SUMS && (tiles <= 2 || heads * tiles <= PREP_OWN_CTAS);
}

PrepThresholds prep_thresholds(float s);
bool prep_operand_ok(const PrepOperand& p, int D);     // alignment, depth and scale the kernel can take
// in_dtype 0 bf16, 1 fp16 (all inputs); w8 / w4: formats of op[]
int prep_launch(PrepCall& p, int in_dtype, bool w8, bool w4, int fp8_fmt, cudaStream_t st);

}  // namespace mpsa
