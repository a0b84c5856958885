// Fused diagonal-tiled mixed-precision attention forward for sm_100a.
//
// Counterpart of block_scaled_batched_attn_kernel (ours/mxfp_attn_kernel.py:103-359) with the parts
// the reference leaves out: causal masking and GQA (taken from its INT8 sibling,
// ours/online_routing.py:68-77, :113-118, :160) and a per-tile precision map.
//
// Persistent CTAs, one per SM.  A work item is a 128-row query tile of one (batch, q-head); the CTA walks the 128-key
// tiles the precision map enables for it:
//   S = Q.K^T   tcgen05.mma block-scaled: kind::mxf8f6f4 (MXFP8 x MXFP8, 4 x K=32) on FP8 tiles,
//               kind::mxf4 / mxf4nvf4 (2 x K=64) on FP4 tiles; Q is resident in shared memory in both formats, K tiles
//               arrive by TMA in the format the map asks for; scale tiles go to TMEM with tcgen05.cp.  The softmax
//               scale * log2(e) is already folded into Q by the quantizer (ours/quant_mxint8.py:494), so S is in the
//               log2 domain.
//   softmax     four threads per query row (two column halves of a tile x two warpgroups that take the tiles in turn)
//               compute P = exp2(S - m) against a FIXED row reference m and keep partial row sums and row maxima.
//   O += P.V    pv_mode 0 (the reference's precision): P in fp16, kind::f16 with V^T in fp16, fp32 accumulation (the
//               reference accumulates each tile in fp16 first, ours/mxfp_attn_kernel.py:340).  pv_mode 1: P is
//               re-quantised to the tile's format (one E8M0 scale per 32 keys) and multiplied with V quantised along
//               the sequence.  P comes from TMEM columns of its own, so that Q.K^T of tile t + 2 never waits for P.V.
//
// The row reference.  Quantised P.V: block-scaled P carries its magnitude in E8M0 codes, and with an integral reference
// the element codes do not depend on it at all; m = 20 serves every row whose maximum M lies in [-44, 84] (P, O and the row
// sums then stay within 2^-64 .. 2^64).  Nothing in a tile depends on the running maximum, and no two threads of a row
// have to agree on anything before the end of the item.  An item with a row outside the window is done again a little
// later, with the row maxima that the first pass found as references.
// fp16 P.V: m starts as the row maximum of the item's first tile, so that it is never above the row's maximum and P keeps
// its 11 bits down to 2^-14 of the largest at least.  It serves scores up to m + 15 (P at most 2^15).  A half tile that goes
// beyond raises m to its own maximum and scales O and the sums, all of it 2^-15 or less from then on.  The half tiles of a row
// decide in their order, each before it hands over its P, so P.V, which takes them in the same order, finds P and O at one
// reference.  (With references rounded down to whole octaves no largest P was exactly 1: 5 % more error with N(0,1) keys.)
//
// Roles: warp 0 loads Q and V, warp 1 loads K and issues Q.K^T, warp 2 issues P.V, warp 3 hands out work items, builds their visit
// lists (the non-skipped cells of the map row) and routes, warps 4.. softmax and epilogue (a warp reaches the TMEM lane
// quarter warp % 4).  Items reach the other roles through a ring of slots, an item ahead; rings and their phases run on
// across items, so an item's Q, K and V loads and its first tiles happen under the previous item's last ones.
//
// What bounds it: instruction issue and latency together, then the exponentials.  A tile takes about 1200 - 1450 cycles; without any
// exponential (timing only) it would still take 0.88 of that, without all of the softmax arithmetic 0.7.  ex2 runs at 16 per clock
// and SM, 1024 cycles for the 16384 scores of a tile; the four softmax warps of a quarter issue some 700 instructions a tile and
// the service warp beside them 130 - 180 more, on a scheduler that has four or five warps to choose from.  Hence:
//  - no branch inside a tile's arithmetic: the instructions on its two sides are scheduled apart, and one that is never taken costs
//    2 %.  Masks and shifts are applied to S in tensor memory beforehand (adjust_scores).
//  - service threads of few instructions, on warps of their own: one thread that requested K and V was busy for 1000 - 1100 of
//    every 1400 cycles and held the kernel up (12 heads of 7803 tokens 231 -> 224 us with K moved to the Q.K^T issuer).
#include "api_internal.h"
#include "common.cuh"
#include "prep.h"
#include "tma_host.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <type_traits>

namespace mpsa {

// ---- organisation of a CTA ------------------------------------------------------------------------------
constexpr int ATT_BM = 128, ATT_BN = 128, ATT_DQK = 128;
constexpr int ATT_KSTAGES = 4;                        // K ring
constexpr int ATT_VSLOTS = 4;                         // V ring, slots of 16 KB: a quantised V^T tile or a 64-key half of an fp16 one
constexpr int ATT_SERVICE_WARPS = 4;                  // 0 loads of Q and V, 1 loads of K and Q.K^T, 2 P.V, 3 visit lists and router
constexpr int ATT_SM_WARPS = 16;                      // softmax: 2 warpgroups (tiles in turn) x 2 column halves x 4 row quarters
constexpr int ATT_THREADS = 32 * (ATT_SERVICE_WARPS + ATT_SM_WARPS);
constexpr int ATT_Q8_BYTES = ATT_BM * 128, ATT_Q4_BYTES = ATT_BM * 64;
constexpr int ATT_Q_BYTES = ATT_Q8_BYTES + ATT_Q4_BYTES;
constexpr int ATT_K_BYTES = ATT_BN * 128;             // slot sized for the FP8 tile; FP4 uses half
constexpr int ATT_V_BYTES = 128 * ATT_BN * 2;         // V^T tile, up to D=128 rows of 128 fp16
constexpr int ATT_MAX_SLOTS = 3;                                          // work items whose visit lists are in shared memory at a time
constexpr int ATT_OFF_Q = 0;                                              // [2] Q8 tile, Q4 tile
constexpr int ATT_OFF_K = ATT_OFF_Q + 2 * ATT_Q_BYTES;
constexpr int ATT_OFF_V = ATT_OFF_K + ATT_KSTAGES * ATT_K_BYTES;
constexpr int ATT_OFF_SFQ = ATT_OFF_V + 2 * ATT_V_BYTES;                  // [2] Q8 scale tile (512 B), Q4 scale tiles (1024 B: NVFP4 has two)
constexpr int ATT_OFF_SFK = ATT_OFF_SFQ + 2 * 1536;                       // [KSTAGES] 1024 B
constexpr int ATT_OFF_SFP = ATT_OFF_SFK + ATT_KSTAGES * 1024;             // P scale tiles [2], V scale tiles [VSLOTS]
constexpr int ATT_OFF_XROW = ATT_OFF_SFP + (2 + ATT_VSLOTS) * 512;    // float [2][2][4][128]: row sums and row maxima of the four threads of a row
constexpr int ATT_OFF_RMAX = ATT_OFF_XROW + 2 * 2 * 4 * 128 * 4;          // fp16 P.V: float [2][128], first-tile maxima
constexpr int ATT_OFF_MROW = ATT_OFF_RMAX + 2 * 128 * 4;                  // float [128]: present row reference (fp16 P.V)
constexpr int ATT_OFF_MSLOT = ATT_OFF_MROW + 128 * 4;                     // float [MAX_SLOTS][128]: row maxima of the item that was in the slot
constexpr int ATT_OFF_BAR = ATT_OFF_MSLOT + ATT_MAX_SLOTS * 128 * 4;
// barriers the softmax threads use in their tile loop, by number
constexpr int ATT_B_SFULL = 32;
constexpr int ATT_B_SFREE = ATT_B_SFULL + 2, ATT_B_PREADY = ATT_B_SFULL + 4, ATT_B_PVDONE = ATT_B_SFULL + 8, ATT_B_ST = ATT_B_SFULL + 14;
constexpr int ATT_B_RBAR = ATT_B_SFULL + 30;
constexpr int ATT_NUM_BARS = ATT_B_RBAR + 16 + 2;
static_assert(ATT_B_PVDONE % 4 == 0, "the four are one another's neighbours by exclusive or of their addresses");
static_assert(4 + 3 * ATT_MAX_SLOTS + ATT_KSTAGES + 2 * ATT_VSLOTS <= ATT_B_SFULL, "barrier numbers overlap");
constexpr int ATT_BAR_BYTES = 1024;                                       // barriers, TMEM slot, router words, item slots
static_assert(ATT_NUM_BARS * 8 + 32 + ATT_MAX_SLOTS * 36 <= ATT_BAR_BYTES, "the barrier block does not fit its share of shared memory");
constexpr int ATT_OFF_EXTRA = ATT_OFF_BAR + ATT_BAR_BYTES;                // fp16 P.V: float [2][4][128], the references of XROW's sums;
constexpr int ATT_EXTRA_BYTES = 2 * 4 * 128 * 4;                          // router: float [4 tiles][2][128], slice maxima
constexpr int ATT_OFF_LIST = ATT_OFF_BAR + ATT_BAR_BYTES;                 // visit lists: n_lists x list_cap uint16 (ATT_EXTRA_BYTES further on where they are used)
constexpr int ATT_MAX_KTILES = 8192;                                      // longest row of the precision map (1M keys)
constexpr int ATT_SMEM_MAX = 232448;
static_assert(ATT_OFF_LIST + ATT_EXTRA_BYTES + ATT_MAX_KTILES * 2 + 1024 <= ATT_SMEM_MAX, "more shared memory than a CTA can have");
// TMEM columns: S0 [0,128) S1 [128,256) O [256,384), scale tiles from 384, P up to 512
constexpr uint32_t ATT_TMEM_COLS = 512;
constexpr uint32_t ATT_COL_S = 0, ATT_COL_O = 256;
constexpr uint32_t ATT_COL_SFQ8 = 384, ATT_COL_SFQ4 = 388;       // 4 columns; 8 columns (NVFP4 uses all 8)
constexpr uint32_t ATT_COL_SFK = 396;                             // two sets of 8
constexpr uint32_t ATT_COL_SFP = 412, ATT_COL_SFV = 420;          // quantised P.V: two sets of 4 each
constexpr uint32_t ATT_COL_P = 448;                               // quantised P: 2 buffers of 32 columns (a tile each)
constexpr uint32_t ATT_COL_P16 = 416;                             // fp16 P: 3 buffers of 32 columns (a 64-key half each)

constexpr int TILE_SKIP = 0, TILE_FP8 = 1, TILE_FP4 = 2;
constexpr uint32_t ENTRY_F8 = 0x8000, ENTRY_MASK = 0x4000, ENTRY_TILE = 0x3fff;   // visit list entries

// Exponentials of a 32-key block that run on the FMA pipe (ex2_poly2).  MXFP4 tiles with quantised P.V, exponentials before the
// block's maximum (LATE): 512 queries of 32K 179 us with 0, 173 with 2, 164 with 4, 170 with 6.  Where they wait for the maximum:
// routed causal 8K 400 us with 0, 397 with 2, 401 with 4.  fp16 P, with 0 / 2 / 4 / 6, back to back under the power limit: NVFP4 video
// 15.49 / 15.38 / 15.55 / 15.82 ms, 32 heads of 8192 884 / 877 / 883 / 896 us; in bursts 8 heads of 8192 264 / 259 / 264 / 261 us.
constexpr int ATT_POLY_LATE = 4, ATT_POLY_EARLY = 2, ATT_POLY_F16 = 2;
constexpr int ATT_F16_EARLY = 4;                      // fp16 P.V: exponentials of the second block that hide the vote on the reference
constexpr int SPLIT_MIN_RUN = 8;                      // tiles of a run at least
constexpr int SPLIT_GAIN = 12;                        // tiles (of 0.7 us) that dividing the keys must save on the busiest CTA
constexpr int SPLIT_MIN_OWN = 4, SPLIT_GAIN_OWN = 7;  // the same two where every part has a CTA to itself
constexpr float ATT_REF_Q = 20.0f;                    // quantised P.V: the row reference, and the window of row maxima it serves
constexpr float ATT_WIN_LO_Q = -64.0f, ATT_WIN_HI_Q = 64.0f;
constexpr float ATT_TOP_F16 = 15.0f;                  // fp16 P.V: scores up to this far above the row reference need no new one (P at most 2^15)
constexpr float ATT_NO_REF = -3e38f;                  // fp16 P.V: reference of a row that has seen no key yet

// Numbering of the items, r counting query tiles from the last.  Causal: heaviest query tile first, item = r * heads + head.
// Otherwise all tiles weigh the same and one head comes after the other: the 148 items that run at a time then share the keys and
// values of a few heads, which stay in L2 (32 heads of 8192 keys: 1.43 -> 0.14 GB from HBM for 0.1 GB of operands,
// and under the power limit 1010 -> 883 us; NVFP4 video 17.7 -> 15.0 ms).
// Division of the keys.  The first n_whole are done by one CTA each; the tiles of the others, laid end to end, are cut into runs
// of run_tiles, one CTA each, so that a grid with fewer items than SMs, or with a last wave that is nearly empty, still
// fills the chip.  An item that several runs share gets its result from attn_combine_kernel.
static __host__ __device__ __forceinline__ int item_number(bool causal, int heads, int nq, int r, int head) { return causal ? r * heads + head : head * nq + r; }
struct SplitPlan {
  int heads, nq, nk, causal, c1;     // c1: visible tiles of query tile 0
  int n_whole, run_tiles;
  int pad;                           // 0, or the places every item takes: a multiple of run_tiles, so that no run holds two items
  __host__ __device__ int row_of(int item) const { return causal ? item / heads : item % nq; }
  __host__ __device__ int head_of(int item) const { return causal ? item % heads : item / nq; }
  __host__ __device__ long long row_tiles(int r) const { return !causal || r == 0 ? nk : nq - 1 - r + c1; }
  __host__ __device__ long long rows_before(int r) const {          // tiles of one head's rows 0 .. r-1
    if (!causal || r <= 1) return (long long)r * nk;
    return nk + (long long)(r - 1) * (nq - 1 + c1) - (long long)(r - 1) * r / 2;
  }
  __host__ __device__ long long start(int item) const {             // tiles of all items before this one
    if (pad) return (long long)item * pad;
    if (!causal) return (long long)item * nk;
    const int r = item / heads;
    return rows_before(r) * heads + (item - r * heads) * row_tiles(r);
  }
  __host__ __device__ int item_at(long long pos, int n_items) const {   // the item that holds a tile position
    int lo = n_whole, hi = n_items - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (start(mid) <= pos) lo = mid; else hi = mid - 1;
    }
    return lo;
  }
};
static __host__ __device__ SplitPlan split_plan(int heads, int S, int Skv, int causal, int n_whole, int run_tiles, int pad) {
  SplitPlan s;
  s.heads = heads; s.nq = (S + ATT_BM - 1) / ATT_BM; s.nk = (Skv + ATT_BN - 1) / ATT_BN; s.causal = causal;
  s.c1 = (ATT_BM - 1 + Skv - S) / ATT_BN + 1;
  s.n_whole = n_whole; s.run_tiles = run_tiles; s.pad = pad;
  return s;
}

struct AttnParams {
  int B, Hq, Hkv, S, Skv, D;        // D = value head dim (64 or 128); Q/K depth is padded to 128
  int qk_steps8, qk_steps4;          // MMA instructions along the depth: 4 and 2, or 2 and 1 when the upper half is padding
  int causal;
  int fp8_fmt;                       // descriptor format field: 0 E4M3, 1 E5M2
  const uint8_t* q8_sf; const uint8_t* q4_sf;   // [B,Hq,nq,512]
  const uint8_t* k8_sf; const uint8_t* k4_sf;   // [B,Hkv,nk,512]
  const uint8_t* v8_sf; const uint8_t* v4_sf;   // [B,Hkv,nk,512] (pv_mode 1)
  int v_tiles;                       // 128-key scale tiles per head in v8_sf / v4_sf (= Skv_pad / 128)
  float fp4_scale;                   // NVFP4 score tiles: product of the tensor scales of Q and K,
  const float* ts_q; const float* ts_k;         // or the two factors in device memory
  const uint8_t* map; long long map_sb, map_sh; // [.., nq, nk], strides may be 0 (broadcast); null: the band rule
  int band, uniform;                 // band rule: MXFP8 within `band` tiles of the diagonal; uniform: every visible tile in this format (0: no)
  void* out; int out_dtype;          // [B,Hq,S,D] contiguous; 0 f32, 1 f16, 2 bf16
  float* lse;                        // optional [B,Hq,S]: log2 of the softmax denominator (incl. the row reference)
  const void* acc_in;                // optional fp32 [B,Hq,S,D] + lse_in [B,Hq,S]: an earlier partial result over OTHER keys;
  const float* lse_in;               // the kernel then writes the merged result
  // router inside the forward (ROUTE kernels): an MXFP4 tile whose statistic reaches tau x that of the row's first key
  // tile gets no P.V and no share of the row sum; it is marked TILE_FP8 in map_rw, appended to the item's visit list and
  // done again in MXFP8 after the row's own tiles.
  float tau;
  uint8_t* map_rw;                   // OUTPUT [B,Hq,nq,nk]: the map used
  float* stat_out;                   // optional [B,Hq,nq,nk]: the statistic of every MXFP4 tile visited
  int* range_flag;                   // optional: set to 1 when an item had to be done again (see the file header)
  int* status;
  int n_items;                       // query tiles x heads x batches
  int n_work, n_whole;               // units handed out: n_whole items, then runs of run_tiles tiles over the other items (SplitPlan)
  int run_tiles, run_pad;
  float* part_o; float* part_lse;    // partial results of items that several runs share: [part][item - n_whole][128][D], [..][128]
  int group;                         // q-heads per KV head
  int* counter;                      // optional, zero on entry: items are handed out in turn instead of by a fixed schedule
  int n_lists, list_cap;             // item slots in use (fewer than ATT_MAX_SLOTS for very long rows) and entries of a visit list
  bool load8, load4;                 // formats of Q in use
  bool out32;                        // every row of `out` starts on a 32-byte boundary
};

__device__ __forceinline__ void tmem_ld32p(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16p(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32p(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ void tmem_st8p(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// Block-scaled MMAs with the A operand (P) in TMEM.
__device__ __forceinline__ void mma_mxf8f6f4_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t sfa,
                                                uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_mxf4_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t sfa,
                                            uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
// 8 floats -> 8 E2M1 codes (round to nearest even, saturating), element 0 in the low nibble.
__device__ __forceinline__ uint32_t pack_e2m1x8(float y0, float y1, float y2, float y3, float y4, float y5, float y6,
                                                float y7) {
  uint32_t r;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(r)
      : "f"(y0), "f"(y1), "f"(y2), "f"(y3), "f"(y4), "f"(y5), "f"(y6), "f"(y7));
  return r;
}
// 4 floats -> 4 fp8 codes (E5M2 or E4M3, round to nearest even, saturating), element 0 in the low byte.
template <bool E4M3>
__device__ __forceinline__ uint32_t pack_fp8x4(float y0, float y1, float y2, float y3) {
  uint32_t r;
  if (E4M3) {
    asm("{\n\t.reg .b16 lo, hi;\n\t"
        "cvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\t"
        "cvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\t"
        "mov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(y0), "f"(y1), "f"(y2), "f"(y3));
  } else {
    asm("{\n\t.reg .b16 lo, hi;\n\t"
        "cvt.rn.satfinite.e5m2x2.f32 lo, %2, %1;\n\t"
        "cvt.rn.satfinite.e5m2x2.f32 hi, %4, %3;\n\t"
        "mov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(y0), "f"(y1), "f"(y2), "f"(y3));
  }
  return r;
}

// Maximum of 32 scores with the three-input max: 16 instructions in four independent chains.
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float block_max32(const uint32_t* sc) {
  float b0 = __uint_as_float(sc[0]), b1 = __uint_as_float(sc[1]), b2 = __uint_as_float(sc[2]), b3 = __uint_as_float(sc[3]);
#pragma unroll
  for (int i = 4; i < 28; i += 8) {
    b0 = max3f(b0, __uint_as_float(sc[i]), __uint_as_float(sc[i + 1]));
    b1 = max3f(b1, __uint_as_float(sc[i + 2]), __uint_as_float(sc[i + 3]));
    b2 = max3f(b2, __uint_as_float(sc[i + 4]), __uint_as_float(sc[i + 5]));
    b3 = max3f(b3, __uint_as_float(sc[i + 6]), __uint_as_float(sc[i + 7]));
  }
  b0 = max3f(b0, __uint_as_float(sc[28]), __uint_as_float(sc[29]));
  b1 = max3f(b1, __uint_as_float(sc[30]), __uint_as_float(sc[31]));
  return fmaxf(max3f(b0, b1, b2), b3);
}

// Packed fp32 pairs (one instruction for two lanes of arithmetic): (a, b) += (c, d) and (a, b) = (c, d) - (e, e).
__device__ __forceinline__ void add2(float& a, float& b, float c, float d) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(c), "f"(d));
}
__device__ __forceinline__ void sub2(float& a, float& b, float c, float d, float neg_e) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(a), "=f"(b) : "f"(c), "f"(d), "f"(neg_e));
}

// 2^x for a pair of values on the FMA pipe, for the share of the exponentials taken off the special-function unit:
// x = n + f with n = round(x) (adding 1.5 * 2^23 leaves n in the low mantissa bits), 2^f on [-0.5, 0.5] by a polynomial of degree 5,
// 2^n by adding n to the exponent field.  Least largest relative error among the polynomials with value 1 at 0 (found by reweighted
// least squares), 1.6e-7 with fp32 rounding, against the 2^-22 = 2.4e-7 that ex2.approx is specified with; zero below 2^-126 like it.
// A NaN must not become a zero probability, by which a key would vanish from its row: its patterns, 0x7fffffff in t and in the polynomial,
// add up to the largest finite number, which spoils the row as a NaN does.  (A NaN again, through a multiplication by 2^n, costs 2.5 %.)
__device__ __forceinline__ void fma2(float& a, float& b, float c, float d, float e) {   // (a, b) = (a, b) * (c, d) + (e, e)
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tmov.b64 z, {%4, %4};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(c), "f"(d), "f"(e));
}
__device__ __forceinline__ void ex2_poly2(float& y0, float& y1, float x0, float x1) {
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-200.0f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-200.0f));
  float t0, t1, n0, n1;
  sub2(t0, t1, x0, x1, 12582912.0f);              // t = x + 1.5 * 2^23
  sub2(n0, n1, t0, t1, -12582912.0f);             // n = round(x), as a float
  const float f0 = x0 - n0, f1 = x1 - n1;
  float p0 = 0.00132647285f, p1 = p0;
  fma2(p0, p1, f0, f1, 0.00967151299f);
  fma2(p0, p1, f0, f1, 0.0555073358f);
  fma2(p0, p1, f0, f1, 0.240222454f);
  fma2(p0, p1, f0, f1, 0.693147004f);
  fma2(p0, p1, f0, f1, 1.0f);
  // (an exponent below the smallest: the sign bit is set)
  y0 = __int_as_float(max(__float_as_int(p0) + (__float_as_int(t0) << 23), 0));
  y1 = __int_as_float(max(__float_as_int(p1) + (__float_as_int(t1) << 23), 0));
}

__host__ __device__ constexpr float exp2_of(int n) { return n < 0 ? 0.5f * exp2_of(n + 1) : n > 0 ? 2.0f * exp2_of(n - 1) : 1.0f; }

// Bounded wait for a tagged word in shared memory: returns the word once its tag (bits 1..) equals `tag`, or -1 after
// the limit (status set) or when another role has already recorded a failure.  The status word and the clock are looked
// at every 1024 probes only.
static __device__ __noinline__ int poll_slow(volatile int* word, int tag, int* status) {
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (true) {
    const int w = *word;
    if ((w >> 1) == tag) return w;
    if ((++spins & 0x3ff) == 0) {
      if (*(volatile int*)status != KS_OK) return -1;
      if (clock64() - t0 > kWaitLimitCycles) { atomicCAS(status, KS_OK, KS_TIMEOUT_PIPE); return -1; }
    }
  }
}
__device__ __forceinline__ int poll_tag(volatile int* word, int tag, int* status) {
  const int w = *word;
  if (__builtin_expect((w >> 1) == tag, 1)) return w;
  return poll_slow(word, tag, status);
}

// floor(d) - emax, `least` at least, as an integer and as a float, without conversion instructions (which share the exponential's
// pipe): d + 1.5 * 2^23 rounded DOWN holds floor(d) in its low mantissa bits (|d| < 2^22).
__device__ __forceinline__ int block_shift(float d, int emax, int least, float& sh_f) {
  const float t = __fadd_rd(fmaxf(d, -1024.0f), 12582912.0f);
  const int sh = max(__float_as_int(t) - 0x4b400000 - emax, least);
  sh_f = fmaxf(t - 12582912.0f - (float)emax, (float)least);
  return sh;
}


// N 16-byte pieces (N even) of one row; wide: the address is 32-byte aligned
template <int N>
__device__ __forceinline__ void store_row(void* dst, const uint32_t* w, bool wide) {
  if (wide) {
#pragma unroll
    for (int i = 0; i < N / 2; ++i)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(reinterpret_cast<uint8_t*>(dst) + 32 * i), "r"(w[8 * i]),
                   "r"(w[8 * i + 1]), "r"(w[8 * i + 2]), "r"(w[8 * i + 3]), "r"(w[8 * i + 4]), "r"(w[8 * i + 5]), "r"(w[8 * i + 6]), "r"(w[8 * i + 7])
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
}

__device__ __forceinline__ void mul2(float& a, float& b, float s) {                // (a, b) *= (s, s)
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(s));
}
__device__ __forceinline__ void fma2s(float& a, float& b, float s, float t) {   // (a, b) = (a, b) * (s, s) + (t, t)
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmov.b64 z, {%3, %3};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(s), "f"(t));
}

// One 32-key block of a query row for the quantised P.V: codes of P = exp2(S - m) in the tile's format and the block's E8M0
// scale code - shared exponent floor(log2(amax P)) - emax = floor(bmax - m) - emax.  lsum accumulates the unrounded P (the reference
// sums P before rounding it, ours/mxfp_attn_kernel.py:325).  A block without a visible key (bmax = -inf) comes out as zeros.
//   LATE 1: the exponentials are taken of S as it is, and power-of-two scaling, which is exact, brings them into the block's range
//           afterwards: they wait for S alone and not for the block's maximum too.  m = ATT_REF_Q enters the scale code only, and
//           lsum lacks it.  (512 queries of 32K 175 -> 172 us, with more of them on the FMA pipe 164.)
//   LATE 0: reference and block exponent are subtracted first.  NVFP4 launches, whose scores need a multiplication there anyway;
//           routed ones, where the block's maximum is wanted early (routed causal 8K 393 us, LATE 407).
//   PMODE 1 / 2: MXFP8 E5M2 / E4M3 (8 words); 3: MXFP4 (4 words)
template <int PMODE, int LATE, int NVF4>
__device__ __forceinline__ uint32_t softmax_block_q(uint32_t* sc, [[maybe_unused]] float mref, float bmax, [[maybe_unused]] float mul,
                                                    uint32_t* pk, float& lsum0, float& lsum1) {
  constexpr int EMAX = (PMODE == 3) ? 2 : ((PMODE == 2) ? 8 : 7);
  constexpr int NW = (PMODE == 3) ? 4 : 8;
  float* y = reinterpret_cast<float*>(sc);
  float sh_f;
  const int sh = block_shift(LATE ? bmax : bmax - mref, EMAX, LATE ? (int)ATT_REF_Q - 126 : -126, sh_f);
  // Passes of independent instructions (the values are rewritten in place)
  if (!LATE) {
    const float ncb = -(mref + sh_f);             // exact: mref is integral in this mode
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      if (NVF4) fma2s(y[i], y[i + 1], mul, ncb);
      else sub2(y[i], y[i + 1], y[i], y[i + 1], ncb);
    }
  }
  constexpr int NPOLY = (PMODE == 3) ? (LATE ? ATT_POLY_LATE : ATT_POLY_EARLY) : 0;
#pragma unroll
  for (int i = 0; i < 32 - NPOLY; ++i) y[i] = ex2(y[i]);
#pragma unroll
  for (int i = 32 - NPOLY; i < 32; i += 2) ex2_poly2(y[i], y[i + 1], y[i], y[i + 1]);
  float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    add2(a0, a1, y[i], y[i + 1]);
    add2(b0, b1, y[i + 2], y[i + 3]);
  }
  a0 += b0;
  a1 += b1;
  if (LATE) {
    const float down = __uint_as_float((uint32_t)(127 - sh) << 23);
#pragma unroll
    for (int i = 0; i < 32; i += 2) mul2(y[i], y[i + 1], down);
    lsum0 += a0;
    lsum1 += a1;
  } else {
    const float two_sh = __uint_as_float((uint32_t)(sh + 127) << 23);
    lsum0 = fmaf(a0, two_sh, lsum0);
    lsum1 = fmaf(a1, two_sh, lsum1);
  }
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    constexpr int E = 32 / NW;                    // elements per word
    if (PMODE == 3) pk[w] = pack_e2m1x8(y[w * E], y[w * E + 1], y[w * E + 2], y[w * E + 3], y[w * E + (E > 4 ? 4 : 0)], y[w * E + (E > 4 ? 5 : 1)],
                                        y[w * E + (E > 4 ? 6 : 2)], y[w * E + (E > 4 ? 7 : 3)]);
    else pk[w] = pack_fp8x4<PMODE == 2>(y[w * E], y[w * E + 1], y[w * E + 2], y[w * E + 3]);
  }
  return (uint32_t)(sh + (LATE ? 127 - (int)ATT_REF_Q : 127));
}

// The same for fp16 P, in two steps: y = exp2(S - m) in place for the elements FROM .. TO - 1 of a block, then 16 words of fp16
// pairs and the sums.
template <int NVF4, int FROM, int TO>
__device__ __forceinline__ void exp_block_f16(uint32_t* sc, float mref, [[maybe_unused]] float mul) {
  float* y = reinterpret_cast<float*>(sc);
#pragma unroll
  for (int i = FROM; i < TO; i += 2) {
    if (NVF4) fma2s(y[i], y[i + 1], mul, -mref);
    else sub2(y[i], y[i + 1], y[i], y[i + 1], -mref);
  }
#pragma unroll
  for (int i = FROM; i < TO; i += 2) {
    if (i < 32 - ATT_POLY_F16) { y[i] = ex2(y[i]); y[i + 1] = ex2(y[i + 1]); }
    else ex2_poly2(y[i], y[i + 1], y[i], y[i + 1]);
  }
}
__device__ __forceinline__ void pack_block_f16(const uint32_t* sc, uint32_t* pk, float& lsum0, float& lsum1) {
  const float* y = reinterpret_cast<const float*>(sc);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    add2(lsum0, lsum1, y[2 * i], y[2 * i + 1]);
    pk[i] = pack_f16x2(y[2 * i], y[2 * i + 1]);
  }
}

// A warp's 32 lanes of n fp32 columns of TMEM, each lane times its own factor.  Rare, and out of the way of the loop that needs it.
static __device__ __noinline__ void scale_f32_columns(uint32_t taddr, int n, float f) {
  uint32_t r[32];
  tc_fence_after();
  _Pragma("unroll 1") for (int c = 0; c < n; c += 32) {
    tmem_ld32p(taddr + c, r);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < 32; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) * f);
    tmem_st32p(taddr + c, r);
  }
  tmem_st_wait();
}

// A warp's 64 columns of S: each lane's `shift` is subtracted, and keys beyond `last` (an index into the columns, by lane) become
// -inf.  The few tiles that need it have their S rewritten before it is read, so that the loop over the tiles has no branch for
// them (two in its body, never taken, cost 4 %: the instructions on the two sides of a branch are scheduled apart).
static __device__ __noinline__ void adjust_scores(uint32_t taddr, int last, float shift) {
  uint32_t r[32];
  _Pragma("unroll 1") for (int c = 0; c < 64; c += 32) {
    tmem_ld32p(taddr + c, r);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < 32; ++k) r[k] = c + k > last ? 0xff800000u : __float_as_uint(__uint_as_float(r[k]) - shift);
    tmem_st32p(taddr + c, r);
  }
  tmem_st_wait();
}

// As scale_f32_columns, for 32 columns of fp16 pairs.
static __device__ __noinline__ void scale_f16_columns(uint32_t taddr, float f) {
  uint32_t r[32];
  tmem_ld32p(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&r[k]));
    r[k] = pack_f16x2(v.x * f, v.y * f);
  }
  tmem_st32p(taddr, r);
  tmem_st_wait();
}

// x = *word (shared memory) if `ready`; ordered behind what `ready` was found out with, which a load beside it would not be.
__device__ __forceinline__ void load_if(float& x, uint32_t word, bool ready) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.f32 %0, [%1];\n\t}" : "+f"(x) : "r"(word), "r"((uint32_t)ready) : "memory");
}

// One slot of the visit-list ring: a work item and its tiles.
struct Slot {
  int qi, h, b;
  int mode;          // 0 an item's ordinary pass; 1 it is done again; -1 no more items
  int from;          // mode 1: slot of the first pass, which left the row maxima
  int n_own;         // tiles of the map row
  int n_total;       // ROUTE: appended tiles included, valid once list_done has completed
  int redo;          // set by the softmax threads: a row maximum lies outside the reference's window
  int part;          // slice of the partial results, -1: the item is this CTA's alone
};

template <int PVQ, int NVF4, int ROUTE, int E4M3, int SPLIT>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q8, const __grid_constant__ CUtensorMap tm_q4,
                const __grid_constant__ CUtensorMap tm_k8, const __grid_constant__ CUtensorMap tm_k4,
                const __grid_constant__ CUtensorMap tm_vt, const __grid_constant__ CUtensorMap tm_vt8,
                const __grid_constant__ CUtensorMap tm_vt4, const AttnParams p) {
  static_assert(!SPLIT || !ROUTE, "routed items stay whole: their appended tiles are not known in advance");
  static_assert(!ROUTE || (PVQ && !NVF4), "the router reads MXFP4 operands and runs with quantised P.V");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024 - (raw & 1023)) & 1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ATT_OFF_BAR);
  uint64_t* q_full = bars;                         // [2] Q tile and scales of the item in this set
  uint64_t* q_empty = bars + 2;                    // [2] its last Q.K^T is done
  uint64_t* list_full = bars + 4;                  // [MAX_SLOTS] item and visit list are there
  uint64_t* list_empty = list_full + ATT_MAX_SLOTS;   // [MAX_SLOTS] every reader is through with the item
  uint64_t* list_done = list_empty + ATT_MAX_SLOTS;   // [MAX_SLOTS] ROUTE: the router has been through the row, the list is final
  uint64_t* k_full = list_done + ATT_MAX_SLOTS;    // [KSTAGES]
  uint64_t* v_full = k_full + ATT_KSTAGES;         // [VSLOTS]
  uint64_t* v_empty = v_full + ATT_VSLOTS;         // [VSLOTS] quantised P.V (fp16 P.V: pv_done says it)
  uint64_t* s_full = bars + ATT_B_SFULL;           // [2]
  uint64_t* s_free = s_full + 2;                   // [2] every owner has read the S buffer
  uint64_t* p_ready = s_free + 2;                  // [4] quantised P: tile t & 1; fp16 P: (tile t & 1, 64-key half)
  uint64_t* pv_done = p_ready + 4;                 // [4] likewise
  uint64_t* o_full = pv_done + 4;                  // the item's last P.V is done
  uint64_t* o_free = o_full + 1;                   // the epilogue has read O
  uint64_t* st_bar = o_free + 1;                   // [4] ROUTE, tile t & 3: its owners have published their slice maxima
  uint64_t* x_bar = st_bar + 4;                    // [4] fp16 P.V: first-tile maxima of the two halves of a row
  uint64_t* m_bar = x_bar + 4;                     // [4] fp16 P.V: row references for the other warpgroup
  uint64_t* l_bar = m_bar + 4;                     // [4] partial sums and maxima of a row quarter
  uint64_t* r_bar = l_bar + 4;                     // [4 row quarters][tile & 1][half] fp16 P.V: this half tile has decided on the reference
  uint64_t* drained = r_bar + 16;                  // [2] an issuer that unwinds: its last tensor operations are done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 2);
  volatile int* dec = reinterpret_cast<volatile int*>(tmem_slot + 4);   // [4], slot tile & 3: (tile << 1 | keep) once the router has decided on the tile
  volatile Slot* slots = reinterpret_cast<volatile Slot*>(tmem_slot + 8);   // [MAX_SLOTS]
  uint16_t* lists = reinterpret_cast<uint16_t*>(smem + ATT_OFF_LIST + (PVQ && !ROUTE ? 0 : ATT_EXTRA_BYTES));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (p.S + ATT_BM - 1) / ATT_BM, nk = (p.Skv + ATT_BN - 1) / ATT_BN;
  const int off = p.Skv - p.S;                      // queries are aligned to the end of the keys
  const int NL = p.n_lists;
  constexpr int VSTAGES = ATT_VSLOTS;               // V ring: a slot holds a quantised tile, or a 64-key half of an fp16 one
  constexpr int VSLOT = ATT_V_BYTES / 2;
  constexpr int SF4 = NVF4 ? 1024 : 512;            // bytes of FP4 scales per 128 rows

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1);
      mbar_init(&s_full[s], 1); mbar_init(&s_free[s], 256);
    }
    for (int s = 0; s < ATT_MAX_SLOTS; ++s) { mbar_init(&list_full[s], 1); mbar_init(&list_empty[s], 3 + ATT_SM_WARPS); mbar_init(&list_done[s], 1); }
    for (int s = 0; s < ATT_KSTAGES; ++s) mbar_init(&k_full[s], 1);
    for (int s = 0; s < ATT_VSLOTS; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int s = 0; s < 4; ++s) { mbar_init(&p_ready[s], PVQ ? 256 : 128); mbar_init(&pv_done[s], 1); }
    mbar_init(o_full, 1);
    mbar_init(o_free, 512);
    for (int s = 0; s < 4; ++s) { mbar_init(&x_bar[s], 2); mbar_init(&st_bar[s], 256); mbar_init(&m_bar[s], 1); mbar_init(&l_bar[s], 4); }
    for (int s = 0; s < 16; ++s) mbar_init(&r_bar[s], 1);
    for (int s = 0; s < 2; ++s) mbar_init(&drained[s], 1);
    fence_mbar_init();
    for (int s = 0; s < 4; ++s) dec[s] = -1;        // no tile decided yet
  }
  if (warp == 1) tmem_alloc(tmem_slot, ATT_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // The set-up above, and what each role can do on its own, runs under the kernel that prepares the operands: they wait for it
  // one by one.

  uint8_t* sK = smem + ATT_OFF_K;
  uint8_t* sV = smem + ATT_OFF_V;
  uint8_t* sSFP = smem + ATT_OFF_SFP;               // [0..1] P scale tiles per S buffer, [2+s] V stage s
  const int v_half_bytes = p.D * 128;               // one 64-key half of a V^T tile

  if (warp == 0) {
    // ------------------------------ Q and V loads ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tm_q8); tma_prefetch_desc(&tm_q4);
      if (PVQ) { tma_prefetch_desc(&tm_vt8); tma_prefetch_desc(&tm_vt4); } else tma_prefetch_desc(&tm_vt);
      grid_dependency_wait();
      bool ok = true;
      int sv = 0, tv = 0;                           // ring slot; pieces requested so far (over all items)
      uint32_t v_par = 1;                           // parity of the phase that frees the slot; a fresh barrier satisfies 1
      int q_loads = 0;
      auto load_q = [&](int slot) {                 // the slot's item, into set q_loads & 1
        const int qb = q_loads & 1;
        ok = mbar_wait(&q_empty[qb], ((q_loads >> 1) & 1) ^ 1, p.status, KS_TIMEOUT_PIPE);
        if (!ok) return;
        const int head = slots[slot].b * p.Hq + slots[slot].h, qi = slots[slot].qi;
        const int q_row = head * p.S + qi * ATT_BM;
        const long long qsf = ((long long)head * nq + qi) * 512;
        uint8_t* dst = smem + ATT_OFF_Q + qb * ATT_Q_BYTES;
        uint8_t* sf = smem + ATT_OFF_SFQ + qb * 1536;
        mbar_arrive_expect_tx(&q_full[qb], (p.load8 ? ATT_Q8_BYTES + 512 : 0) + (p.load4 ? ATT_Q4_BYTES + SF4 : 0));
        if (p.load8) {
          tma_load_2d(dst, &tm_q8, &q_full[qb], 0, q_row);
          bulk_load(sf, p.q8_sf + qsf, 512, &q_full[qb]);
        }
        if (p.load4) {
          tma_load_2d(dst + ATT_Q8_BYTES, &tm_q4, &q_full[qb], 0, q_row);
          bulk_load(sf + 512, p.q4_sf + (NVF4 ? 2 * qsf : qsf), SF4, &q_full[qb]);
        }
        ++q_loads;
      };
      const uint32_t v_s0 = smem_u32(sV), vsf_s0 = smem_u32(sSFP + 2 * 512);
      const uint32_t vf0 = smem_u32(v_full), ve0 = smem_u32(PVQ ? v_empty : pv_done);
      int ls = 0;
      uint32_t l_par = 0;                           // list slot and its phase parity
      _Pragma("unroll 1") for (int seq = 0; ok; ++seq) {
        ok = mbar_wait(&list_full[ls], l_par, p.status, KS_TIMEOUT_PIPE);
        if (!ok || slots[ls].mode < 0) break;
        if (q_loads == seq) load_q(ls);
        if (!ok) break;
        const uint16_t* vl = lists + ls * p.list_cap;
        const int hk = slots[ls].b * p.Hkv + slots[ls].h / p.group;
        const uint8_t* v8sf = p.v8_sf + (long long)hk * p.v_tiles * 512;
        const uint8_t* v4sf = p.v4_sf + (long long)hk * p.v_tiles * 512;
        const int v_row = hk * p.D;
        const int ns = ls + 1 == NL ? 0 : ls + 1;
        int iv = 0;
        _Pragma("unroll 1") for (int ph = 0; ph <= ROUTE && ok; ++ph) {
          if (ph == 1) ok = mbar_wait(&list_done[ls], l_par, p.status, KS_TIMEOUT_PIPE);
          if (!ok) break;
          const int hi = ph == 0 ? slots[ls].n_own : slots[ls].n_total;
          const int q_at = ph == 0 ? max(0, hi - 4) : -1;
          uint32_t e = iv < hi ? vl[iv] : 0;
          _Pragma("unroll 1") for (; iv < hi; ++iv) {
            const uint32_t e_next = iv + 1 < hi ? vl[iv + 1] : 0;  // fetched a tile ahead of its use
            // the next item's Q under this one's last tiles, where the item is known and the set free by then
            if (iv == q_at && NL > 1 && q_loads == seq + 1 && mbar_test_wait(&list_full[ns], ns == 0 ? l_par ^ 1 : l_par) && slots[ns].mode >= 0 &&
                mbar_test_wait(&q_empty[q_loads & 1], ((q_loads >> 1) & 1) ^ 1)) load_q(ns);
            const int j = e & ENTRY_TILE;
            if (PVQ == 0) {
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {      // 64-key halves; P.V of the half four before has to be done
                if (ok) ok = mbar_wait_at(ve0 + sv * 8, v_par, p.status, KS_TIMEOUT_PIPE);
                if (!ok) break;
                mbar_arrive_expect_tx_at(vf0 + sv * 8, v_half_bytes);
                tma_load_2d_at(v_s0 + sv * VSLOT, &tm_vt, vf0 + sv * 8, j * ATT_BN + 64 * hf, v_row);
                ++tv;
                if (++sv == VSTAGES) { sv = 0; v_par ^= 1; }
              }
            } else {
              // V^T tile in the tile's format: D rows of 128 (MXFP8) or 64 (MXFP4) bytes, and its scale tile
              ok = mbar_wait_at(ve0 + sv * 8, v_par, p.status, KS_TIMEOUT_PIPE);
              if (!ok) break;
              const bool f8 = (e & ENTRY_F8) != 0;
              mbar_arrive_expect_tx_at(vf0 + sv * 8, (f8 ? v_half_bytes : v_half_bytes / 2) + 512);
              tma_load_2d_at(v_s0 + sv * VSLOT, f8 ? &tm_vt8 : &tm_vt4, vf0 + sv * 8, f8 ? j * ATT_BN : j * (ATT_BN / 2), v_row);
              bulk_load_at(vsf_s0 + sv * 512, (f8 ? v8sf : v4sf) + (long long)j * 512, 512, vf0 + sv * 8);
              ++tv;
              if (++sv == VSTAGES) { sv = 0; v_par ^= 1; }
            }
            if (!ok) break;
            e = e_next;
          }
        }
        if (!ok) break;
        mbar_arrive(&list_empty[ls]);
        if (++ls == NL) { ls = 0; l_par ^= 1; }
      }
      if (!ok) {
        // unwind: copies in flight land before shared memory is released
        _Pragma("unroll 1") for (int u = max(0, q_loads - 2); u < q_loads; ++u) mbar_drain(&q_full[u & 1], (u >> 1) & 1);
        _Pragma("unroll 1") for (int u = max(0, tv - VSTAGES); u < tv; ++u) mbar_drain(&v_full[u % VSTAGES], (u / VSTAGES) & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ K loads and Q.K^T -------------------------
    // S(t) goes to accumulator t & 1 as soon as its K tile has landed and the softmax threads have read S(t - 2).  The same
    // thread requests the K tiles: when S(t - 2) has been read its MMAs are over, so the slot of tile t - 2 takes tile t + 2.
    if (elect_one()) {
      tma_prefetch_desc(&tm_k8); tma_prefetch_desc(&tm_k4);
      grid_dependency_wait();
      uint32_t id8[4], id4[2];
#pragma unroll
      for (int j = 0; j < 4; ++j) id8[j] = idesc_with_sf_id(idesc_block_scaled(p.fp8_fmt, p.fp8_fmt, ATT_BM, ATT_BN, 1), j, j);
#pragma unroll
      for (int j = 0; j < 2; ++j) id4[j] = idesc_with_sf_id(idesc_block_scaled(1, 1, ATT_BM, ATT_BN, 1), 2 * j, 2 * j);
      const uint32_t idn = idesc_block_scaled(1, 1, ATT_BM, ATT_BN, 0);   // NVFP4: E4M3 scales, four per instruction
      const uint64_t k8d0 = sdesc_kmajor_sw128(smem_u32(sK));
      const uint64_t k4d0 = sdesc_kmajor_sw64(smem_u32(sK));
      const uint64_t sfk0 = sdesc_sf_tile(smem_u32(smem + ATT_OFF_SFK));
      const uint32_t sfq8 = tmem + ATT_COL_SFQ8, sfq4 = tmem + ATT_COL_SFQ4;
      const bool half8 = p.qk_steps8 == 2, half4 = p.qk_steps4 == 1;
      bool ok = true;
      int t = 0;                                    // tile counter over all items: K ring slot t mod 4, S buffer t mod 2
      const uint32_t sfree0 = smem_u32(s_free);
      int ls = 0;
      uint32_t l_par = 0;
      // The request side, some tiles ahead: item (its slot and phase parity), position in its list (the end: its list is to be
      // opened, or extended by the appended tiles, or left).
      const uint32_t k_s0 = smem_u32(sK), ksf_s0 = smem_u32(smem + ATT_OFF_SFK), kf0 = smem_u32(k_full);
      int rk = 0, rs = 0, ri = 0, r_hi = 0, r_row = 0, r_state = 0;      // r_state: 0 not open, 1 own tiles, 2 all of them
      uint32_t rq_par = 0;
      const uint8_t *r8sf = nullptr, *r4sf = nullptr;
      // tile number rk; false: what comes next is not known yet (or there is nothing more).  May wait where the tile is needed now.
      auto request_k = [&](bool wait) -> bool {
        _Pragma("unroll 1") while (ri == r_hi) {
          if (r_state == 0) {
            if (wait) { ok = mbar_wait(&list_full[rs], rq_par, p.status, KS_TIMEOUT_PIPE); if (!ok) return false; }
            else if (!mbar_test_wait(&list_full[rs], rq_par)) return false;
            if (slots[rs].mode < 0) return false;
            const int hk = slots[rs].b * p.Hkv + slots[rs].h / p.group;
            r_row = hk * p.Skv;
            r8sf = p.k8_sf + (long long)hk * nk * 512;
            r4sf = p.k4_sf + (long long)hk * nk * SF4;
            ri = 0;
            r_hi = slots[rs].n_own;
            r_state = ROUTE ? 1 : 2;
          } else if (r_state == 1) {
            if (wait) { ok = mbar_wait(&list_done[rs], rq_par, p.status, KS_TIMEOUT_PIPE); if (!ok) return false; }
            else if (!mbar_test_wait(&list_done[rs], rq_par)) return false;
            r_hi = slots[rs].n_total;
            r_state = 2;
          } else {
            ri = r_hi = r_state = 0;
            if (++rs == NL) { rs = 0; rq_par ^= 1; }
          }
        }
        const uint32_t e = lists[rs * p.list_cap + ri++];
        const int j = e & ENTRY_TILE, s = rk & (ATT_KSTAGES - 1);
        const bool f8 = (e & ENTRY_F8) != 0;
        const uint32_t bar = kf0 + s * 8, sf = ksf_s0 + s * 1024;
        mbar_arrive_expect_tx_at(bar, f8 ? ATT_K_BYTES + 512 : ATT_K_BYTES / 2 + SF4);
        tma_load_2d_at(k_s0 + s * ATT_K_BYTES, f8 ? &tm_k8 : &tm_k4, bar, 0, r_row + j * ATT_BN);
        bulk_load_at(sf, f8 ? r8sf + j * 512u : r4sf + j * (uint32_t)SF4, f8 ? 512 : SF4, bar);
        ++rk;
        return true;
      };
      _Pragma("unroll 1") for (int seq = 0; ok; ++seq) {
        const int qb = seq & 1;
        ok = mbar_wait(&list_full[ls], l_par, p.status, KS_TIMEOUT_PIPE);
        if (!ok || slots[ls].mode < 0) break;
        const uint16_t* vl = lists + ls * p.list_cap;
        const uint64_t q8d = sdesc_kmajor_sw128(smem_u32(smem + ATT_OFF_Q + qb * ATT_Q_BYTES));
        const uint64_t q4d = sdesc_kmajor_sw64(smem_u32(smem + ATT_OFF_Q + qb * ATT_Q_BYTES + ATT_Q8_BYTES));
        const uint64_t sfq = sdesc_sf_tile(smem_u32(smem + ATT_OFF_SFQ + qb * 1536));
        int i = 0;
        bool q_there = false;
        _Pragma("unroll 1") for (int ph = 0; ph <= ROUTE && ok; ++ph) {
          int hi;
          if (ph == 0) {
            hi = slots[ls].n_own;
          } else {
            ok = mbar_wait(&list_done[ls], l_par, p.status, KS_TIMEOUT_PIPE);
            if (!ok) break;
            hi = slots[ls].n_total;
          }
          if (!ok) break;
          uint32_t e = i < hi ? vl[i] : 0;
          _Pragma("unroll 1") do {
            if (i < hi && rk > t) {                 // (else its K has to be requested first)
              if (!q_there) {                       // the item's first tile: K has been asked for before Q is waited for
                ok = mbar_wait(&q_full[qb], (seq >> 1) & 1, p.status, KS_TIMEOUT_TMA);
                // the Q scale columns are overwritten: the previous item's last Q.K^T has to be done with them
                if (ok && t > 0) ok = mbar_wait(&s_full[(t - 1) & 1], ((t - 1) >> 1) & 1, p.status, KS_TIMEOUT_MMA);
                if (!ok) break;
                tc_fence_after();
                tc_cp_32x128b_warpx4(sfq8, sfq);
                tc_cp_32x128b_warpx4(sfq4, sfq + (512 >> 4));
                if (NVF4) tc_cp_32x128b_warpx4(sfq4 + 4, sfq + (1024 >> 4));
                q_there = true;
              }
              const uint32_t e_next = vl[min(i + 1, hi - 1)];      // fetched a tile ahead of its use
              const int bsel = t & 1, sk = t & (ATT_KSTAGES - 1);
              // (K first, so that only one wait lies between the release of S and the MMAs)
              ok = mbar_wait_at(kf0 + sk * 8, (t >> 2) & 1, p.status, KS_TIMEOUT_TMA) &&
                   mbar_wait_at(sfree0 + bsel * 8, ((t >> 1) & 1) ^ 1, p.status, KS_TIMEOUT_PIPE);
              if (!ok) break;
              tc_fence_after();
              const uint32_t d = tmem + ATT_COL_S + bsel * 128;
              const uint32_t sfk = tmem + ATT_COL_SFK + bsel * 8;
              const uint64_t ksf = sfk0 + (uint32_t)(sk * (1024 >> 4));
              tc_cp_32x128b_warpx4(sfk, ksf);
              if (e & ENTRY_F8) {
                const uint64_t kd = k8d0 + (uint32_t)(sk * (ATT_K_BYTES >> 4));
                mma_mxf8f6f4(d, q8d, kd, id8[0], sfq8, sfk, 0);
                mma_mxf8f6f4(d, q8d + 2, kd + 2, id8[1], sfq8, sfk, 1);
                if (!half8) {
                  mma_mxf8f6f4(d, q8d + 4, kd + 4, id8[2], sfq8, sfk, 1);
                  mma_mxf8f6f4(d, q8d + 6, kd + 6, id8[3], sfq8, sfk, 1);
                }
              } else {
                const uint64_t kd = k4d0 + (uint32_t)(sk * (ATT_K_BYTES >> 4));
                if (NVF4) {
                  mma_nvf4(d, q4d, kd, idn, sfq4, sfk, 0);
                  if (!half4) {
                    tc_cp_32x128b_warpx4(sfk + 4, ksf + (512 >> 4));
                    mma_nvf4(d, q4d + 2, kd + 2, idn, sfq4 + 4, sfk + 4, 1);
                  }
                } else {
                  mma_mxf4(d, q4d, kd, id4[0], sfq4, sfk, 0);
                  if (!half4) mma_mxf4(d, q4d + 2, kd + 2, id4[1], sfq4, sfk, 1);
                }
              }
              tc_commit(&s_full[bsel]);
              ++i;
              ++t;
              e = e_next;
            }
            // S(t - 3) has been read, so the slot of tile t - 3 is free for tile t + 1 (at the start all slots are)
            _Pragma("unroll 1") while (rk < max(t + 2, ATT_KSTAGES) && request_k(rk <= t && i < hi)) {}
          } while (ok && i < hi);
        }
        if (ok && !q_there) ok = mbar_wait(&q_full[qb], (seq >> 1) & 1, p.status, KS_TIMEOUT_TMA);    // (an item without tiles: its set is free once it has landed)
        if (!ok) break;
        tc_commit(&q_empty[qb]);
        mbar_arrive(&list_empty[ls]);
        if (++ls == NL) { ls = 0; l_par ^= 1; }
      }
      if (!ok) {                                    // unwind: operands and accumulators are in use until then
        tc_commit(&drained[0]);
        mbar_drain(&drained[0], 0);
        _Pragma("unroll 1") for (int u = max(0, rk - ATT_KSTAGES); u < rk; ++u) mbar_drain(&k_full[u % ATT_KSTAGES], (u / ATT_KSTAGES) & 1);
      }
    }
  } else if (warp == 2) {
    // ------------------------------ P.V issuer --------------------------------
    // O += P(t).V(t) as soon as V has landed and the softmax threads have stored P (quantised P: the tile; fp16 P: 64-key
    // halves).  ROUTE: an MXFP4 tile the router leaves out gets no MMA (the commits still go out: the loader and the
    // softmax carry on).
    grid_dependency_wait();
    if (elect_one()) {
      const uint64_t vd0 = sdesc_kmajor_sw128(smem_u32(sV));        // + slot * (VSLOT >> 4)
      const uint64_t v4d0 = sdesc_kmajor_sw64(smem_u32(sV));        // MXFP4 V^T tile (64-byte rows)
      const uint64_t sfp0 = sdesc_sf_tile(smem_u32(sSFP));          // P scale tiles [2], then V scale tiles per stage
      const uint32_t idesc_pv = idesc_f16(0, 0, ATT_BM, p.D);
      uint32_t idp8[4], idp4[2];                                    // P.V block-scaled: M=128, N=D
#pragma unroll
      for (int j = 0; j < 4; ++j) idp8[j] = idesc_with_sf_id(idesc_block_scaled(p.fp8_fmt, p.fp8_fmt, ATT_BM, p.D, 1), j, j);
#pragma unroll
      for (int j = 0; j < 2; ++j) idp4[j] = idesc_with_sf_id(idesc_block_scaled(1, 1, ATT_BM, p.D, 1), 2 * j, 2 * j);
      bool ok = true;
      int sv = 0, t = 0, pb = 0;                    // V ring slot; tile counter; fp16 P: half-buffer
      uint32_t v_par = 0, r_par = 0;                // phase parities: v_full[sv]; p_ready of tile t
      int ls = 0;
      uint32_t l_par = 0;
      _Pragma("unroll 1") for (int seq = 0; ok; ++seq) {
        ok = mbar_wait(&list_full[ls], l_par, p.status, KS_TIMEOUT_PIPE);
        if (!ok || slots[ls].mode < 0) break;
        ok = mbar_wait(o_free, (seq & 1) ^ 1, p.status, KS_TIMEOUT_PIPE);    // the previous item's O has been read
        if (!ok) break;
        const uint16_t* vl = lists + ls * p.list_cap;
        uint32_t acc = 0;                           // 1 once an MMA has written O
        int i = 0;
        _Pragma("unroll 1") for (int ph = 0; ph <= ROUTE && ok; ++ph) {
          int hi;
          if (ph == 0) {
            hi = slots[ls].n_own;
          } else {
            ok = mbar_wait(&list_done[ls], l_par, p.status, KS_TIMEOUT_PIPE);
            if (!ok) break;
            hi = slots[ls].n_total;
          }
          uint32_t e = i < hi ? vl[i] : 0;
          _Pragma("unroll 1") for (; i < hi; ++i) {
            const uint32_t e_next = i + 1 < hi ? vl[i + 1] : 0;
            if (PVQ == 0) {
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                ok = mbar_wait(&v_full[sv], v_par, p.status, KS_TIMEOUT_TMA);
                if (ok) ok = mbar_wait(&p_ready[(t & 1) * 2 + hf], r_par, p.status, KS_TIMEOUT_PIPE);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ptm = tmem + ATT_COL_P16 + pb * 32;
                const uint64_t vh = vd0 + (uint64_t)(sv * (VSLOT >> 4));
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)      // 16 keys per instruction, 8 TMEM columns of P
                  mma_f16_ts(tmem + ATT_COL_O, ptm + ks * 8, vh + (uint64_t)(2 * ks), idesc_pv, (hf > 0 || ks > 0) ? 1u : acc);
                tc_commit(&pv_done[(t & 1) * 2 + hf]);    // (frees the V slot too: slot and barrier both follow the half's number)
                if (++pb == 3) pb = 0;
                if (++sv == VSTAGES) { sv = 0; v_par ^= 1; }
              }
              if (!ok) break;
              acc = 1;
            } else {
              ok = mbar_wait(&v_full[sv], v_par, p.status, KS_TIMEOUT_TMA);
              if (!ok) break;
              const int bsel = t & 1;
              ok = mbar_wait(&p_ready[bsel], r_par, p.status, KS_TIMEOUT_PIPE);
              if (!ok) break;
              bool keep = true;
              if (ROUTE && !(e & ENTRY_F8)) {
                // the router's word for this tile: written while P was being stored, as a rule (asked for first, this thread would
                // poll for a third of its time)
                const int d = poll_tag(&dec[t & 3], t, p.status);
                if (d < 0) { ok = false; break; }
                keep = (d & 1) != 0;
              }
              if (keep) {
                tc_fence_after();
                const uint32_t ptm = tmem + ATT_COL_P + bsel * 32;
                const uint32_t sfp = tmem + ATT_COL_SFP + bsel * 4, sfv = tmem + ATT_COL_SFV + bsel * 4;
                tc_cp_32x128b_warpx4(sfp, sfp0 + (uint64_t)(bsel * (512 >> 4)));
                tc_cp_32x128b_warpx4(sfv, sfp0 + (uint64_t)((2 + sv) * (512 >> 4)));
                if (e & ENTRY_F8) {
                  const uint64_t vd = vd0 + (uint64_t)(sv * (VSLOT >> 4));
#pragma unroll
                  for (int ks = 0; ks < 4; ++ks)    // 32 keys per instruction, 8 TMEM columns of P
                    mma_mxf8f6f4_ts(tmem + ATT_COL_O, ptm + ks * 8, vd + 2 * ks, idp8[ks], sfp, sfv, ks > 0 ? 1u : acc);
                } else {
                  const uint64_t vd = v4d0 + (uint64_t)(sv * (VSLOT >> 4));
#pragma unroll
                  for (int ks = 0; ks < 2; ++ks)    // 64 keys per instruction, 8 TMEM columns of P
                    mma_mxf4_ts(tmem + ATT_COL_O, ptm + ks * 8, vd + 2 * ks, idp4[ks], sfp, sfv, ks > 0 ? 1u : acc);
                }
                acc = 1;
              }
              tc_commit(&pv_done[bsel]);
              tc_commit(&v_empty[sv]);
              if (++sv == VSTAGES) { sv = 0; v_par ^= 1; }
            }
            if (t & 1) r_par ^= 1;
            ++t;
            e = e_next;
          }
        }
        if (!ok) break;
        tc_commit(o_full);
        mbar_arrive(&list_empty[ls]);
        if (++ls == NL) { ls = 0; l_par ^= 1; }
      }
      if (!ok) { tc_commit(&drained[1]); mbar_drain(&drained[1], 0); }
    }
  } else if (warp == 3) {
    // ------------------------------ work items, visit lists and router ----------
    // The first item is known without asking anybody, and its list under the band rule too: it is there when the operands are (first
    // scores 2.5 -> 1.9 us after them).
    if (ROUTE || p.map) grid_dependency_wait();
    bool ok = true;
    int emitted = 0, reclaimed = 0;                 // slots filled, and taken back
    int next_local = 0;                             // static schedule: items taken so far
    int redo_item = -1, redo_from = 0;              // work to be done again: it is the next to be handed out
    const int heads = p.Hq * p.B;
    int held[ATT_MAX_SLOTS];                        // work in each slot, -1: nothing that could come back
    // Work is an item number; a share of a run's also has the run in wrun (0: the whole item).
    [[maybe_unused]] int held_run[ATT_MAX_SLOTS], redo_run = 0;
    [[maybe_unused]] int run = 0;                   // this CTA's present run, from 1
    [[maybe_unused]] long long run_pos = 0, run_end = 0;
    const SplitPlan plan = split_plan(heads, p.S, p.Skv, p.causal, p.n_whole, p.run_tiles, p.run_pad);
    [[maybe_unused]] const long long run_base = SPLIT ? plan.start(p.n_whole) : 0;
    auto reclaim = [&]() {
      const int s = reclaimed % NL;
      ok = __all_sync(0xffffffffu, mbar_wait(&list_empty[s], (reclaimed / NL) & 1, p.status, KS_TIMEOUT_PIPE));
      ++reclaimed;
      int it = -1, rw = 0;
#pragma unroll
      for (int k = 0; k < ATT_MAX_SLOTS; ++k) if (k == s) { it = held[k]; if (SPLIT) rw = held_run[k]; }
      if (ok && it >= 0 && slots[s].redo) { redo_item = it; redo_run = rw; redo_from = s; }
    };
    // The next item into the next slot, which is free: first what has to be done again, then the schedule.  Items are
    // numbered heaviest query tile first; after a CTA's first they are taken from a counter in memory where the caller gives one, else in
    // snake order over the CTAs, which evens out the sum.  false: nothing left.
    auto emit = [&]() -> bool {
      int item, mode = 0, wrun = 0;
      if (redo_item >= 0) {
        item = redo_item;
        if (SPLIT) wrun = redo_run;
        mode = 1;
        redo_item = -1;
      } else if (SPLIT && run_pos < run_end) {
        item = plan.item_at(run_pos, p.n_items);
        wrun = run;
        run_pos = plan.start(item + 1);
      } else {
        if (p.counter && emitted > 0) {
          int n = 0;
          if (lane == 0) n = (int)gridDim.x + atomicAdd(p.counter, 1);
          item = __shfl_sync(0xffffffffu, n, 0);
        } else {
          item = next_local * (int)gridDim.x + ((next_local & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
          ++next_local;
        }
        if (item >= p.n_work) return false;
        if (SPLIT && item >= p.n_whole) {
          wrun = run = item - p.n_whole + 1;
          run_pos = run_base + (long long)(run - 1) * p.run_tiles;
          run_end = min(run_pos + p.run_tiles, plan.start(p.n_items));
          item = plan.item_at(run_pos, p.n_items);
          run_pos = plan.start(item + 1);
        }
      }
      const int s = emitted % NL;
      const int r = plan.row_of(item), bh = plan.head_of(item);
      const int qi = nq - 1 - r, b = bh / p.Hq, h = bh - b * p.Hq;
      // ordered compaction of the item's map row, 32 cells at a time; the map comes from memory, or from the band rule
      uint16_t* vl = lists + s * p.list_cap;
      const long long row_off = (long long)b * p.map_sb + (long long)h * p.map_sh + (long long)qi * nk;
      const bool from_rw = ROUTE && mode > 0;       // done again: the map as the router left it
      const uint8_t* row = from_rw ? p.map_rw + row_off : (p.map ? p.map + row_off : nullptr);
      const int last_key = min(p.S - 1, qi * ATT_BM + ATT_BM - 1) + off;    // last key any row of the tile may see
      int base = 0, j_lo = 0, j_hi = nk, part = -1;
      if (SPLIT && wrun > 0) {                     // the run's share of the item
        const long long it0 = plan.start(item), it1 = it0 + plan.row_tiles(r);
        const long long a = run_base + (long long)(wrun - 1) * p.run_tiles, e = a + p.run_tiles;
        if (it0 < a || it1 > e) {
          part = wrun - 1 - (int)((it0 - run_base) / p.run_tiles);
          j_lo = (int)(max(a, it0) - it0);
          j_hi = (int)(min(e, it1) - it0);          // (padded places at the end: no tile)
        }
      }
      _Pragma("unroll 1") for (int i0 = j_lo; i0 < j_hi; i0 += 32) {
        const int j = i0 + lane;
        int c = TILE_SKIP;
        if (j < j_hi) {
          if (row) c = __ldcg(row + j);
          else {
            c = p.uniform ? p.uniform : (abs(qi + off / ATT_BN - j) < p.band ? TILE_FP8 : TILE_FP4);
            if (p.causal && j * ATT_BN > last_key) c = TILE_SKIP;
          }
          if (ROUTE && !from_rw) p.map_rw[row_off + j] = (uint8_t)c;
        }
        const uint32_t vis = __ballot_sync(0xffffffffu, c != TILE_SKIP);
        if (c != TILE_SKIP) {
          const bool mask = (p.causal && j * ATT_BN + ATT_BN - 1 > qi * ATT_BM + off) || (j * ATT_BN + ATT_BN > p.Skv);
          vl[base + __popc(vis & ((1u << lane) - 1u))] = (uint16_t)(j | (c == TILE_FP8 ? ENTRY_F8 : 0) | (mask ? ENTRY_MASK : 0));
        }
        base += __popc(vis);
        if (!ROUTE && !row && p.causal && (i0 + 32) * ATT_BN > last_key) break;
      }
      __syncwarp();
      if (lane == 0) {
        slots[s].qi = qi; slots[s].h = h; slots[s].b = b; slots[s].mode = mode; slots[s].from = redo_from; slots[s].n_own = base; slots[s].n_total = base;
        slots[s].redo = 0;
        if (SPLIT) slots[s].part = part;
        mbar_arrive(&list_full[s]);                 // release: entries (__syncwarp) and slot are visible to who waits
      }
#pragma unroll
      for (int k = 0; k < ATT_MAX_SLOTS; ++k) if (k == s) { held[k] = mode == 0 || ROUTE ? item : -1; if (SPLIT) held_run[k] = wrun; }
      ++emitted;
      return true;
    };
    // Router: statistic of every MXFP4 tile = mean over the query rows of the row maximum.  Lane l takes rows l, 32 + l,
    // 64 + l, 96 + l of the published slice maxima; the four 32-row sums are formed by the same butterfly and added in the
    // same order as in route_stat_kernel / route_stat_finish_kernel, so the statistic is the same bit for bit.
    [[maybe_unused]] uint32_t st_par = 0;                 // phase parities of st_bar, as bits
    [[maybe_unused]] int t = 0;
    auto route = [&](int seq) {
      const int s = seq % NL;
      uint16_t* vl = lists + s * p.list_cap;
      const int nv = slots[s].n_own;
      int appended = 0;
      {
        const bool decided = slots[s].mode != 0;    // done again: its list has the decisions of the first pass
        const int qi = slots[s].qi, h = slots[s].h, b = slots[s].b;
        const long long row_off = (long long)b * p.map_sb + (long long)h * p.map_sh + (long long)qi * nk;
        const float inv_rows = 1.0f / (float)min(ATT_BM, p.S - qi * ATT_BM);
        float sink = 0.0f;                          // statistic of the row's first key tile (0 until it has been seen)
        _Pragma("unroll 1") for (int i = 0; i < nv; ++i) {
          const uint32_t e = vl[i];
          if (e & ENTRY_F8) continue;               // MXFP8 by the band rule: nothing to decide
          const int tt = t + i, buf = tt & 3;
          ok = __all_sync(0xffffffffu, mbar_wait(&st_bar[buf], (st_par >> buf) & 1, p.status, KS_TIMEOUT_PIPE));
          st_par ^= 1u << buf;
          if (!ok) break;
          const float* rm = reinterpret_cast<const float*>(smem + ATT_OFF_EXTRA) + buf * 2 * 128;
          float pq[4];
#pragma unroll
          for (int qq = 0; qq < 4; ++qq) {
            const int r = qq * 32 + lane;
            const float mxr = fmaxf(rm[r], rm[128 + r]);
            pq[qq] = (qi * ATT_BM + r < p.S && mxr != -INFINITY) ? mxr * inv_rows : 0.0f;
          }
          const bool up = (lane & 16) != 0, up8 = (lane & 8) != 0;
          const float r0 = __shfl_xor_sync(0xffffffffu, up ? pq[0] : pq[2], 16), r1 = __shfl_xor_sync(0xffffffffu, up ? pq[1] : pq[3], 16);
          const float u0 = (up ? pq[2] : pq[0]) + r0, u1 = (up ? pq[3] : pq[1]) + r1;
          float w = (up8 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, up8 ? u0 : u1, 8);
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
          const float s0 = __shfl_sync(0xffffffffu, w, 0), s1 = __shfl_sync(0xffffffffu, w, 8), s2 = __shfl_sync(0xffffffffu, w, 16), s3 = __shfl_sync(0xffffffffu, w, 24);
          const float stat = ((s0 + s1) + s2) + s3;
          const int j = e & ENTRY_TILE;
          if (j == 0) sink = stat;
          const bool keep = decided || !(stat >= sink * p.tau);
          if (lane == 0) {
            dec[tt & 3] = (tt << 1) | (keep ? 1 : 0);     // one word: readers poll it, nothing else to publish
            if (!keep) {
              // promoted: the MXFP4 result of this tile is left out; the tile is done again in MXFP8 after the row's own tiles
              p.map_rw[row_off + j] = TILE_FP8;
              vl[nv + appended] = (uint16_t)(e | ENTRY_F8);
            }
            if (p.stat_out && !decided) p.stat_out[(((long long)b * p.Hq + h) * nq + qi) * nk + j] = stat;
          }
          if (!keep) ++appended;
          __syncwarp();
        }
      }
      if (lane == 0) {
        slots[s].n_total = nv + appended;           // the list is complete (also after a failure: the others see the status word)
        mbar_arrive(&list_done[s]);
      }
      t += nv + appended;
    };
    // An item is handed out before the previous one is routed.  When the schedule is exhausted the slots are taken back,
    // which shows what has to be done again.
    const int ahead = NL > 1 ? 2 : 1;
    int seq = 0;                                    // items routed
    bool exhausted = false;
    _Pragma("unroll 1") while (ok) {
      if (!PVQ && exhausted && emitted - reclaimed < NL) break;    // (no item comes back: the end can be said at once)
      const bool want = !exhausted && emitted - seq < ahead;
      if (want ? emitted - reclaimed >= NL : (seq == emitted && reclaimed < emitted)) {
        reclaim();
        if (redo_item >= 0) exhausted = false;
      } else if (want) {
        exhausted = !emit();
        if (!ROUTE) grid_dependency_wait();         // (before the counter and the next items; it is over by the second time)
      } else if (seq < emitted) {
        if (ROUTE) route(seq);
        ++seq;
      } else {
        break;
      }
    }
    if (ok && lane == 0) {
      // the next slot, which is free, says that there is nothing more
      const int s = emitted % NL;
      slots[s].mode = -1;
      mbar_arrive(&list_full[s]);
    }
  } else {
    // ------------------------------ softmax and epilogue ----------------------
    const int sw = warp - ATT_SERVICE_WARPS;
    const int q = warp & 3;                         // TMEM lane quarter this warp may access
    const int g = (sw >> 2) & 1;                    // half of the tile's keys
    const int wg = sw >> 3;                         // warpgroup: owns S and P buffer wg, i.e. the tiles t = wg mod 2
    const int r_in = q * 32 + lane;                 // row inside the tile == TMEM lane
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const uint32_t slice_addr = lane_base + ATT_COL_S + wg * 128 + g * 64;
    const uint32_t p_addr = lane_base + (PVQ ? ATT_COL_P + wg * 32 : ATT_COL_P16);
    float* xrow = reinterpret_cast<float*>(smem + ATT_OFF_XROW);
    float* rmax = reinterpret_cast<float*>(smem + ATT_OFF_RMAX);
    float* mrow = reinterpret_cast<float*>(smem + ATT_OFF_MROW);
    float* mslot = reinterpret_cast<float*>(smem + ATT_OFF_MSLOT);
    uint8_t* psf_dst = sSFP + wg * 512 + lane * 16 + q * 4 + g * 2;
    grid_dependency_wait();
    const float nvmul = NVF4 ? (p.ts_q ? *p.ts_q * *p.ts_k : p.fp4_scale) : 1.0f;   // scores of NVFP4 tiles lack the tensor scales
    // An item's epilogue is put off until this thread has done its first tile of the next item, so that neither the last
    // P.V nor the warpgroup that had the last tile is waited for.  (Not with fp16 P.V: there a P buffer of the next
    // item's second tile is free only once O has been read.)
    constexpr bool DEFER = PVQ != 0;
    constexpr bool LATE = PVQ && !NVF4 && !ROUTE;   // softmax_block_q; row sums lack the reference, an item done again has its S shifted first
    [[maybe_unused]] bool again = false;            // the item is done again, with references of its own
    bool ok = true;
    int t0 = 0;                                     // tiles of the items before this one
    int pb16 = (2 * wg + g) % 3;                    // fp16 P.V: P buffer of the next tile's half
    const uint32_t a_wg = smem_u32(bars) + wg * 8;  // shared address of barrier 0 of this warpgroup's pairs
    // fp16 P.V.  The four warps of a row quarter are numbered 2 wg + g, in the order of their half tiles.  r_bar of the warp before
    // this one - the same tile's first half, or the second one of the other warpgroup's tile - is its turn to decide on the row
    // reference.
    const uint32_t a_pr16 = smem_u32(&p_ready[wg * 2 + g]), a_pv16 = smem_u32(&pv_done[(wg * 2 + g + 1) & 3]);
    const uint32_t a_turn = (a_pv16 ^ 16) + (ATT_B_RBAR - ATT_B_PVDONE) * 8 + (r_in & 96), a_decided = a_pr16 + (ATT_B_RBAR - ATT_B_PREADY) * 8 + (r_in & 96);
    // phase parities to wait for, as bits: 1 this warpgroup's tile count; fp16 P.V: 2 P.V of the half tile three before, 4 the half
    // tile before (turn and P.V)
    uint32_t par = PVQ ? 0 : ((g == 1 && wg == 1) ? 0u : 2u) | ((g == 0 && wg == 0) ? 4u : 0u);
    float* lref = reinterpret_cast<float*>(smem + ATT_OFF_EXTRA);
    [[maybe_unused]] float* rmax_w = reinterpret_cast<float*>(smem + ATT_OFF_EXTRA) + (wg * 2 + g) * 128 + r_in;   // + 512 floats for tiles 2, 3 of 4
    float m_redo = 0.0f;                            // row reference of an item that is done again: the maximum its first pass found
    float mref = 0.0f, l_run = 0.0f, m_run = -INFINITY;   // row reference; partial row sum and maximum over this thread's keys
    [[maybe_unused]] float pend_l = 0.0f;           // ROUTE: row sum of this warpgroup's last tile, if it was MXFP4, until the decision on it is looked up
    [[maybe_unused]] int pend_t = 0;
    int ls = 0, seq = 0, n_tiles = 0, i = 0, lim = 0;
    uint32_t l_par = 0;
    bool in_item = false, second = false;           // second: ROUTE, the appended tiles
    bool epi = false;                               // an epilogue is outstanding: item seq - 1, in slot epi_ls
    int epi_ls = 0, epi_part = 0;
    auto last_key = [&]() { return p.causal ? min(p.Skv - 1, slots[ls].qi * ATT_BM + r_in + off) : p.Skv - 1; };
    auto settle = [&]() {                           // the last of the item's own tiles
      if (pend_l != 0.0f) {
        const int d = poll_tag(&dec[pend_t & 3], pend_t, p.status);
        if (d < 0) ok = false;
        l_run += (d & 1) ? pend_l : 0.0f;
        pend_l = 0.0f;
      }
    };
    _Pragma("unroll 1") while (ok) {
      bool do_epi = false;
      if (in_item && i < n_tiles) {
        // ---- a run of tiles.  The first 32 columns of a tile are requested under the previous tile's last steps. ----
        const uint16_t* vl = lists + ls * p.list_cap;
        uint32_t e = vl[i];
        bool more;
        _Pragma("unroll 1") do {
          const uint32_t ec = e;
          const int t = t0 + i;
          i += 2;
          more = i < n_tiles && !epi;
          if (more) e = vl[i];
          float lsum0 = 0.0f, lsum1 = 0.0f;
          uint32_t sc[32];
          ok &= mbar_wait_at(a_wg + ATT_B_SFULL * 8, par & 1, p.status, KS_TIMEOUT_MMA);
          __syncwarp();
          tc_fence_after();
          if (__builtin_expect((ec & ENTRY_MASK) || (LATE && again), 0))
            adjust_scores(slice_addr, ec & ENTRY_MASK ? lim - ((int)(ec & ENTRY_TILE) * ATT_BN + g * 64) : 64, LATE && again ? m_redo : 0.0f);
          tmem_ld32p(slice_addr, sc);
          if (PVQ) {
            uint32_t pk[16];
            uint32_t psc;
            auto tile = [&](auto pm_c) {            // 3 MXFP4, 1 / 2 MXFP8 E5M2 / E4M3
              constexpr int PM = decltype(pm_c)::value;
              constexpr int PW = PM == 3 ? 4 : 8;   // words of codes per block
              constexpr int NV = (NVF4 && PM == 3) ? 1 : 0;
              tmem_ld_wait();
              const float b0 = NV ? block_max32(sc) * nvmul : block_max32(sc);
              psc = softmax_block_q<PM, LATE, NV>(sc, mref, b0, nvmul, pk, lsum0, lsum1);
              tmem_ld32p(slice_addr + 32, sc);
              tmem_ld_wait();
              tc_fence_before();
              mbar_arrive_at(a_wg + ATT_B_SFREE * 8);   // S has been read: Q.K^T of tile t + 2 may overwrite it
              const bool p_free = mbar_test_wait_at(a_wg + ATT_B_PVDONE * 8, (par & 1) ^ 1);   // (its answer is used after the arithmetic)
              const float b1 = NV ? block_max32(sc) * nvmul : block_max32(sc), bm = fmaxf(b0, b1);
              m_run = fmaxf(m_run, bm);
              if (ROUTE && PM == 3) {               // published before the block's arithmetic, so that the router decides under it
                rmax_w[(par & 1) * 512] = bm;
                mbar_arrive_at(a_wg + (ATT_B_ST + (par & 1) * 2) * 8);
              }
              psc |= softmax_block_q<PM, LATE, NV>(sc, mref, b1, nvmul, pk + PW, lsum0, lsum1) << 8;
              // the P buffer and its scale tile: P.V of tile t - 2 has read them (a fresh barrier satisfies the first wait)
              if (!__all_sync(0xffffffffu, p_free)) ok &= mbar_wait_at(a_wg + ATT_B_PVDONE * 8, (par & 1) ^ 1, p.status, KS_TIMEOUT_MMA);
              __syncwarp();
              tc_fence_after();
              // P.V of the tile before, which has been waited for, came after the decision on that tile: its share of the row sum
              if (ROUTE) l_run += (dec[(t & 3) ^ 2] & 1) ? pend_l : 0.0f;
              if (PM == 3) tmem_st8p(p_addr + g * 8, pk);
              else tmem_st16p(p_addr + g * 16, pk);
            };
            if (!(ec & ENTRY_F8)) tile(std::integral_constant<int, 3>{});
            else tile(std::integral_constant<int, E4M3 ? 2 : 1>{});
            // this row's block scales go into the 128x4 scale tile of the P buffer, which the P.V issuer copies to TMEM:
            // row r, block k at byte (r % 32) * 16 + (r / 32) * 4 + k
            *reinterpret_cast<uint16_t*>(psf_dst) = (uint16_t)psc;
            fence_proxy_async_smem();               // make the tile visible to tcgen05.cp
          } else {
            uint32_t pk[32];
            const float mul = (NVF4 && !(ec & ENTRY_F8)) ? nvmul : 1.0f;
            bool dead = false;
            _Pragma("unroll 1") while (true) {
              tmem_ld_wait();
              m_run = fmaxf(m_run, block_max32(sc) * mul);
              exp_block_f16<NVF4, 0, 32>(sc, mref, mul);
              uint32_t sn[32];                      // (read before the first block is packed, whose arithmetic then fills the gaps of this one's)
              tmem_ld32p(slice_addr + 32, sn);
              tmem_ld_wait();
              pack_block_f16(sc, pk, lsum0, lsum1);
#pragma unroll
              for (int k = 0; k < 32; ++k) sc[k] = sn[k];
              m_run = fmaxf(m_run, block_max32(sc) * mul);      // (no earlier score goes beyond: it would have raised the reference)
              const bool stays = __all_sync(0xffffffffu, ok && !(m_run - mref > ATT_TOP_F16));
              exp_block_f16<NVF4, 0, ATT_F16_EARLY>(sc, mref, mul);    // (under the vote)
              if (__builtin_expect(stays, 1)) break;
              if (!__all_sync(0xffffffffu, ok)) { dead = true; break; }
              // A row goes beyond its reference: this half raises it in its turn, once the half before it has decided, and hands
              // the turn on where every half does.
              ok &= mbar_wait_at(a_turn, (par >> 2) & 1, p.status, KS_TIMEOUT_PIPE);
              __syncwarp();
              const float mc = mrow[r_in], m_new = m_run - mc > ATT_TOP_F16 ? m_run : mc;
              if (__any_sync(0xffffffffu, m_new != mc)) {
                // O is at mc: it is scaled once P.V of the half before this one is done.  (That of the half two before it comes first:
                // the wait for a phase has to know that the one before is over.)
                ok &= mbar_wait_at(a_pv16, (par >> 1) & 1, p.status, KS_TIMEOUT_MMA);
                ok &= mbar_wait_at(a_pv16 ^ 16, (par >> 2) & 1, p.status, KS_TIMEOUT_MMA);
                __syncwarp();
                scale_f32_columns(lane_base + ATT_COL_O, p.D, ex2(mc - m_new));
                mrow[r_in] = m_new;
                __syncwarp();
              }
              l_run *= ex2(mref - m_new);
              mref = m_new;
              lsum0 = lsum1 = 0.0f;
              tmem_ld32p(slice_addr, sc);           // the tile again
            }
            if (dead) { ok = false; break; }
            tc_fence_before();
            mbar_arrive_at(a_wg + ATT_B_SFREE * 8);
            exp_block_f16<NVF4, ATT_F16_EARLY, 32>(sc, mref, mul);
            // What has to be there before P is stored, asked for in one vote: this half's turn (the half before it has decided), the
            // reference as it was, and the P buffer of this half, number h = 2t + g over all items: h mod 3.  P.V of half h - 3 has
            // read it: the other half of this warpgroup's previous tile (g = 0), or the first half of the other warpgroup's (g = 1).
            const bool turn = mbar_try_wait(a_turn, (par >> 2) & 1);
            float m_now = __int_as_float(0x7fffffff);
            const bool room = mbar_try_wait(a_pv16, (par >> 1) & 1);
            pack_block_f16(sc, pk + 16, lsum0, lsum1);
            load_if(m_now, smem_u32(mrow + r_in), turn);
            bool moved = false;
            if (!__all_sync(0xffffffffu, turn && room && m_now == mref)) {
              ok &= mbar_wait_at(a_turn, (par >> 2) & 1, p.status, KS_TIMEOUT_PIPE);
              __syncwarp();
              m_now = mrow[r_in];
              moved = __any_sync(0xffffffffu, m_now != mref);
              ok &= mbar_wait_at(a_pv16, (par >> 1) & 1, p.status, KS_TIMEOUT_MMA);
              __syncwarp();
            }
            mbar_arrive_lane0(a_decided, lane);
            tc_fence_after();
            tmem_st16p(p_addr + pb16 * 32, pk);
            tmem_st16p(p_addr + pb16 * 32 + 16, pk + 16);
            if (__builtin_expect(moved, 0)) {       // a half before this one has raised the reference meanwhile
              const float f = ex2(mref - m_now);
              tmem_st_wait();
              scale_f16_columns(p_addr + pb16 * 32, f);
              l_run *= f;
              lsum0 *= f;
              lsum1 *= f;
              mref = m_now;
            }
            pb16 = pb16 == 2 ? 0 : pb16 + 1;        // four halves further on
          }
          par ^= PVQ ? 1 : 7;
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive_at(PVQ ? a_wg + ATT_B_PREADY * 8 : a_pr16);
          if (ROUTE) {
            pend_l = ec & ENTRY_F8 ? 0.0f : lsum0 + lsum1;     // counts only if the router keeps the tile
            pend_t = t;
            if (ec & ENTRY_F8) l_run += lsum0 + lsum1;
          } else {
            l_run += lsum0 + lsum1;
          }
          if (PVQ && !__all_sync(0xffffffffu, ok)) { ok = false; break; }
        } while (more);
        if (PVQ == 0) ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        do_epi = DEFER && epi;
      } else if (in_item) {
        if (epi) {
          do_epi = true;                            // this warpgroup has no tile in this item: the previous one first
        } else if (ROUTE && !second) {
          settle();
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&list_done[ls], l_par, p.status, KS_TIMEOUT_PIPE));
          if (!ok) break;
          n_tiles = slots[ls].n_total;
          second = true;
        } else {
          // the item's tiles are done: publish the partial results
          epi_part = (((t0 & 1) ^ wg) << 1) | g;    // the same order of summation whichever warpgroup owned the first tile
          float* xl = xrow + (seq & 1) * 1024 + epi_part * 128 + r_in;
          xl[0] = LATE ? l_run * exp2_of(-(int)ATT_REF_Q) : l_run;
          if (PVQ) {
            xl[512] = m_run;
          } else {
            // what rounding to fp16 makes of this thread's largest P
            const float p_max = ex2(m_run - mref);
            xl[512] = __half2float(__float2half_rn(p_max)) - p_max;
            lref[(seq & 1) * 512 + epi_part * 128 + r_in] = mref;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&l_bar[q]);
          t0 += n_tiles;
          epi = true;
          epi_ls = ls;
          in_item = false;
          ++seq;
          if (++ls == NL) { ls = 0; l_par ^= 1; }
          do_epi = !DEFER;
        }
      } else {
        // an outstanding epilogue comes first when no item is there to put it before (the last one waits for the epilogue
        // itself: it may have to be done again)
        do_epi = epi && !__all_sync(0xffffffffu, mbar_test_wait(&list_full[ls], l_par));
        int mode = 0;
        if (!do_epi) {
          ok = __all_sync(0xffffffffu, mbar_wait(&list_full[ls], l_par, p.status, KS_TIMEOUT_PIPE));
          if (!ok) break;
          mode = slots[ls].mode;
          do_epi = PVQ && epi && mode == 1;         // m_redo may still be in use
        }
        if (do_epi) {
        } else if (mode < 0) {
          break;
        } else {
          in_item = true;
          second = false;
          again = mode == 1;
          n_tiles = slots[ls].n_own;
          const int m_glob = slots[ls].qi * ATT_BM + r_in;
          lim = last_key();                         // last visible key of this row
          l_run = 0.0f;
          m_run = -INFINITY;
          if (PVQ && mode == 1) m_redo = mslot[slots[ls].from * 128 + r_in];
          mref = PVQ ? (mode == 1 ? m_redo : ATT_REF_Q) : ATT_NO_REF;
          i = (t0 & 1) ^ wg;                        // first tile of the list this warpgroup owns
          if (PVQ == 0 && n_tiles == 0 && i == 0 && lane == 0) {   // no exchange, but the barriers' phases follow the items
            mbar_arrive(&x_bar[q]);
            if (g == 0) mbar_arrive(&m_bar[q]);
          }
          if (PVQ == 0 && n_tiles > 0) {
            // the row's first reference: the maximum of the item's first tile, found by its owners.  (Every thread of the row is
            // through with the item before: its epilogue has waited for all of them.)
            if (i == 0) {
              ok = __all_sync(0xffffffffu, mbar_wait(&s_full[wg], par & 1, p.status, KS_TIMEOUT_MMA));
              if (!ok) break;
              tc_fence_after();
              const uint32_t e = lists[ls * p.list_cap];
              if (e & ENTRY_MASK) adjust_scores(slice_addr, lim - ((int)(e & ENTRY_TILE) * ATT_BN + g * 64), 0.0f);
              float mx = -INFINITY;
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                uint32_t sc[32];
                tmem_ld32p(slice_addr + c * 32, sc);
                tmem_ld_wait();
                mx = fmaxf(mx, block_max32(sc));
              }
              rmax[g * 128 + r_in] = mx;
              __syncwarp();
              if (lane == 0) mbar_arrive(&x_bar[q]);
              ok = __all_sync(0xffffffffu, mbar_wait(&x_bar[q], seq & 1, p.status, KS_TIMEOUT_PIPE));
              if (!ok) break;
              mref = fmaxf(rmax[r_in], rmax[128 + r_in]) * (NVF4 && !(e & ENTRY_F8) ? nvmul : 1.0f);
              if (!(mref > ATT_NO_REF)) mref = ATT_NO_REF;   // no visible key, or only NaN
              // rows of the ragged tail hold no data, and their scales belong to none: they never ask for another reference
              if (m_glob >= p.S) mref = -ATT_NO_REF;
              if (g == 0) {
                mrow[r_in] = mref;
                __syncwarp();
                if (lane == 0) mbar_arrive(&m_bar[q]);
              }
            } else {
              ok = __all_sync(0xffffffffu, mbar_wait(&m_bar[q], seq & 1, p.status, KS_TIMEOUT_PIPE));
              if (!ok) break;
              mref = mrow[r_in];
            }
          }
        }
      }
      if (do_epi) {
        // ---- epilogue of the previous item, number seq - 1: add the row's four partial sums, O / l ----
        const int seq_e = seq - 1;
        const float* xl = xrow + (seq_e & 1) * 1024 + r_in;
        ok = __all_sync(0xffffffffu, mbar_wait(&l_bar[q], seq_e & 1, p.status, KS_TIMEOUT_PIPE));
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(o_full, seq_e & 1, p.status, KS_TIMEOUT_MMA));
        if (!ok) break;
        tc_fence_after();
        float l_tot = ((xl[0] + xl[128]) + xl[256]) + xl[384];      // sum of the row
        float m_tot = 0.0f, ref_last = 0.0f, l_div = l_tot;         // quantised P.V: its maximum; fp16 P.V: the reference that O is at; what O is divided by
        if (PVQ) {
          m_tot = fmaxf(fmaxf(xl[512], xl[640]), fmaxf(xl[768], xl[896]));
        } else {
          // O is divided by a sum that has the largest P of each thread as fp16 has it: where one P carries the row, its rounding
          // cancels.  (The log2 denominator is that of the unrounded sum.)
          const float* rl = lref + (seq_e & 1) * 512 + r_in;
          l_div += ((xl[512] + xl[640]) + xl[768]) + xl[896];
          ref_last = fmaxf(fmaxf(rl[0], rl[128]), fmaxf(rl[256], rl[384]));
          const float ref_first = fminf(fminf(rl[0], rl[128]), fminf(rl[256], rl[384]));
          if (__builtin_expect(__any_sync(0xffffffffu, ref_first != ref_last), 0)) {     // some sums are at an earlier reference
            l_tot = l_div = 0.0f;
            _Pragma("unroll 1") for (int k = 0; k < 512; k += 128) {
              const float f = ex2(rl[k] - ref_last);
              l_tot += xl[k] * f;
              l_div += xl[512 + k] * f;
            }
            l_div += l_tot;
          }
        }
        const int mode = slots[epi_ls].mode;
        const bool tiles = (ROUTE ? slots[epi_ls].n_total : slots[epi_ls].n_own) > 0;
        const int m_glob = slots[epi_ls].qi * ATT_BM + r_in;
        const int head = slots[epi_ls].b * p.Hq + slots[epi_ls].h;
        const long long row = (long long)head * p.S + m_glob;
        // a share of an item: fp32 and the log2 denominator, into its slice of the partial results
        const int part = SPLIT ? slots[epi_ls].part : -1;
        const int item = SPLIT ? item_number(p.causal, p.Hq * p.B, nq, nq - 1 - slots[epi_ls].qi, head) : 0;
        const float ref = PVQ ? (mode == 1 ? m_redo + (LATE ? ATT_REF_Q : 0.0f) : ATT_REF_Q) : ref_last;
        const bool has_o = epi_part * 32 < p.D;     // this thread's 32 columns of O
        uint32_t o[32];
        if (tiles) {
          tmem_ld32p(lane_base + ATT_COL_O + (has_o ? epi_part * 32 : 0), o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) o[k] = 0;
        }
        tc_fence_before();
        mbar_arrive(o_free);
        // Routed, the first pass's maxima include those of tiles that were then done again in MXFP8 and may lie far above every score that
        // counts.  Such a maximum may be inside the window while what counts is below it: the row sum, which holds nothing else, shows it.
        // An item done again with those maxima as references may be so once more, with the maxima of that pass, which are exact.
        if (PVQ && (mode == 0 || ROUTE)) {
          const float over = m_tot - ref;           // rows of the ragged tail hold no data
          if (m_glob < p.S && m_tot != -INFINITY &&
              (over < ATT_WIN_LO_Q || (mode == 0 && (over > ATT_WIN_HI_Q || (ROUTE && l_tot < exp2_of((int)ATT_WIN_LO_Q)))))) {
            slots[epi_ls].redo = 1;
            if (p.range_flag) *p.range_flag = 1;
          }
          if (epi_part == 0) mslot[epi_ls * 128 + r_in] = m_tot == -INFINITY ? 0.0f : ceilf(m_tot);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&list_empty[epi_ls]);
        epi = false;
        if (m_glob < p.S) {
          float inv_l = l_tot > 0.0f ? 1.0f / l_div : 0.0f;
          float lse_row = 0.0f, w_prev = 0.0f;      // w_prev: weight of the earlier partial result (merge mode)
          if (p.lse || part >= 0) lse_row = l_tot > 0.0f ? ref + log2f(l_tot) : -INFINITY;
          if (p.acc_in) {
            // two normalised partial results over disjoint key sets combine with weights 2^(lse_i - lse),
            // lse = log2(2^lse_a + 2^lse_b); every thread of a row computes the same numbers
            const float la = p.lse_in[row];
            const float lm = fmaxf(la, lse_row);
            if (lm != -INFINITY) {
              const float ea = exp2f(la - lm), eb = exp2f(lse_row - lm);
              const float inv = 1.0f / (ea + eb);
              w_prev = ea * inv;
              inv_l *= eb * inv;
              lse_row = lm + log2f(ea + eb);
            }
          }
          // log2(sum_k exp2(S_k)): lets partial results be merged
          const long long prow = ((long long)part * (p.n_items - p.n_whole) + item - p.n_whole) * ATT_BM + r_in;
          if (part >= 0) { if (epi_part == 0) p.part_lse[prow] = lse_row; }
          else if (p.lse && epi_part == 0) p.lse[row] = lse_row;
          if (has_o) {
            const long long o_off = row * p.D + epi_part * 32;
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * inv_l);
            if (p.acc_in) {
              const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.acc_in) + o_off);
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float4 a = src[k];
                o[4 * k] = __float_as_uint(fmaf(a.x, w_prev, __uint_as_float(o[4 * k])));
                o[4 * k + 1] = __float_as_uint(fmaf(a.y, w_prev, __uint_as_float(o[4 * k + 1])));
                o[4 * k + 2] = __float_as_uint(fmaf(a.z, w_prev, __uint_as_float(o[4 * k + 2])));
                o[4 * k + 3] = __float_as_uint(fmaf(a.w, w_prev, __uint_as_float(o[4 * k + 3])));
              }
            }
            // a lane writes 32 columns of its own row, so that a store instruction touches 32 lines: the fewest and
            // widest stores there are (32 bytes a lane where the output is 32-byte aligned)
            if (part >= 0) {
              store_row<8>(p.part_o + prow * p.D + epi_part * 32, o, true);
            } else if (p.out_dtype == 0) {
              store_row<8>(reinterpret_cast<float*>(p.out) + o_off, o, p.out32);
            } else {
#pragma unroll
              for (int k = 0; k < 16; ++k) {
                const float x = __uint_as_float(o[2 * k]), y = __uint_as_float(o[2 * k + 1]);
                if (p.out_dtype == 1) o[k] = pack_f16x2(x, y);
                else { const __nv_bfloat162 hb = __floats2bfloat162_rn(x, y); o[k] = *reinterpret_cast<const uint32_t*>(&hb); }
              }
              store_row<4>(reinterpret_cast<uint16_t*>(p.out) + o_off, o, p.out32);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, ATT_TMEM_COLS);
}

// ---- merging partial attention results -----------------------------------------------------------
// Two softmax-normalised partial outputs over disjoint key sets, with their log2 denominators, combine to
// the result over the union: w_i = 2^(lse_i - lse), lse = log2(2^lse_a + 2^lse_b).  acc (fp32) and
// lse_acc are updated in place; one thread per 4 output elements.
__global__ void __launch_bounds__(256) attn_merge_kernel(float* acc, float* lse_acc, const void* part, int part_dtype,
                                                         const float* lse_part, long long rows, int D) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;     // index of a 4-element group
  const long long per_row = D / 4;
  if (i >= rows * per_row) return;
  const long long r = i / per_row;
  const float la = lse_acc[r], lb = lse_part[r];
  const float lm = fmaxf(la, lb);
  float wa = 0.0f, wb = 0.0f, lnew = -INFINITY;
  if (lm != -INFINITY) {
    const float ea = exp2f(la - lm), eb = exp2f(lb - lm);
    const float inv = 1.0f / (ea + eb);
    wa = ea * inv;
    wb = eb * inv;
    lnew = lm + log2f(ea + eb);
  }
  float4 a = reinterpret_cast<float4*>(acc)[i];
  float4 bv;
  if (part_dtype == 0) {
    bv = reinterpret_cast<const float4*>(part)[i];
  } else {
    const uint2 raw = reinterpret_cast<const uint2*>(part)[i];
    if (part_dtype == 1) {
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
      const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
      bv = make_float4(f0.x, f0.y, f1.x, f1.y);
    } else {
      const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      bv = make_float4(f0.x, f0.y, f1.x, f1.y);
    }
  }
  a.x = (wa == 0.0f ? 0.0f : a.x * wa) + (wb == 0.0f ? 0.0f : bv.x * wb);
  a.y = (wa == 0.0f ? 0.0f : a.y * wa) + (wb == 0.0f ? 0.0f : bv.y * wb);
  a.z = (wa == 0.0f ? 0.0f : a.z * wa) + (wb == 0.0f ? 0.0f : bv.z * wb);
  a.w = (wa == 0.0f ? 0.0f : a.w * wa) + (wb == 0.0f ? 0.0f : bv.w * wb);
  reinterpret_cast<float4*>(acc)[i] = a;
  __syncwarp();
  if (i % per_row == 0) lse_acc[r] = lnew;
}

// Results of the items that several runs share (SplitPlan): the partial results of a row combine with weights
// 2^(lse_i - max lse), as above.  A quarter warp per row, 16 or 8 columns a lane, so that a thread has 64 bytes of every part in
// flight: with a warp per row the kernel waited for its loads (156 items of 2 parts: 12.7 us, now 4; 32 items of 6: 6.7, now 4).
template <int W>                                    // columns of a lane: D / 8
__global__ void __launch_bounds__(128) attn_combine_kernel(const float* part_o, const float* part_lse, SplitPlan s, int n_items, void* out,
                                                           int out_dtype, int S) {
  grid_dependency_wait();
  constexpr int D = W * 8;
  const int n_shared = n_items - s.n_whole, k = blockIdx.x, item = s.n_whole + k;
  const int r_in = blockIdx.y * 16 + (threadIdx.x >> 3), sub = threadIdx.x & 7;
  const long long base = s.start(s.n_whole), it0 = s.start(item) - base;
  const int r = s.row_of(item), m = (s.nq - 1 - r) * ATT_BM + r_in;
  const int parts = (int)((it0 + s.row_tiles(r) - 1) / s.run_tiles - it0 / s.run_tiles) + 1;
  if (parts == 1 || m >= S) return;                 // (a single run has written the output itself)
  const long long stride = (long long)n_shared * ATT_BM, row0 = (long long)k * ATT_BM + r_in;
  const float* src = part_o + row0 * D + sub * 4;   // lane `sub` takes columns 32 c + 4 sub .. + 3
  float acc[W], den = 0.0f, lm = -1e30f;            // finite: a part without a visible key (lse -inf, O zero) weighs nothing
#pragma unroll
  for (int c = 0; c < W; ++c) acc[c] = 0.0f;
#pragma unroll 4
  for (int i = 0; i < parts; ++i) {                 // branch-free, so that the loads of several parts go out together
    const float l = __ldcg(part_lse + i * stride + row0);
    float4 v[W / 4];
#pragma unroll
    for (int c = 0; c < W / 4; ++c) v[c] = __ldcg(reinterpret_cast<const float4*>(src + i * stride * D + c * 32));
    const float nm = fmaxf(lm, l), w0 = exp2f(lm - nm), w1 = exp2f(l - nm);
    lm = nm;
    den = fmaf(den, w0, w1);
#pragma unroll
    for (int c = 0; c < W / 4; ++c) {
      acc[4 * c] = fmaf(acc[4 * c], w0, v[c].x * w1);
      acc[4 * c + 1] = fmaf(acc[4 * c + 1], w0, v[c].y * w1);
      acc[4 * c + 2] = fmaf(acc[4 * c + 2], w0, v[c].z * w1);
      acc[4 * c + 3] = fmaf(acc[4 * c + 3], w0, v[c].w * w1);
    }
  }
  const float inv = den > 0.0f ? 1.0f / den : 0.0f;
  const long long o = ((long long)s.head_of(item) * S + m) * D + sub * 4;
#pragma unroll
  for (int c = 0; c < W / 4; ++c) {
    const float x0 = acc[4 * c] * inv, x1 = acc[4 * c + 1] * inv, x2 = acc[4 * c + 2] * inv, x3 = acc[4 * c + 3] * inv;
    if (out_dtype == 0) {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + o + c * 32) = make_float4(x0, x1, x2, x3);
    } else {
      uint2 h;
      if (out_dtype == 1) {
        h = make_uint2(pack_f16x2(x0, x1), pack_f16x2(x2, x3));
      } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(x0, x1), b = __floats2bfloat162_rn(x2, x3);
        h = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
      }
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(out) + o + c * 32) = h;
    }
  }
}

// ---- V^T preparation: V [B,Hkv,Skv,D] (any 16-bit/32-bit float, strided) -> fp16 [B,Hkv,D,Skv_pad],
// keys beyond Skv zero-filled.  The reference casts V to fp16 on the host (ours/mxfp_attn_kernel.py:29-31);
// the transpose makes V the K-major B operand of P.V.
template <typename T>
__global__ void __launch_bounds__(256) prepare_vt_kernel(const T* v, __half* vt, int H, int Skv, int D, int Skv_pad,
                                                         long long vs_b, long long vs_h, long long vs_l) {
  __shared__ float tile[64][65];
  const int bh = blockIdx.z, b = bh / H, h = bh % H;
  const int s0 = blockIdx.x * 64, d0 = blockIdx.y * 64;
  const T* src = v + (long long)b * vs_b + (long long)h * vs_h;
  for (int i = threadIdx.x; i < 64 * 64; i += 256) {
    const int sl = i >> 6, dl = i & 63;
    const int s = s0 + sl, d = d0 + dl;
    tile[sl][dl] = (s < Skv && d < D) ? (float)src[(long long)s * vs_l + d] : 0.0f;
  }
  __syncthreads();
  __half* dst = vt + (long long)bh * D * Skv_pad;
  for (int i = threadIdx.x; i < 64 * 64; i += 256) {
    const int dl = i >> 6, sl = i & 63;
    const int s = s0 + sl, d = d0 + dl;
    if (d < D && s < Skv_pad) dst[(long long)d * Skv_pad + s] = __float2half_rn(tile[sl][dl]);
  }
}

// ---- band-rule precision map: FP8 iff |i + off/T - j| < band, else FP4; causal => tiles entirely above
// the diagonal are SKIP.  Tiles are T x T; `off` = Skv - S aligns queries to the end of the keys.
__global__ void route_band_kernel(uint8_t* map, int nq, int nk, int T, int causal, int band, int off, int S) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= nk) return;
  map += (long long)blockIdx.z * nq * nk;             // one copy of the map per (batch, head) when launched with grid.z > 1
  uint8_t v = (abs(i + off / T - j) < band) ? TILE_FP8 : TILE_FP4;
  if (causal) {
    const int last_q = min(S - 1, i * T + T - 1);       // last query row of the tile
    if (j * T > last_q + off) v = TILE_SKIP;
  }
  map[(long long)i * nk + j] = v;
}

}  // namespace mpsa

using namespace mpsa;

extern "C" int mpsa_route_band(void* map, int nq, int nk, int tile, int causal, int band, int S, int Skv, void* stream) {
  if (!map || nq <= 0 || nk <= 0 || tile <= 0 || band < 0) return set_error(MPSA_ERR_BAD_ARG, "route_band: bad argument");
  if (nq > 65535) return set_error(MPSA_ERR_UNSUPPORTED, "route_band: more than 65535 query tiles");
  dim3 grid((nk + 127) / 128, nq);
  route_band_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>((uint8_t*)map, nq, nk, tile, causal, band, Skv - S, S);
  return check_launch("route_band");
}

extern "C" int mpsa_attn_merge(void* acc, void* lse_acc, const void* part, int part_dtype, const void* lse_part,
                               long long rows, int D, void* stream) {
  if (!acc || !lse_acc || !part || !lse_part || rows <= 0)
    return set_error(MPSA_ERR_BAD_ARG, "attn_merge: null pointer or bad shape");
  if (D != 32 && D != 64 && D != 128)      // a row's threads must sit in one warp (in-place update of lse_acc)
    return set_error(MPSA_ERR_UNSUPPORTED, "attn_merge: head_dim must be 32, 64 or 128");
  if (part_dtype < 0 || part_dtype > 2) return set_error(MPSA_ERR_BAD_ARG, "attn_merge: part_dtype must be 0 (f32), 1 (f16) or 2 (bf16)");
  if (((uintptr_t)acc % 16) || ((uintptr_t)part % 16)) return set_error(MPSA_ERR_BAD_ARG, "attn_merge: 16-byte aligned buffers needed");
  const long long groups = rows * (D / 4);
  const long long blocks = (groups + 255) / 256;
  if (blocks > 0x7fffffffll) return set_error(MPSA_ERR_UNSUPPORTED, "attn_merge: too many rows");
  attn_merge_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((float*)acc, (float*)lse_acc, part, part_dtype,
                                                                     (const float*)lse_part, rows, D);
  return check_launch("attn_merge");
}

extern "C" int mpsa_prepare_vt(const void* v, int in_dtype, void* vt, int B, int H, int Skv, int D, int Skv_pad,
                               long long vs_b, long long vs_h, long long vs_l, void* stream) {
  if (!v || !vt || B <= 0 || H <= 0 || Skv <= 0 || D <= 0) return set_error(MPSA_ERR_BAD_ARG, "prepare_vt: bad argument");
  if (Skv_pad < Skv || Skv_pad % 8) return set_error(MPSA_ERR_BAD_ARG, "prepare_vt: Skv_pad must be >= Skv and a multiple of 8");
  if (B * H > 65535) return set_error(MPSA_ERR_UNSUPPORTED, "prepare_vt: B*H must be below 65536");
  if (in_dtype != 2 && (D == 64 || D == 128) && Skv_pad % 128 == 0 && !((uintptr_t)v % 16) && !((uintptr_t)vt % 16) && !((vs_b * 2) % 16) &&
      !((vs_h * 2) % 16) && !((vs_l * 2) % 16)) {
    PrepCall c;
    c.D = D;
    c.v.v = v; c.v.B = B; c.v.H = H; c.v.Skv = Skv; c.v.pitch = Skv_pad; c.v.vs_b = vs_b; c.v.vs_h = vs_h; c.v.vs_l = vs_l; c.v.vt16 = vt;
    return prep_launch(c, in_dtype, true, false, 1, (cudaStream_t)stream);
  }
  dim3 grid((Skv_pad + 63) / 64, (D + 63) / 64, B * H);
  cudaStream_t st = (cudaStream_t)stream;
  if (in_dtype == 0) prepare_vt_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)v, (__half*)vt, H, Skv, D, Skv_pad, vs_b, vs_h, vs_l);
  else if (in_dtype == 1) prepare_vt_kernel<__half><<<grid, 256, 0, st>>>((const __half*)v, (__half*)vt, H, Skv, D, Skv_pad, vs_b, vs_h, vs_l);
  else if (in_dtype == 2) prepare_vt_kernel<float><<<grid, 256, 0, st>>>((const float*)v, (__half*)vt, H, Skv, D, Skv_pad, vs_b, vs_h, vs_l);
  else return set_error(MPSA_ERR_BAD_ARG, "prepare_vt: in_dtype must be 0 (bf16), 1 (fp16) or 2 (fp32)");
  return check_launch("prepare_vt");
}

namespace mpsa {

int sm_count() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices];      // zero-initialised; a property of the device, the same for every thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

namespace {
struct AttnMaps { CUtensorMap q8, q4, k8, k4, vt, vt8, vt4; };

template <int PVQ, int NVF4, int ROUTE, int E4M3, int SPLIT = 0>
int launch_attn(int grid, size_t smem, cudaStream_t st, bool after_prep, const AttnMaps& m, const AttnParams& p) {
  auto kern = attn_fwd_kernel<PVQ, NVF4, ROUTE, E4M3, SPLIT>;
  // the opt-in for more than 48 KB of dynamic shared memory is a per-device attribute of the kernel
  if (!allow_smem<(((PVQ * 2 + NVF4) * 2 + ROUTE) * 2 + E4M3) * 2 + SPLIT>(kern, ATT_SMEM_MAX))
    return set_error(MPSA_ERR_LAUNCH, "attn_fwd: cannot reserve %d bytes of shared memory", ATT_SMEM_MAX);
  launch_dependent(kern, dim3(grid), ATT_THREADS, smem, st, after_prep, m.q8, m.q4, m.k8, m.k4, m.vt, m.vt8, m.vt4, p);
  return check_launch("attn_fwd");
}

// Whether to cut items into runs, from where on, and how long a run is; returns the number of partial slices (0: no cut).
// In tiles of work per CTA: without a cut the busiest CTA of the schedule has at least `whole`, the larger of the mean and
// k times the lightest of the (k - 1) * SMs + 1 heaviest items, for every k; with one it has the mean of what is cut.  A cut
// costs the combination (5 us), partial results in fp32 and one more item a CTA: with 12 tiles to save it breaks even (12
// heads of 1560 tokens, 26 tiles against 14: 29.6 us either way).  16 queries against 32768 keys, 32 heads on 148 SMs, 256
// tiles against 56: 195 -> 58 us; 512 queries, 256 against 221: 199 -> 187 us.  Short runs over light items lose (8 heads of
// 2500 tokens, causal, runs of 12 tiles in up to 12 items: 28 -> 48 us), parts with a CTA to themselves gain from 7 tiles on
// (16 queries of 2048 keys, 16 tiles against 4: 20.2 -> 16.4 us).
int split_choose(const AttnCall& c, int nq, int nk, int& n_whole, int& run_tiles, int& pad) {
  pad = 0;
  const int heads = c.B * c.Hq, n_items = nq * heads, sms = sm_count();
  const SplitPlan all = split_plan(heads, c.S, c.Skv, c.causal, 0, 1, 0);
  const long long total = all.start(n_items);
  long long whole = (total + sms - 1) / sms;
  for (long long k = 1; (k - 1) * sms < n_items; ++k) whole = std::max(whole, k * all.row_tiles((int)((k - 1) * sms) / heads));
  n_whole = n_items / sms * sms;
  // what is left over gets runs of at least SPLIT_MIN_RUN tiles; too little for that: one more wave joins it
  auto run_of = [&](int first) { return (total - all.start(first) + sms - 1) / sms; };
  if (n_whole > 0 && run_of(n_whole) < SPLIT_MIN_RUN) n_whole -= sms;
  run_tiles = (int)std::max<long long>(SPLIT_MIN_RUN, run_of(n_whole));
  const long long cut = (all.start(n_whole) + sms - 1) / sms + run_tiles;
  if (n_items * 2 <= sms) {
    // so few items that each gets CTAs of its own: equal parts, one a CTA, which saves the second item a CTA
    const int n = (int)all.row_tiles(0), k = std::min(sms / n_items, (n + SPLIT_MIN_OWN - 1) / SPLIT_MIN_OWN), run = (n + k - 1) / k;
    if (k > 1 && whole - run >= SPLIT_GAIN_OWN && run <= cut + SPLIT_GAIN - SPLIT_GAIN_OWN) {
      n_whole = 0; run_tiles = run; pad = (n + run - 1) / run * run;
      return pad / run + 1;
    }
  }
  if (n_whole == n_items || whole - cut < SPLIT_GAIN) { n_whole = n_items; run_tiles = 1; return 0; }
  return (int)((all.row_tiles(n_whole / heads) - 1) / run_tiles) + 2;
}
}  // namespace

long long attn_split_bytes(const AttnCall& c) {
  if (c.route || c.fp4_kind) return 0;
  const int nq = (c.S + ATT_BM - 1) / ATT_BM, nk = (c.Skv + ATT_BN - 1) / ATT_BN;
  if ((long long)nq * c.Hq * c.B >= (1ll << 30)) return 0;
  int n_whole, run_tiles, pad;
  const int parts = split_choose(c, nq, nk, n_whole, run_tiles, pad);
  return (long long)parts * ((long long)nq * c.Hq * c.B - n_whole) * ATT_BM * (c.D + 1) * 4;
}

int attn_forward(const AttnCall& call, cudaStream_t st) {
  AttnCall c = call;
  if (c.map || c.route || !c.uniform) c.need8 = c.need4 = true;
  // a format that is never selected is not loaded; its tensor maps need an address all the same
  if (!c.need8) { c.q8 = c.q4; c.q8_sf = c.q4_sf; c.k8 = c.k4; c.k8_sf = c.k4_sf; c.vt8 = c.vt4; c.v8_sf = c.v4_sf; }
  if (!c.need4) { c.q4 = c.q8; c.q4_sf = c.q8_sf; c.k4 = c.k8; c.k4_sf = c.k8_sf; c.vt4 = c.vt8; c.v4_sf = c.v8_sf; }
  if (!c.q8 || !c.q8_sf || !c.q4 || !c.q4_sf || !c.k8 || !c.k8_sf || !c.k4 || !c.k4_sf || !c.out || !c.status)
    return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: null pointer");
  if (c.pv_mode != 0 && c.pv_mode != 1) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: pv_mode must be 0 (fp16 P.V) or 1 (quantised P.V)");
  if (c.pv_mode == 0 && !c.vt) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: pv_mode 0 needs vt");
  if (c.pv_mode == 1 && (!c.vt8 || !c.v8_sf || !c.vt4 || !c.v4_sf)) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: pv_mode 1 needs vt8, v8_sf, vt4, v4_sf");
  if (c.B <= 0 || c.Hq <= 0 || c.Hkv <= 0 || c.S <= 0 || c.Skv <= 0) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: non-positive shape");
  if (c.Hq % c.Hkv) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: Hq must be a multiple of Hkv");
  if (c.D != 64 && c.D != 128) return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd: head_dim must be 64 or 128");
  if (c.out_dtype < 0 || c.out_dtype > 2) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: out_dtype must be 0 (f32), 1 (f16) or 2 (bf16)");
  if (c.fp8_fmt != 0 && c.fp8_fmt != 1) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: fp8_fmt must be 0 (E4M3) or 1 (E5M2)");
  if (c.fp4_kind != 0 && c.fp4_kind != 1) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: fp4_kind must be 0 (MXFP4) or 1 (NVFP4)");
  if ((c.acc_in != nullptr) != (c.lse_in != nullptr)) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: acc_in and lse_in go together");
  if (c.acc_in && (c.out_dtype != 0 || !c.lse || c.acc_in == c.out || c.lse_in == c.lse || ((uintptr_t)c.acc_in % 16)))
    return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: merging needs fp32 out, lse, a 16-byte aligned acc_in, and outputs distinct from the inputs");
  if (c.fp4_kind == 1 && !c.ts_q && !(c.fp4_scale > 0.0f)) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: NVFP4 needs a positive fp4_scale");
  if (c.causal && c.Skv < c.S) return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd: causal needs Skv >= S");
  const int nq = (c.S + ATT_BM - 1) / ATT_BM, nk = (c.Skv + ATT_BN - 1) / ATT_BN;
  if (nk > ATT_MAX_KTILES) return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd: at most %d keys", ATT_MAX_KTILES * ATT_BN);
  if (c.route && nk > ATT_MAX_KTILES / 2)           // the visit list holds the row's own tiles and as many promoted ones
    return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd_routed: at most %d key tiles", ATT_MAX_KTILES / 2);
  if (c.Skv_pad < c.Skv || c.Skv_pad % 128) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: Skv_pad must be a multiple of 128, at least Skv");
  const void* ptrs[] = {c.q8, c.q8_sf, c.q4, c.q4_sf, c.k8, c.k8_sf, c.k4, c.k4_sf, c.vt, c.vt8, c.v8_sf, c.vt4, c.v4_sf, c.out};
  for (const void* ptr : ptrs)
    if ((uintptr_t)ptr % 16) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: every tensor base must be 16-byte aligned");
  if ((long long)c.B * c.Hq * c.S >= (1ll << 31) || (long long)c.B * c.Hkv * c.Skv >= (1ll << 31))
    return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd: B*H*S must fit in 31 bits");
  const long long n_items = (long long)nq * c.Hq * c.B;
  if (n_items >= (1ll << 30)) return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd: too many query tiles");

  AttnMaps m;
  const uint64_t qrows = (uint64_t)c.B * c.Hq * c.S, krows = (uint64_t)c.B * c.Hkv * c.Skv, vrows = (uint64_t)c.B * c.Hkv * c.D;
  // an absent format's maps are copies of the other's (they are not dereferenced): encoding takes 0.4 us of the host's time each
  bool bad = false;
  if (c.need8) bad = make_tmap_2d_bytes(&m.q8, c.q8, ATT_DQK, qrows, ATT_DQK, 128, ATT_BM, CU_TENSOR_MAP_SWIZZLE_128B) ||
                     make_tmap_2d_bytes(&m.k8, c.k8, ATT_DQK, krows, ATT_DQK, 128, ATT_BN, CU_TENSOR_MAP_SWIZZLE_128B);
  if (c.need4) bad = bad || make_tmap_2d_bytes(&m.q4, c.q4, ATT_DQK / 2, qrows, ATT_DQK / 2, 64, ATT_BM, CU_TENSOR_MAP_SWIZZLE_64B) ||
                     make_tmap_2d_bytes(&m.k4, c.k4, ATT_DQK / 2, krows, ATT_DQK / 2, 64, ATT_BN, CU_TENSOR_MAP_SWIZZLE_64B);
  if (!c.need8) { m.q8 = m.q4; m.k8 = m.k4; }
  if (!c.need4) { m.q4 = m.q8; m.k4 = m.k8; }
  if (c.pv_mode == 0) {
    bad = bad || make_tmap_2d_b16(&m.vt, c.vt, c.Skv_pad, vrows, (uint64_t)c.Skv_pad * 2, 64, c.D, CU_TENSOR_MAP_SWIZZLE_128B);
    m.vt8 = m.vt4 = m.vt;
  } else {
    if (c.need8) bad = bad || make_tmap_2d_bytes(&m.vt8, c.vt8, c.Skv_pad, vrows, c.Skv_pad, 128, c.D, CU_TENSOR_MAP_SWIZZLE_128B);
    if (c.need4) bad = bad || make_tmap_2d_bytes(&m.vt4, c.vt4, c.Skv_pad / 2, vrows, c.Skv_pad / 2, 64, c.D, CU_TENSOR_MAP_SWIZZLE_64B);
    if (!c.need8) m.vt8 = m.vt4;
    if (!c.need4) m.vt4 = m.vt8;
    m.vt = m.vt8;
  }
  if (bad) return set_error(MPSA_ERR_LAUNCH, "attn_fwd: cuTensorMapEncodeTiled failed");

  AttnParams p;
  p.B = c.B; p.Hq = c.Hq; p.Hkv = c.Hkv; p.S = c.S; p.Skv = c.Skv; p.D = c.D; p.causal = c.causal; p.fp8_fmt = c.fp8_fmt;
  p.qk_steps8 = c.depth64 ? 2 : 4; p.qk_steps4 = c.depth64 ? 1 : 2;
  p.q8_sf = (const uint8_t*)c.q8_sf; p.q4_sf = (const uint8_t*)c.q4_sf;
  p.k8_sf = (const uint8_t*)c.k8_sf; p.k4_sf = (const uint8_t*)c.k4_sf;
  p.v8_sf = (const uint8_t*)c.v8_sf; p.v4_sf = (const uint8_t*)c.v4_sf; p.v_tiles = c.Skv_pad / 128;
  p.fp4_scale = c.fp4_scale; p.ts_q = (const float*)c.ts_q; p.ts_k = (const float*)c.ts_k;
  p.map = (const uint8_t*)c.map; p.map_sb = c.map_sb; p.map_sh = c.map_sh; p.band = c.band; p.uniform = c.uniform;
  p.out = c.out; p.out_dtype = c.out_dtype; p.lse = (float*)c.lse; p.acc_in = c.acc_in; p.lse_in = (const float*)c.lse_in;
  p.tau = c.tau; p.map_rw = (uint8_t*)c.map_rw; p.stat_out = (float*)c.stat_out; p.range_flag = c.range_flag; p.status = c.status;
  p.n_items = (int)n_items; p.group = c.Hq / c.Hkv; p.counter = c.counter;
  p.out32 = (uintptr_t)c.out % 32 == 0; p.load8 = c.need8; p.load4 = c.need4;
  p.list_cap = ((c.route ? 2 * nk : nk) + 7) & ~7;
  const int off_list = ATT_OFF_LIST + (c.pv_mode == 0 || c.route ? ATT_EXTRA_BYTES : 0);
  p.n_lists = std::min(ATT_MAX_SLOTS, (ATT_SMEM_MAX - 1024 - off_list) / (p.list_cap * 2));
  const size_t smem = off_list + (size_t)p.n_lists * p.list_cap * 2 + 1024;
  int parts = 0, n_whole = p.n_items, run_tiles = 1, pad = 0;
  if (c.partial) parts = split_choose(c, nq, nk, n_whole, run_tiles, pad);
  const long long n_shared = p.n_items - n_whole;
  const SplitPlan plan = split_plan(c.B * c.Hq, c.S, c.Skv, c.causal, n_whole, run_tiles, pad);
  p.n_whole = n_whole; p.run_tiles = run_tiles; p.run_pad = pad;
  p.n_work = n_whole + (int)((plan.start(p.n_items) - plan.start(n_whole) + run_tiles - 1) / run_tiles);
  p.part_o = (float*)c.partial;
  p.part_lse = p.part_o + parts * n_shared * ATT_BM * c.D;
  const int grid = std::min(p.n_work, sm_count());                     // one persistent CTA per SM
  const bool e4 = c.fp8_fmt == 0, dep = c.after_prep;
  int rc;
  if (parts > 0) {
    if (c.pv_mode == 0) rc = launch_attn<0, 0, 0, 0, 1>(grid, smem, st, dep, m, p);
    else rc = e4 ? launch_attn<1, 0, 0, 1, 1>(grid, smem, st, dep, m, p) : launch_attn<1, 0, 0, 0, 1>(grid, smem, st, dep, m, p);
  } else if (c.route) rc = e4 ? launch_attn<1, 0, 1, 1>(grid, smem, st, dep, m, p) : launch_attn<1, 0, 1, 0>(grid, smem, st, dep, m, p);
  else if (c.pv_mode == 0) rc = c.fp4_kind ? launch_attn<0, 1, 0, 0>(grid, smem, st, dep, m, p) : launch_attn<0, 0, 0, 0>(grid, smem, st, dep, m, p);
  else if (c.fp4_kind) rc = e4 ? launch_attn<1, 1, 0, 1>(grid, smem, st, dep, m, p) : launch_attn<1, 1, 0, 0>(grid, smem, st, dep, m, p);
  else rc = e4 ? launch_attn<1, 0, 0, 1>(grid, smem, st, dep, m, p) : launch_attn<1, 0, 0, 0>(grid, smem, st, dep, m, p);
  if (rc || parts == 0) return rc;
  launch_dependent(c.D == 64 ? attn_combine_kernel<8> : attn_combine_kernel<16>, dim3((unsigned)n_shared, ATT_BM / 16), 128, 0, st, true,
                   (const float*)p.part_o, (const float*)p.part_lse, plan, p.n_items, c.out, c.out_dtype, c.S);
  return check_launch("attn_combine");
}

}  // namespace mpsa

extern "C" int mpsa_attn_fwd(const void* q8, const void* q8_sf, const void* q4, const void* q4_sf, const void* k8,
                             const void* k8_sf, const void* k4, const void* k4_sf, const void* vt, const void* vt8,
                             const void* v8_sf, const void* vt4, const void* v4_sf, int pv_mode, const void* map,
                             long long map_sb, long long map_sh, void* out, int out_dtype, void* lse, int B, int Hq,
                             int Hkv, int S, int Skv, int D, int Skv_pad, int causal, int fp8_fmt, int fp4_kind,
                             float fp4_scale, int* range_flag, const void* acc_in, const void* lse_in, int* status,
                             void* stream) {
  if (!map) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd: null pointer");
  AttnCall c;
  c.q8 = q8; c.q8_sf = q8_sf; c.q4 = q4; c.q4_sf = q4_sf; c.k8 = k8; c.k8_sf = k8_sf; c.k4 = k4; c.k4_sf = k4_sf;
  c.vt = vt; c.vt8 = vt8; c.v8_sf = v8_sf; c.vt4 = vt4; c.v4_sf = v4_sf; c.pv_mode = pv_mode;
  c.map = map; c.map_sb = map_sb; c.map_sh = map_sh; c.out = out; c.out_dtype = out_dtype; c.lse = lse;
  c.B = B; c.Hq = Hq; c.Hkv = Hkv; c.S = S; c.Skv = Skv; c.D = D; c.Skv_pad = Skv_pad; c.causal = causal; c.fp8_fmt = fp8_fmt;
  c.fp4_kind = fp4_kind; c.fp4_scale = fp4_scale; c.range_flag = range_flag; c.acc_in = acc_in; c.lse_in = lse_in; c.status = status;
  return attn_forward(c, (cudaStream_t)stream);
}

// The forward with the online router inside it (no stand-alone statistic pass): MXFP8 inside the diagonal band, MXFP4
// elsewhere unless the MXFP4 statistic of a tile reaches tau x that of the row's first key tile, in which case the tile is
// done in MXFP8.  Quantised P.V, causal, one launch; `map` ends up as mpsa_route_online would have written it.
extern "C" int mpsa_attn_fwd_routed(const void* q8, const void* q8_sf, const void* q4, const void* q4_sf, const void* k8,
                                    const void* k8_sf, const void* k4, const void* k4_sf, const void* vt8, const void* v8_sf,
                                    const void* vt4, const void* v4_sf, void* map, int band, float tau, void* out,
                                    int out_dtype, void* lse, void* lse_final, void* stat, void* stat_scratch, int B, int Hq,
                                    int Hkv, int S, int Skv, int D, int Skv_pad, int fp8_fmt, int stages, int* range_flag,
                                    int* status, void* stream) {
  if (!map || !lse || !range_flag) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd_routed: null pointer");
  (void)stat_scratch;
  if (stages < 1 || stages > 15) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd_routed: stages is a mask of 1 (band map) and 2 (forward); 4 and 8 are accepted and ignored");
  if (band < 1) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd_routed: band must be at least 1");
  if (lse_final == lse) return set_error(MPSA_ERR_BAD_ARG, "attn_fwd_routed: lse_final must be another buffer than lse (or null)");
  const int nq = (S + ATT_BM - 1) / ATT_BM, nk = (Skv + ATT_BN - 1) / ATT_BN;
  AttnCall c;
  c.q8 = q8; c.q8_sf = q8_sf; c.q4 = q4; c.q4_sf = q4_sf; c.k8 = k8; c.k8_sf = k8_sf; c.k4 = k4; c.k4_sf = k4_sf;
  c.vt8 = vt8; c.v8_sf = v8_sf; c.vt4 = vt4; c.v4_sf = v4_sf; c.pv_mode = 1;
  c.map_sh = (long long)nq * nk; c.map_sb = c.map_sh * Hq; c.map_rw = map; c.band = band; c.route = true; c.tau = tau;
  c.out = out; c.out_dtype = out_dtype; c.lse = lse_final ? lse_final : lse; c.stat_out = stat;
  c.B = B; c.Hq = Hq; c.Hkv = Hkv; c.S = S; c.Skv = Skv; c.D = D; c.Skv_pad = Skv_pad; c.causal = 1; c.fp8_fmt = fp8_fmt;
  c.range_flag = range_flag; c.status = status;
  if (stages & 2) return attn_forward(c, (cudaStream_t)stream);       // writes the band map itself, row by row
  if (stages & 1) {
    if (B <= 0 || Hq <= 0 || nq <= 0 || nk <= 0 || nq > 65535 || (long long)B * Hq > 65535)
      return set_error(MPSA_ERR_UNSUPPORTED, "attn_fwd_routed: too many tiles or heads");
    route_band_kernel<<<dim3((nk + 127) / 128, nq, B * Hq), 128, 0, (cudaStream_t)stream>>>((uint8_t*)map, nq, nk, 128, 1, band, Skv - S, S);
    return check_launch("route_band");
  }
  return MPSA_OK;
}
