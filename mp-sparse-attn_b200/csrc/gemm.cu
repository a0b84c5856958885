// Standalone block-scaled GEMM  C[M,N] = alpha * (A . sa) (B . sb)^T  for sm_100a.
//
// Counterpart of block_scaled_matmul_kernel (ours/block_scaled_matmul.py:154-267): A is [M, K] and
// B is [N, K], both K-major, quantised along K; the scales arrive as 512-byte 128x4 tiles
// [rows/128, K/vec/4, 32, 4, 4] (:45-66, :382-384).
//
// Design: persistent pairs of CTAs (cta_group::2).  A pair computes 256 x BN tiles of C: each CTA holds the accumulator of
// its own 128 rows and, in shared memory, its 128 rows of A and HALF of the tile's rows of B, which the tensor cores of both
// SMs read.  With one CTA per 128 x 256 tile an MMA of 32 bytes of K reads 12 KB of shared memory in its 128 cycles while TMA
// writes another 12 KB: 190 bytes per clock where an SM has 128, a ceiling of 0.67 of the tensor rate.  A pair needs 128.
// Measured, 8192^3 to bf16, 20 launches: MXFP8 489 -> 384 - 391 us (2.8 PFLOP/s), MXFP4 272 -> 195 - 200, NVFP4 300 -> 222 - 227.  A 256-column MXFP8 stage
// takes 600 cycles for 512 of tensor work at the 1.4 - 1.6 GHz that the power limit leaves; the FP4 modes also load a stage's
// 35 - 39 KB per SM in what would be 512 cycles.  1500 x 4096 x 4096 NVFP4: 27 -> 18 us; 180 x 6256 x 512: 9 -> 6 us, launch
// and first loads.
//   warp 0       TMA producer: 128-byte slabs of A and B (128-byte swizzle) and the scale tiles into a ring of stages; both CTAs'
//                copies report to the first CTA's barrier
//   warp 1       of the first CTA: tcgen05.cp of the scale tiles (each CTA's shared memory to its own TMEM), tcgen05.mma for both
//   warps 2, 3   of the first CTA: the scale copies of NVFP4, which has twelve per stage
//   warps 4-11   epilogue: a warp takes its 32 lanes and half of the columns into registers, hands the accumulator back,
//                and only then scales, converts and writes through shared memory with TMA stores, under the next tile's MMAs
// The ring runs on across tiles.  All hand-offs go through mbarriers with bounded waits.  When one expires the roles leave their
// loops; then, as at the ordinary end, the first CTA's producer waits for every copy that either producer has requested (drain.h), and
// every issuing thread for its own tensor operations, before a CTA gives up its memory.
//
//   mode 0  MXFP8  kind::mxf8f6f4  K=32 per instruction, one E8M0 scale per 32 elements
//   mode 1  MXFP4  kind::mxf4      K=64 per instruction, two E8M0 scales
//   mode 2  NVFP4  kind::mxf4nvf4  K=64 per instruction, four E4M3 scales (16-element blocks)
#include "api_internal.h"
#include "common.cuh"
#include "drain.h"
#include "tma_host.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <algorithm>

namespace mpsa {

constexpr int GEMM_BM = 256;                         // rows of a pair's tile
constexpr int GEMM_SLAB = 128;                       // bytes of K per stage and row
constexpr int GEMM_EPI_WARPS = 8;
constexpr int GEMM_THREADS = 128 + 32 * GEMM_EPI_WARPS;
constexpr int GEMM_STAGING = GEMM_EPI_WARPS * 2048;  // a 32-row, 64-byte box per epilogue warp
constexpr int GEMM_BARS = 320;                       // mbarriers, the TMEM slot and the peer's count
constexpr int GEMM_SMEM_MAX = 232448;
constexpr uint32_t GEMM_TMEM_COLS = 512;

// per-mode geometry, all compile-time: the single-thread loops must stay short
template <int MODE, int BN>
struct GemmShape {
  static constexpr int EPB = MODE == 0 ? 1 : 2;               // elements per byte
  static constexpr int K_STAGE = GEMM_SLAB * EPB;             // elements of K per stage
  static constexpr int CHUNK = MODE == 2 ? 64 : 128;          // K elements covered by one scale tile
  static constexpr int NC = K_STAGE / CHUNK;                  // scale tiles per stage and 128 rows: 1, 2, 4
  static constexpr int MPC = 4 / NC;                          // instructions per scale tile (4 instructions per stage)
  static constexpr int NT = BN / 128;                         // 128-row scale tiles of B
  static constexpr int A_BYTES = 128 * GEMM_SLAB, B_BYTES = BN / 2 * GEMM_SLAB;
  static constexpr int SFA_BYTES = NC * 512, SFB_BYTES = NT * NC * 512;
  static constexpr int LOADED = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;   // per CTA and stage
  static constexpr int STAGE_BYTES = (LOADED + 1023) / 1024 * 1024;
  static constexpr int NACC = BN == 256 ? 1 : 2;              // accumulators in TMEM: two only where the columns allow it
  static constexpr int SF_COL0 = NACC * BN;                   // scale sets behind them, one per stage
  static constexpr int SF_SET = 4 * NC * (1 + NT);
  static constexpr int FIT_SMEM = (GEMM_SMEM_MAX - GEMM_BARS - GEMM_STAGING) / STAGE_BYTES;
  static constexpr int FIT_TMEM = ((int)GEMM_TMEM_COLS - SF_COL0) / SF_SET;
  static constexpr int FIT = FIT_SMEM < FIT_TMEM ? FIT_SMEM : FIT_TMEM;
  static constexpr int STAGES = FIT < 8 ? FIT : 8;
  static constexpr int SMEM = STAGES * STAGE_BYTES + GEMM_STAGING + GEMM_BARS;
  static_assert(STAGES >= 4 && SMEM <= GEMM_SMEM_MAX, "the ring does not fit");
};

struct GemmParams {
  int M, N, batch;
  int n_stages_k;         // stages along K
  int nchunks;            // scale tiles along K
  int a_fmt, b_fmt;       // element format field of the instruction descriptor
  int mt, nt, n_tiles;    // tiles of a problem along M and N, of all problems
  int mrt, nrt;           // 128-row scale tiles of A and B per problem
  void* c; long long ldc; int out_dtype;   // 0 f32, 1 f16, 2 bf16, 3 fp8 e5m2
  bool tma_store;
  float alpha;
  int* status;
};

// ---- pairs of CTAs ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t leader_addr(const void* p) {        // the same shared-memory object in the first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_complete_tx(uint64_t* bar, uint32_t bytes) {      // counts bytes off as an arriving copy does
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// a TMA load into this CTA's shared memory that reports to a barrier of the pair (no multicast)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(m), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t base, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}
// arrive on the barrier at this offset in both CTAs when every tcgen05 operation issued so far by this thread is done
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3) : "memory");
}
// ... in this CTA only
__device__ __forceinline__ void tc_commit_pair_local(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_cp_sf_pair(uint32_t tmem, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(sdesc) : "memory");
}
template <int MODE>
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t acc) {
  if (MODE == 0)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc) : "memory");
  else if (MODE == 1)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(m), "r"(smem_u32(src)), "r"(x),
               "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_out16(float x, float y, int out_dtype) {
  if (out_dtype == 1) { const __half2 h = __floats2half2_rn(x, y); return *reinterpret_cast<const uint32_t*>(&h); }
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_out8(const float* v) {
  uint32_t r = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) r |= (uint32_t)__nv_cvt_float_to_fp8(v[i], __NV_SATFINITE, __NV_E5M2) << (8 * i);
  return r;
}

// Tiles in bands of GEMM_BAND row tiles, columns walked inside a band: the pairs that run at the same time then share the
// operand rows of a nearly square block of C (8192^3, one byte an element: 36 MB a round instead of 70; 406 -> 380 us, and
// 16 rows gained nothing at 8192^3 and lost a fifth at 4096^3).
constexpr int GEMM_BAND = 8;
__device__ __forceinline__ void gemm_tile(const GemmParams& p, int tile, int& mi, int& ni, int& z) {
  const int per = p.mt * p.nt;
  z = tile / per;
  const int rest = tile - z * per;
  const int band = rest / (GEMM_BAND * p.nt), in = rest - band * GEMM_BAND * p.nt;
  const int h = min(GEMM_BAND, p.mt - band * GEMM_BAND);
  ni = in / h;
  mi = band * GEMM_BAND + in - ni * h;
}

template <int MODE, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_block_scaled_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                         const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                         const __grid_constant__ CUtensorMap tmap_c, const GemmParams p) {
  using G = GemmShape<MODE, BN>;
  constexpr int ST = G::STAGES, NC = G::NC;
  constexpr bool SPLIT = MODE == 2;                      // scale copies on warps of their own
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* staging = smem + ST * G::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + GEMM_STAGING);    // [ST] first CTA: both CTAs' copies of the stage have landed
  uint64_t* empty = full + ST;                           // [ST] the stage's MMAs are done
  uint64_t* sf_ready = empty + ST;                       // [ST] SPLIT: the stage's scale tiles are in TMEM
  uint64_t* acc_full = sf_ready + ST;                    // [2]
  uint64_t* acc_free = acc_full + 2;                     // [2] first CTA: every epilogue warp of both CTAs has read the accumulator
  uint64_t* drained = acc_free + 2;                      // [3] the issuing threads' last operations are done
  uint64_t* peer_left = drained + 3;                     // first CTA: the other one's producer has left its count
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(peer_left + 1);
  int* peer_issued = reinterpret_cast<int*>(tmem_slot + 1);   // first CTA: stages that the other one has requested

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int KT = p.n_stages_k;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); mbar_init(&sf_ready[s], 2); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], 2 * GEMM_EPI_WARPS); }
    for (int s = 0; s < 3; ++s) mbar_init(&drained[s], 1);
    mbar_init(peer_left, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, GEMM_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                        // the peer's barriers are initialised
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dependency_wait();                                // the set-up above ran under the previous kernel on the stream
  grid_dependents_go();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a); tma_prefetch_desc(&tmap_b); tma_prefetch_desc(&tmap_sfa); tma_prefetch_desc(&tmap_sfb);
      bool ok = true;
      int s = 0, issued = 0;
      uint32_t e_par = 1;                                // parity that a never-used barrier already satisfies
      _Pragma("unroll 1") for (int tile = pair; tile < p.n_tiles && ok; tile += n_pairs) {
        int mi, ni, z;
        gemm_tile(p, tile, mi, ni, z);
        const int ya = z * p.M + mi * GEMM_BM + (int)rank * 128, yb = z * p.N + ni * BN + (int)rank * (BN / 2);
        // scale tiles: 4 rows of 128 bytes each, those of a 128-row tile one after the other along K
        int sfa_y = ((z * p.mrt + mi * 2 + (int)rank) * p.nchunks) * 4;
        int sfb_y = ((z * p.nrt + ni * G::NT) * p.nchunks) * 4;
        _Pragma("unroll 1") for (int kt = 0; kt < KT; ++kt) {
          ok = mbar_wait(&empty[s], e_par, p.status, KS_TIMEOUT_PIPE);
          if (!ok) break;
          uint8_t* st = smem + s * G::STAGE_BYTES;
          const uint32_t bar = leader_addr(&full[s]);
          if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * G::LOADED);
          tma_load_2d_pair(st + G::A_BYTES + G::B_BYTES, &tmap_sfa, bar, 0, sfa_y);
#pragma unroll
          for (int t = 0; t < G::NT; ++t)
            tma_load_2d_pair(st + G::A_BYTES + G::B_BYTES + G::SFA_BYTES + t * NC * 512, &tmap_sfb, bar, 0, sfb_y + t * p.nchunks * 4);
          tma_load_2d_pair(st, &tmap_a, bar, kt * GEMM_SLAB, ya);
          tma_load_2d_pair(st + G::A_BYTES, &tmap_b, bar, kt * GEMM_SLAB, yb);
          sfa_y += NC * 4;
          sfb_y += NC * 4;
          ++issued;
          if (++s == ST) { s = 0; e_par ^= 1; }
        }
      }
      // Neither CTA's shared memory is released while copies into it are in flight, whoever has given up: the first CTA, where they
      // all report, sees every requested stage land (at the ordinary end they have), and the other one leaves with it.
      if (rank == 1) {
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(leader_addr(peer_issued)), "r"(issued) : "memory");
        mbar_arrive_cluster(leader_addr(peer_left));
      } else {
        mbar_drain(peer_left, 0);
        const int other = *(volatile int*)peer_issued;
        _Pragma("unroll 1") for (int u = drain_first(issued, other, ST); u < drain_end(issued, other); ++u) {
          const DrainStep step = drain_step(u, issued, other);
          if (step == DRAIN_ARM) mbar_arrive_expect_tx(&full[u % ST], G::LOADED);
          else if (step == DRAIN_FILL) mbar_complete_tx(&full[u % ST], G::LOADED);
          mbar_drain(&full[u % ST], (u / ST) & 1);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (rank == 0 && elect_one()) {
      uint32_t idj[4];                                   // instruction descriptors of the four instructions of a stage
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (MODE == 0) idj[j] = idesc_with_sf_id(idesc_block_scaled(p.a_fmt, p.b_fmt, GEMM_BM, BN, 1), j, j);
        else if (MODE == 1) idj[j] = idesc_with_sf_id(idesc_block_scaled(1, 1, GEMM_BM, BN, 1), (j & 1) * 2, (j & 1) * 2);
        else idj[j] = idesc_block_scaled(1, 1, GEMM_BM, BN, 0);
      }
      const uint64_t ad0 = sdesc_kmajor_sw128(smem_u32(smem)), bd0 = sdesc_kmajor_sw128(smem_u32(smem + G::A_BYTES));
      const uint64_t sd0 = sdesc_sf_tile(smem_u32(smem + G::A_BYTES + G::B_BYTES));
      bool ok = true;
      int s = 0, acc = 0;
      uint32_t f_par = 0, a_par = 1;
      _Pragma("unroll 1") for (int tile = pair; tile < p.n_tiles && ok; tile += n_pairs) {
        ok = mbar_wait(&acc_free[acc], a_par, p.status, KS_TIMEOUT_PIPE);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem + acc * BN;
        int left = p.nchunks;
        _Pragma("unroll 1") for (int kt = 0; kt < KT; ++kt) {
          ok = mbar_wait(&full[s], f_par, p.status, KS_TIMEOUT_TMA);
          if (SPLIT && ok) ok = mbar_wait(&sf_ready[s], f_par, p.status, KS_TIMEOUT_TMA);
          if (!ok) break;
          tc_fence_after();
          const uint64_t step = (uint64_t)s * (G::STAGE_BYTES >> 4);
          const uint64_t ad = ad0 + step, bd = bd0 + step;
          const uint32_t sfa_t = tmem + G::SF_COL0 + s * G::SF_SET, sfb_t = sfa_t + 4 * NC;
          if (!SPLIT) {
            const uint64_t sd = sd0 + step;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              tc_cp_sf_pair(sfa_t + 4 * c, sd + c * 32);
#pragma unroll
              for (int t = 0; t < G::NT; ++t) tc_cp_sf_pair(sfb_t + 4 * (c * G::NT + t), sd + (NC + t * NC + c) * 32);
            }
          }
          const int n = left >= NC ? 4 : left * G::MPC;  // fewer instructions in the last stage of a K that does not fill it
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = j / G::MPC;                    // scale tile of this instruction
            if (j < n) mma_pair<MODE>(d, ad + 2 * j, bd + 2 * j, idj[j], sfa_t + 4 * c, sfb_t + 4 * G::NT * c, (kt > 0 || j > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty[s]);
          left -= NC;
          if (++s == ST) { s = 0; f_par ^= 1; }
        }
        if (!ok) break;
        tc_commit_pair(&acc_full[acc]);
        if (++acc == G::NACC) { acc = 0; a_par ^= 1; }
      }
      tc_commit_pair_local(&drained[0]);                 // the operands and the accumulators are in use until then
      mbar_drain(&drained[0], 0);
    }
  } else if (warp < 4) {
    // ------------------------------ scale copies (NVFP4) -----------------------
    // warp 2 the first two scale tiles of each operand and stage, warp 3 the others
    if (SPLIT && rank == 0 && elect_one()) {
      const uint64_t sd0 = sdesc_sf_tile(smem_u32(smem + G::A_BYTES + G::B_BYTES));
      const int c0 = (warp - 2) * (NC / 2);
      bool ok = true;
      int s = 0;
      uint32_t f_par = 0;
      _Pragma("unroll 1") for (int tile = pair; tile < p.n_tiles && ok; tile += n_pairs) {
        _Pragma("unroll 1") for (int kt = 0; kt < KT; ++kt) {
          // the stage was requested only after the MMAs that read this scale set the last time round were done
          ok = mbar_wait(&full[s], f_par, p.status, KS_TIMEOUT_TMA);
          if (!ok) break;
          tc_fence_after();
          const uint64_t sd = sd0 + (uint64_t)s * (G::STAGE_BYTES >> 4);
          const uint32_t sfa_t = tmem + G::SF_COL0 + s * G::SF_SET, sfb_t = sfa_t + 4 * NC;
#pragma unroll
          for (int k = 0; k < NC / 2; ++k) {
            const int c = c0 + k;
            tc_cp_sf_pair(sfa_t + 4 * c, sd + c * 32);
#pragma unroll
            for (int t = 0; t < G::NT; ++t) tc_cp_sf_pair(sfb_t + 4 * (c * G::NT + t), sd + (NC + t * NC + c) * 32);
          }
          tc_commit_pair_local(&sf_ready[s]);
          if (++s == ST) { s = 0; f_par ^= 1; }
        }
      }
      tc_commit_pair_local(&drained[warp - 1]);
      mbar_drain(&drained[warp - 1], 0);
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    const int q = warp & 3, half = (warp - 4) >> 2;      // TMEM lane quarter this warp may touch; half of the columns
    constexpr int HC = BN / 2;                           // columns of a warp
    uint8_t* stg = staging + (warp - 4) * 2048;
    int acc = 0;
    uint32_t a_par = 0;
    bool ok = true;
    _Pragma("unroll 1") for (int tile = pair; tile < p.n_tiles; tile += n_pairs) {
      int mi, ni, z;
      gemm_tile(p, tile, mi, ni, z);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], a_par, p.status, KS_TIMEOUT_MMA));
      if (!ok) break;
      tc_fence_after();
      uint32_t r[HC];
#pragma unroll
      for (int ch = 0; ch < HC / 32; ++ch)
        tmem_ld32(tmem + acc * BN + half * HC + ch * 32 + ((uint32_t)(q * 32) << 16), *reinterpret_cast<uint32_t(*)[32]>(r + ch * 32));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_addr(&acc_free[acc]));
      if (++acc == G::NACC) { acc = 0; a_par ^= 1; }
      const int row0 = mi * GEMM_BM + (int)rank * 128 + q * 32, col0 = ni * BN + half * HC;
      if (row0 >= p.M || col0 >= p.N) continue;
      if (p.tma_store) {
        // 64-byte boxes of 32 rows: a lane writes its row's 16-byte pieces with the 64-byte swizzle (no bank conflicts)
        uint8_t* line = stg + lane * 64;
        const int sw = (lane >> 1) & 3;
        auto begin_box = [&] {
          if (lane == 0) bulk_wait_read();               // the warp's previous box has left the staging area
          __syncwarp();
        };
        auto end_box = [&](int x) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (x < p.N) tma_store_3d(&tmap_c, stg, x, row0, z);
            bulk_commit();
          }
        };
#pragma unroll
        for (int i = 0; i < HC; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * p.alpha);
        const float* v = reinterpret_cast<const float*>(r);
        if (p.out_dtype == 0) {
#pragma unroll
          for (int bx = 0; bx < HC / 16; ++bx) {
            begin_box();
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(line + ((i ^ sw) << 4)) = make_uint4(r[bx * 16 + 4 * i], r[bx * 16 + 4 * i + 1], r[bx * 16 + 4 * i + 2], r[bx * 16 + 4 * i + 3]);
            end_box(col0 + bx * 16);
          }
        } else if (p.out_dtype == 3) {
#pragma unroll
          for (int bx = 0; bx < HC / 64; ++bx) {
            begin_box();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float* u = v + bx * 64 + 16 * i;
              *reinterpret_cast<uint4*>(line + ((i ^ sw) << 4)) = make_uint4(pack_out8(u), pack_out8(u + 4), pack_out8(u + 8), pack_out8(u + 12));
            }
            end_box(col0 + bx * 64);
          }
        } else {
#pragma unroll
          for (int bx = 0; bx < HC / 32; ++bx) {
            begin_box();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float* u = v + bx * 32 + 8 * i;
              *reinterpret_cast<uint4*>(line + ((i ^ sw) << 4)) =
                  make_uint4(pack_out16(u[0], u[1], p.out_dtype), pack_out16(u[2], u[3], p.out_dtype),
                             pack_out16(u[4], u[5], p.out_dtype), pack_out16(u[6], u[7], p.out_dtype));
            }
            end_box(col0 + bx * 32);
          }
        }
      } else {
        // C is not aligned for TMA: element stores
        const int row = row0 + lane, esz = p.out_dtype == 0 ? 4 : (p.out_dtype == 3 ? 1 : 2);
        if (row < p.M) {
          uint8_t* o = reinterpret_cast<uint8_t*>(p.c) + (((long long)z * p.M + row) * p.ldc + col0) * esz;
#pragma unroll
          for (int i = 0; i < HC; ++i) {
            const float v = __uint_as_float(r[i]) * p.alpha;
            if (col0 + i < p.N) {
              if (p.out_dtype == 0) reinterpret_cast<float*>(o)[i] = v;
              else if (p.out_dtype == 3) o[i] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E5M2);
              else reinterpret_cast<uint16_t*>(o)[i] = (uint16_t)pack_out16(v, 0.0f, p.out_dtype);
            }
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();                      // the staging area goes away with the CTA
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                        // neither CTA leaves while the other's MMAs or barriers may touch it
  if (warp == 1) tmem_dealloc_pair(tmem, GEMM_TMEM_COLS);
}

namespace {
struct GemmMaps { CUtensorMap a, b, sfa, sfb, c; };

template <int MODE, int BN>
int launch_gemm_shape(const GemmMaps& m, GemmParams& p, cudaStream_t st) {
  using G = GemmShape<MODE, BN>;
  auto kernel = gemm_block_scaled_kernel<MODE, BN>;
  if (!allow_smem<MODE * 2 + (BN == 256)>(kernel, G::SMEM))
    return set_error(MPSA_ERR_LAUNCH, "gemm_block_scaled: cannot reserve %d bytes of shared memory", G::SMEM);
  const int pairs = std::min(p.n_tiles, std::max(1, sm_count() / 2));
  launch_dependent(kernel, dim3(2 * pairs), GEMM_THREADS, G::SMEM, st, overlaps_previous(st), m.a, m.b, m.sfa, m.sfb, m.c, p);
  return check_launch("gemm_block_scaled");
}
}  // namespace

}  // namespace mpsa

using namespace mpsa;

static int launch_gemm(const void* a, const void* a_scale, const void* b, const void* b_scale, void* c, int batch, int M,
                       int N, int K, long long lda_bytes, long long ldb_bytes, long long ldc, int mode, int a_fmt, int b_fmt,
                       int out_dtype, float alpha, int* status, void* stream) {
  if (!a || !b || !a_scale || !b_scale || !c || !status)
    return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: null pointer");
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: non-positive shape");
  if (batch > 65535 || (long long)batch * M >= (1ll << 31) || (long long)batch * N >= (1ll << 31))
    return set_error(MPSA_ERR_UNSUPPORTED, "gemm_block_scaled: batch too large");
  if (mode < 0 || mode > 2) return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: mode must be 0 (mxfp8), 1 (mxfp4) or 2 (nvfp4)");
  if (out_dtype < 0 || out_dtype > 3) return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: out_dtype must be 0..3");
  const int chunk = mode == 2 ? 64 : 128;
  if (K % chunk != 0) return set_error(MPSA_ERR_UNSUPPORTED, "gemm_block_scaled: K must be a multiple of %d for this mode", chunk);
  if (mode == 0 && !((a_fmt == 0 || a_fmt == 1) && (b_fmt == 0 || b_fmt == 1)))
    return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: mxfp8 element formats are 0 (E4M3) or 1 (E5M2)");
  const int epb = mode == 0 ? 1 : 2;
  const long long kbytes = K / epb;
  if (((uintptr_t)a % 16) || ((uintptr_t)b % 16) || (lda_bytes % 16) || (ldb_bytes % 16) || lda_bytes < kbytes ||
      ldb_bytes < kbytes || ((uintptr_t)a_scale % 16) || ((uintptr_t)b_scale % 16))
    return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: operands need 16-byte aligned bases and row pitches >= K bytes");
  if (ldc < N) return set_error(MPSA_ERR_BAD_ARG, "gemm_block_scaled: ldc < N");
  GemmParams p;
  p.M = M; p.N = N; p.batch = batch; p.a_fmt = a_fmt; p.b_fmt = b_fmt;
  p.nchunks = K / chunk; p.n_stages_k = (K + GEMM_SLAB * epb - 1) / (GEMM_SLAB * epb);
  p.mt = (M + GEMM_BM - 1) / GEMM_BM; p.mrt = (M + 127) / 128; p.nrt = (N + 127) / 128;
  p.c = c; p.ldc = ldc; p.out_dtype = out_dtype; p.alpha = alpha; p.status = status;
  // Width of a pair's tile.  256 columns halve the traffic of A per product, 128 columns fill more pairs when there are few
  // tiles.  Cost of a schedule, in the time of a 128-column stage: rounds of tiles x (stages along K, and what a tile costs on
  // top of them).  The weights are measured with both widths forced: a 256-column stage takes 1.5 times as long (bound by its
  // loads and the power limit rather than by its products), and the single 256-column accumulator leaves a tile 4.5 stages of
  // its own where two 128-column ones leave 1.5 (1500 x 4096 x 4096 NVFP4, 2 rounds against 3: 19.8 and 17.9 us; 2048 x 2048 x
  // 8192 MXFP8, 1 round against 2: 27.2 and 29.6 us; 3000 x 5000 x 2048 MXFP8, 4 against 7: 33.0 and 33.5 us).
  const int pairs = std::max(1, sm_count() / 2);
  const int nc = mode == 0 ? 1 : (mode == 1 ? 2 : 4);
  auto cost = [&](int bn) {
    const long long rounds = ((long long)batch * p.mt * ((N + bn - 1) / bn) + pairs - 1) / pairs;
    return (double)rounds * (bn == 256 ? 1.5 * p.n_stages_k + 4.5 : p.n_stages_k + 1.5);
  };
  const int bn = cost(128) < cost(256) ? 128 : 256;
  p.nt = (N + bn - 1) / bn;
  const long long tiles = (long long)batch * p.mt * p.nt;
  if (tiles >= (1ll << 30)) return set_error(MPSA_ERR_UNSUPPORTED, "gemm_block_scaled: too many tiles");
  p.n_tiles = (int)tiles;
  const int esz = out_dtype == 0 ? 4 : (out_dtype == 3 ? 1 : 2);
  p.tma_store = (uintptr_t)c % 16 == 0 && (ldc * esz) % 16 == 0;
  GemmMaps m;
  bool bad = make_tmap_2d_bytes(&m.a, a, kbytes, (uint64_t)batch * M, lda_bytes, GEMM_SLAB, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
             make_tmap_2d_bytes(&m.b, b, kbytes, (uint64_t)batch * N, ldb_bytes, GEMM_SLAB, bn / 2, CU_TENSOR_MAP_SWIZZLE_128B) ||
             make_tmap_2d_bytes(&m.sfa, a_scale, 128, (uint64_t)batch * p.mrt * p.nchunks * 4, 128, 128, 4 * nc, CU_TENSOR_MAP_SWIZZLE_NONE) ||
             make_tmap_2d_bytes(&m.sfb, b_scale, 128, (uint64_t)batch * p.nrt * p.nchunks * 4, 128, 128, 4 * nc, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (p.tma_store) bad = bad || make_tmap_3d_store(&m.c, c, esz, N, M, batch, ldc * esz, (uint64_t)M * ldc * esz, 32);
  else m.c = m.a;                                        // not used
  if (bad) return set_error(MPSA_ERR_LAUNCH, "gemm_block_scaled: cuTensorMapEncodeTiled failed");
  const cudaStream_t st = (cudaStream_t)stream;
  if (mode == 0) return bn == 256 ? launch_gemm_shape<0, 256>(m, p, st) : launch_gemm_shape<0, 128>(m, p, st);
  if (mode == 1) return bn == 256 ? launch_gemm_shape<1, 256>(m, p, st) : launch_gemm_shape<1, 128>(m, p, st);
  return bn == 256 ? launch_gemm_shape<2, 256>(m, p, st) : launch_gemm_shape<2, 128>(m, p, st);
}

extern "C" int mpsa_gemm_block_scaled(const void* a, const void* a_scale, const void* b, const void* b_scale,
                                      void* c, int M, int N, int K, long long lda_bytes, long long ldb_bytes,
                                      long long ldc, int mode, int a_fmt, int b_fmt, int out_dtype, float alpha,
                                      int* status, void* stream) {
  return launch_gemm(a, a_scale, b, b_scale, c, 1, M, N, K, lda_bytes, ldb_bytes, ldc, mode, a_fmt, b_fmt, out_dtype, alpha,
                     status, stream);
}

extern "C" int mpsa_gemm_block_scaled_batched(const void* a, const void* a_scale, const void* b, const void* b_scale,
                                              void* c, int batch, int M, int N, int K, int mode, int a_fmt, int b_fmt,
                                              int out_dtype, float alpha, int* status, void* stream) {
  const long long kbytes = K / (mode == 0 ? 1 : 2);
  return launch_gemm(a, a_scale, b, b_scale, c, batch, M, N, K, kbytes, kbytes, N, mode, a_fmt, b_fmt, out_dtype, alpha,
                     status, stream);
}
