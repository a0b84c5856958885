// The whole attention call on 16-bit inputs behind one C entry: operand preparation and the forward, two launches (one more for the
// column sums of smooth K where prep_own_sums says so, two more for NVFP4, one more where keys are divided), every intermediate in one
// workspace of the caller.  A short call is bound by the host: seven to nine launches, as many allocations and a C call for each cost 174 -
// 192 us of its time where the GPU needs 14; through this entry and native.cpp a whole call takes 10.
// Also the reference's two-operand quantizers in one launch.
#include "../../include/mpsa.h"
#include "api_internal.h"
#include "prep.h"

namespace mpsa {
namespace {

struct Carver {                       // cuts the workspace into 256-byte aligned pieces; base null: only adds up
  uint8_t* base;
  long long used = 0;
  uint8_t* take(long long bytes) {
    const long long at = used;
    used = (used + bytes + 255) & ~255ll;
    return base ? base + at : nullptr;
  }
};

// Fills in both launches' parameters; returns the workspace size in bytes, or a negative code.
long long plan(const mpsa_attention_args& a, uint8_t* ws, PrepCall& pc, AttnCall& ac, bool& w8, bool& w4) {
  if (a.B <= 0 || a.Hq <= 0 || a.Hkv <= 0 || a.S <= 0 || a.Skv <= 0 || (a.D != 64 && a.D != 128))
    return set_error(MPSA_ERR_BAD_ARG, "attention: bad shape");
  if (a.in_dtype != 0 && a.in_dtype != 1) return set_error(MPSA_ERR_UNSUPPORTED, "attention: inputs must be bf16 or fp16");
  if (a.uniform < 0 || a.uniform > 2 || (a.route && a.uniform)) return set_error(MPSA_ERR_BAD_ARG, "attention: bad precision rule");
  const bool prepared = a.k == nullptr, nvfp4 = a.fp4_kind == 1;
  if (a.fp4_kind != 0 && (!nvfp4 || a.D != 128 || prepared || a.smooth_k || a.route || a.uniform))
    return set_error(MPSA_ERR_UNSUPPORTED, "attention: NVFP4 score tiles go with depth 128, the band rule and keys in 16 bits");
  const long long qrows = (long long)a.B * a.Hq * a.S, krows = (long long)a.B * a.Hkv * a.Skv;
  const long long nq = (a.S + 127) / 128, nk = (a.Skv + 127) / 128;
  const int pitch = prepared ? a.Skv_pad : (int)nk * 128;
  w8 = a.uniform != 2;
  w4 = a.uniform != 1 && !nvfp4;
  const bool q4 = w4 || nvfp4;
  const int sf4 = nvfp4 ? 1024 : 512;                   // bytes of FP4 scales per 128 rows
  Carver cv{ws};
  int* counter = (int*)cv.take(4);
  uint8_t* const words = nvfp4 ? cv.take(16) : nullptr; // two maxima, two tensor scales
  if (nvfp4) {
    pc.op[0].amax = (unsigned*)words; pc.op[1].amax = (unsigned*)words + 1;
    ac.ts_q = (float*)words + 2; ac.ts_k = (float*)words + 3;
  }
  PrepOperand& q = pc.op[0];
  q.x = a.q; q.B = a.B; q.H = a.Hq; q.L = a.S; q.xs_b = a.q_sb; q.xs_h = a.q_sh; q.xs_l = a.q_sl; q.s = a.q_scale;
  ac.q8 = q.fp8_codes = w8 ? cv.take(qrows * 128) : nullptr;
  ac.q8_sf = q.sf8_tiled = w8 ? cv.take((long long)a.B * a.Hq * nq * 512) : nullptr;
  ac.q4 = q.fp4_packed = q4 ? cv.take(qrows * 64) : nullptr;
  ac.q4_sf = q.sf4_tiled = q4 ? cv.take((long long)a.B * a.Hq * nq * sf4) : nullptr;
  // rows of 128 depth elements whatever D is: with D = 64 the upper half is never multiplied (depth64)
  q.o8_l = 128; q.o8_h = 128ll * a.S; q.o8_b = q.o8_h * a.Hq; q.p4_row = 64;
  if (prepared) {
    ac.k8 = a.k8; ac.k8_sf = a.k8_sf; ac.k4 = a.k4; ac.k4_sf = a.k4_sf;
    ac.vt = a.vt; ac.vt8 = a.vt8; ac.v8_sf = a.v8_sf; ac.vt4 = a.vt4; ac.v4_sf = a.v4_sf;
  } else {
    PrepOperand& k = pc.op[1];
    k.x = a.k; k.B = a.B; k.H = a.Hkv; k.L = a.Skv; k.xs_b = a.k_sb; k.xs_h = a.k_sh; k.xs_l = a.k_sl; k.s = 1.0f;
    ac.k8 = k.fp8_codes = w8 ? cv.take(krows * 128) : nullptr;
    ac.k8_sf = k.sf8_tiled = w8 ? cv.take((long long)a.B * a.Hkv * nk * 512) : nullptr;
    ac.k4 = k.fp4_packed = q4 ? cv.take(krows * 64) : nullptr;
    ac.k4_sf = k.sf4_tiled = q4 ? cv.take((long long)a.B * a.Hkv * nk * sf4) : nullptr;
    k.o8_l = 128; k.o8_h = 128ll * a.Skv; k.o8_b = k.o8_h * a.Hkv; k.p4_row = 64;
    k.own_sums = a.smooth_k && prep_own_sums((long long)a.B * a.Hkv, a.Skv, a.D) && a.fp8_fmt == 1;     // (no instances for E4M3)
    if (a.smooth_k && !k.own_sums) {
      k.nchunk = col_sum_chunks(a.Skv);
      k.part = (float*)cv.take((long long)a.B * a.Hkv * k.nchunk * a.D * 4);
    }
    PrepV& v = pc.v;
    v.v = a.v; v.B = a.B; v.H = a.Hkv; v.Skv = a.Skv; v.pitch = pitch; v.vs_b = a.v_sb; v.vs_h = a.v_sh; v.vs_l = a.v_sl;
    const long long vrows = (long long)a.B * a.Hkv * a.D, vtiles = (long long)a.B * a.Hkv * nk * 512;
    if (a.pv_mode == 0) {
      v.vt16 = cv.take(vrows * pitch * 2);
      ac.vt = v.vt16;
    } else {
      ac.vt8 = v.vt8 = w8 ? cv.take(vrows * pitch) : nullptr;
      ac.v8_sf = v.v8_sf = w8 ? cv.take(vtiles) : nullptr;
      ac.vt4 = v.vt4 = q4 ? cv.take(vrows * pitch / 2) : nullptr;
      ac.v4_sf = v.v4_sf = q4 ? cv.take(vtiles) : nullptr;
    }
  }
  ac.map_sh = nq * nk;
  ac.map_sb = ac.map_sh * a.Hq;
  if (a.route) ac.map_rw = cv.take((long long)a.B * a.Hq * nq * nk);
  pc.D = a.D;
  pc.zero0 = counter;
  pc.zero1 = a.range_flag;
  ac.counter = counter; ac.range_flag = a.range_flag;
  ac.pv_mode = a.pv_mode; ac.band = a.band; ac.uniform = a.uniform; ac.route = a.route != 0; ac.tau = a.tau;
  ac.need8 = w8; ac.need4 = q4; ac.fp4_kind = a.fp4_kind; ac.depth64 = a.D == 64;
  ac.out = a.out; ac.out_dtype = a.out_dtype; ac.B = a.B; ac.Hq = a.Hq; ac.Hkv = a.Hkv; ac.S = a.S; ac.Skv = a.Skv; ac.D = a.D;
  ac.Skv_pad = pitch; ac.causal = a.causal; ac.fp8_fmt = a.fp8_fmt; ac.status = a.status;
  ac.after_prep = true;
  if (const long long bytes = attn_split_bytes(ac)) ac.partial = cv.take(bytes);
  return cv.used;
}

}  // namespace
}  // namespace mpsa

using namespace mpsa;

extern "C" long long mpsa_attention_workspace(const mpsa_attention_args* a) {
  if (!a) return set_error(MPSA_ERR_BAD_ARG, "attention: null pointer");
  PrepCall pc;
  AttnCall ac;
  bool w8, w4;
  return plan(*a, nullptr, pc, ac, w8, w4);
}

extern "C" int mpsa_attention(const mpsa_attention_args* a, void* stream) {
  if (!a || !a->q || !a->out || !a->workspace || !a->status || (a->k && !a->v))
    return set_error(MPSA_ERR_BAD_ARG, "attention: null pointer");
  PrepCall pc;
  AttnCall ac;
  bool w8, w4;
  const long long need = plan(*a, (uint8_t*)a->workspace, pc, ac, w8, w4);
  if (need < 0) return (int)need;
  if (a->workspace_bytes < need || (uintptr_t)a->workspace % 256)
    return set_error(MPSA_ERR_BAD_ARG, "attention: the workspace must hold %lld bytes and be 256-byte aligned", need);
  if (!prep_operand_ok(pc.op[0], a->D) || (pc.op[1].x && !prep_operand_ok(pc.op[1], a->D)))
    return set_error(MPSA_ERR_BAD_ARG, "attention: q and k need 16-byte aligned bases and strides and a positive scale");
  if (pc.v.v && (((uintptr_t)a->v % 16) || (a->v_sb * 2) % 16 || (a->v_sh * 2) % 16 || (a->v_sl * 2) % 16))
    return set_error(MPSA_ERR_BAD_ARG, "attention: v needs a 16-byte aligned base and strides");
  const cudaStream_t st = (cudaStream_t)stream;
  if (pc.op[1].part)
    if (int rc = col_sums(a->k, a->in_dtype, a->B, a->Hkv, a->Skv, a->D, a->k_sb, a->k_sh, a->k_sl, (float*)pc.op[1].part, pc.op[1].nchunk, st))
      return rc;
  pc.after_sums = pc.op[1].part != nullptr;
  if (a->fp4_kind && cudaMemsetAsync(pc.op[0].amax, 0, 2 * sizeof(unsigned), st) != cudaSuccess) return check_launch("attention");
  if (int rc = prep_launch(pc, a->in_dtype, w8, w4, a->fp8_fmt == 0 ? 2 : 1, st)) return rc;
  for (int i = 0; a->fp4_kind && i < 2; ++i) {
    const PrepOperand& o = pc.op[i];
    if (int rc = nvfp4_quant(o.x, a->in_dtype, o.B, o.H, o.L, a->D, o.xs_b, o.xs_h, o.xs_l, o.s, o.amax, o.fp4_packed, o.sf4_tiled,
                             (float*)(i ? ac.ts_k : ac.ts_q), st))
      return rc;
  }
  return attn_forward(ac, st);
}

extern "C" int mpsa_quant_pair(const mpsa_quant_pair_args* a, void* stream) {
  if (!a || !a->x[0] || !a->x[1]) return set_error(MPSA_ERR_BAD_ARG, "quant_pair: null pointer");
  if (a->in_dtype != 0 && a->in_dtype != 1) return set_error(MPSA_ERR_UNSUPPORTED, "quant_pair: inputs must be bf16 or fp16");
  if (a->fp8_fmt < 0 || a->fp8_fmt > 2) return set_error(MPSA_ERR_BAD_ARG, "quant_pair: fp8_fmt must be 0 (MXFP4), 1 (E5M2) or 2 (E4M3)");
  PrepCall pc;
  pc.D = a->D;
  for (int i = 0; i < 2; ++i) {
    PrepOperand& o = pc.op[i];
    if (a->B <= 0 || a->H[i] <= 0 || a->L[i] <= 0 || !a->codes[i] || !a->scales[i])
      return set_error(MPSA_ERR_BAD_ARG, "quant_pair: null pointer or non-positive shape");
    o.x = a->x[i]; o.B = a->B; o.H = a->H[i]; o.L = a->L[i]; o.s = a->s[i];
    o.xs_b = a->x_sb[i]; o.xs_h = a->x_sh[i]; o.xs_l = a->x_sl[i];
    if ((uintptr_t)a->codes[i] % 16 || a->c_sb[i] % 16 || a->c_sh[i] % 16 || a->c_sl[i] % 16 || (uintptr_t)a->scales[i] % 4 ||
        !prep_operand_ok(o, a->D))
      return set_error(MPSA_ERR_UNSUPPORTED, "quant_pair: depth 64 or a multiple of 128, 16-byte aligned pointers and strides, positive scales");
    if (a->fp8_fmt == 0) {
      o.fp4_unpacked = (uint8_t*)a->codes[i]; o.o4_b = a->c_sb[i]; o.o4_h = a->c_sh[i]; o.o4_l = a->c_sl[i];
      o.sc4_rows = (uint8_t*)a->scales[i];
    } else {
      o.fp8_codes = (uint8_t*)a->codes[i]; o.o8_b = a->c_sb[i]; o.o8_h = a->c_sh[i]; o.o8_l = a->c_sl[i];
      o.sc8_rows = (uint8_t*)a->scales[i];
    }
  }
  return prep_launch(pc, a->in_dtype, a->fp8_fmt != 0, a->fp8_fmt == 0, a->fp8_fmt == 0 ? 1 : a->fp8_fmt, (cudaStream_t)stream);
}
