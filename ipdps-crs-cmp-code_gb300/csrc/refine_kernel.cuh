// CRS refine kernels: the candidates semb_filter_kernel kept, evaluated with the direct
// search kernels' own FP32 arithmetic.
//
// Half a warp per (CDP, t0), one kept candidate per lane (all lanes walk the aperture
// together: the candidates of one t0 read nearby samples of the same trace, so the loads
// mostly share sectors).  The sums of a candidate are formed operation by operation as
// the direct kernel forms them, so that its semblance, stack and rank are the ones it
// would have there:
//
//   plain    the reference's sums in aperture order;
//   batched  the staged entries' arithmetic in the staging order: chunk by chunk, in-range
//            traces in aperture order, then the others from the last to the first, the
//            chunk's energy folded into the Kahan total; the central traces' sums (Z0)
//            apart.  Where a chunk ends follows from the windows of the candidate's
//            pass (plan_chunk), which each lane works out for its own pass as it goes.
//
// What bounds it: instruction issue, about 95 (batched) or 45 (plain) instructions per
// aperture trace and half warp.  Half warps because 4 to 12 candidates of a t0 are
// usually kept: with a whole warp per t0 the batched refine of 32 CDPs of the 500 x 48 line
// took 6.5 ms, with half warps 3.0 (the filter in front of it: 33).
#pragma once

#include "filter_kernel.cuh"

namespace semb {

struct RefineParams {
  KParams k;              // the direct configuration: stores, apertures, passes, capacity, outputs
  const int2* head;       // the filter's output
  const int2* pool;
  const float4* runs;     // the filter's candidate runs, rc slots each
  int rc;
  const int2* tasks;
  int ntasks;
  int na, nb, nc;
  int nbp;                // the direct configuration's slots per (A, C) group
  int z0;                 // batched: it shares the central traces' sums
};

constexpr int kRefineLanes = 16;   // lanes per (CDP, t0): a warp takes 32 / kRefineLanes of them

// The kept candidates of one item, dealt out to its lanes.
struct Kept {
  const int2* e = nullptr;
  int n = 0, total = 0, rc = 0;

  // false: the item fell back
  __device__ __forceinline__ bool load(const RefineParams& R, int64_t item) {
    const int2 h = __ldg(R.head + item);
    if (h.y < 0) return false;
    e = R.pool + h.x;
    rc = R.rc;
    n = h.y;
    for (int q = 0; q < n; ++q) total += __popc(__ldg(&e[q].y));
    return true;
  }
  // slot index (run * rc + slot) of candidate i, -1 past the end
  __device__ __forceinline__ int at(int i) const {
    if (i >= total) return -1;
    for (int q = 0; q < n; ++q) {
      const int2 v = __ldg(e + q);
      const int c = __popc(v.y);
      if (i < c) return v.x * rc + (int)__fns((unsigned)v.y, 0, i + 1);
      i -= c;
    }
    return -1;
  }
};

// Fold the candidates of an item's lanes (sem > 0, idx) into its running top-K (every lane
// of the item holds the same list).  All lanes of the warp take part.
template <int K>
__device__ __forceinline__ void fold_top(float sem, int idx, float stk, float (&fs)[K], int (&fi)[K], float (&fk)[K]) {
#pragma unroll 1
  for (int q = 0; q < K; ++q) {
    float bs = sem, bk = stk;
    int bi = idx;
#pragma unroll
    for (int o = kRefineLanes / 2; o > 0; o >>= 1) {
      const float os = __shfl_xor_sync(0xffffffffu, bs, o), ok = __shfl_xor_sync(0xffffffffu, bk, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(os, oi, bs, bi)) {
        bs = os;
        bi = oi;
        bk = ok;
      }
    }
    if (bi == idx) sem = 0.f, idx = 0x7fffffff;   // taken
    float cs = bs, ck = bk;
    int ci = bi;
#pragma unroll
    for (int p = 0; p < K; ++p) {
      if (cs > 0.f && better(cs, ci, fs[p], fi[p])) {
        const float ts = fs[p], tk = fk[p];
        const int ti = fi[p];
        fs[p] = cs;
        fi[p] = ci;
        fk[p] = ck;
        cs = ts;
        ci = ti;
        ck = tk;
      }
    }
  }
}

// ---- plain form -------------------------------------------------------------------

template <int W>
__global__ void __launch_bounds__(256) k_refine_plain(RefineParams R) {
  const KParams& P = R.k;
  const int lane = threadIdx.x & 31;
  constexpr int G = kRefineLanes, PER = kTB / (32 / G);   // warps per task
  const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= (int64_t)R.ntasks * PER) return;
  const int2 td = R.tasks[unit / PER];
  const int cdp = td.x, t0 = td.y + (int)(unit % PER) * (32 / G) + lane / G;
  const int64_t item = (int64_t)cdp * P.ns + min(t0, P.ns - 1);
  Kept kept;
  const bool live = t0 < P.ns && kept.load(R, item);
  const int most = __reduce_max_sync(0xffffffffu, live ? kept.total : 0);
  if (!__any_sync(0xffffffffu, live)) return;
  const int64_t e0 = P.ap_off[cdp], e1 = P.ap_off[cdp + 1];
  const int napert = (int)(e1 - e0);
  const float Tsec = __fmul_rn(P.dt, (float)t0);
  const float tau_lo = (float)P.tau, tau_hi = (float)(P.ns - P.tau - 1);
  float fs[1] = {0.f}, fk[1] = {0.f};
  int fi[1] = {0x7fffffff};
  for (int r0 = 0; r0 < most; r0 += G) {
    const int slot = live ? kept.at(r0 + lane % G) : -1;
    const int g = slot >= 0 ? max(__float_as_int(__ldg(&R.runs[slot].w)), 0) : 0;
    const int ia = g / (R.nc * R.nb), ib = (g / R.nc) % R.nb, ic = g % R.nc;
    const float4 cv = __ldg(P.cand + ((int64_t)ic * R.na + ia) * R.nb + ib);
    float num[W];
#pragma unroll
    for (int j = 0; j < W; ++j) num[j] = 0.f;
    float den = 0.f, lin = 0.f;
    int M = 0;
#pragma unroll 4
    for (int64_t e = e0; e < e1; ++e) {
      const float4 gm = __ldg(P.ap_geo + e);
      const int tr = __ldg(P.ap_tr + e);
      float t = __fadd_rn(Tsec, __fmul_rn(cv.x, gm.x));
      t = __fadd_rn(__fadd_rn(__fmul_rn(t, t), __fmul_rn(cv.y, gm.y)), __fmul_rn(cv.z, gm.z));
      t = (t < 0.0f) ? -1.0f : __fsqrt_rn(t);
      t = __fmul_rn(t, P.idt);
      const bool ok = (t >= tau_lo) && (t < tau_hi);
      const float y = __fadd_rz(t, 8388608.0f);
      const float x = ok ? __fsub_rn(t, __fsub_rn(y, 8388608.0f)) : 0.0f;
      // an out-of-range trace adds zeros: read its first samples with weight 0 instead
      const float* s = P.samples + (int64_t)tr * P.pitch + (ok ? __float_as_int(y) - 0x4B000000 - P.tau : 0);
      float s1 = ok ? __ldg(s) : 0.f;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float s0 = s1;
        s1 = ok ? __ldg(s + j + 1) : 0.f;
        const float v = __fadd_rn(__fmul_rn(__fsub_rn(s1, s0), x), s0);
        num[j] = __fadd_rn(num[j], v);
        den = __fadd_rn(den, __fmul_rn(v, v));
        lin = __fadd_rn(lin, v);
      }
      M += ok ? 1 : 0;
    }
    float acsq = 0.f;
#pragma unroll
    for (int j = 0; j < W; ++j) acsq = __fadd_rn(acsq, __fmul_rn(num[j], num[j]));
    const float mf = (float)M;
    const bool ok = slot >= 0 && (den > kEpsilonF) && (mf > kEpsilonF) && (napert - M < 2);
    const float sem = ok ? __fdiv_rn(acsq, __fmul_rn(den, mf)) : 0.f;
    const float stk = ok ? __fdiv_rn(lin, __fmul_rn((float)W, mf)) : 0.f;
    fold_top<1>(sem > 0.f ? sem : 0.f, sem > 0.f ? g : 0x7fffffff, stk, fs, fi, fk);
  }
  if (live && lane % G == 0) {
    const bool none = !(fs[0] > 0.f);
    P.ctr[item] = none ? 0 : fi[0];
    P.str[item] = none ? 0.f : fs[0];
    P.stk[item] = none ? P.stt00[cdp] : fk[0];
  }
}

// ---- batched form -----------------------------------------------------------------

// Window samples s_0 .. s_W at sample rel of trace tr as the staging converts them, and the
// differences of the LAY_PD entry.  CT: the differences take the scale in one rounding, as
// convert_chunk forms them; the central traces' sums (central_add) take them of two rounded
// samples.
template <int W, bool CT>
__device__ __forceinline__ void store_samples(const KParams& P, int tr, int rel, float (&s)[W + 8], float& d0,
                                              float& d2) {
  const int64_t at = (int64_t)tr * P.pitch + rel;
  if (P.storage == STORE_F32) {
#pragma unroll
    for (int u = 0; u <= W; ++u) s[u] = __ldg(P.samples + at + u);
    if (W == 3) {
      d0 = __fsub_rn(s[1], s[0]);
      d2 = __fsub_rn(s[3], s[2]);
    }
  } else {
    const float sc = __ldg(P.scale + tr);
    float h[W + 1];
#pragma unroll
    for (int u = 0; u <= W; ++u) {
      const uint32_t b = __ldg(P.samples16 + at + u);
      h[u] = P.storage == STORE_F16 ? half_bits_to_float(b) : __uint_as_float(b << 16);
      s[u] = __fmul_rn(h[u], sc);
    }
    if (W == 3) {
      d0 = CT ? __fmaf_rn(h[1], sc, -s[0]) : __fsub_rn(s[1], s[0]);
      d2 = CT ? __fmaf_rn(h[3], sc, -s[2]) : __fsub_rn(s[3], s[2]);
    }
  }
#pragma unroll
  for (int u = W + 1; u < W + 8; ++u) s[u] = 0.f;
}

// LAY: the direct kernel's accumulation layout (LAY_PD for w = 3, LAY_P2).
template <int W, int LAY>
__global__ void __launch_bounds__(256) k_refine_fast(RefineParams R) {
  const KParams& P = R.k;
  const int lane = threadIdx.x & 31;
  constexpr int G = kRefineLanes, PER = kTB / (32 / G);   // warps per task
  const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= (int64_t)R.ntasks * PER) return;
  const int2 td = R.tasks[unit / PER];
  const int cdp = td.x, t0 = td.y + (int)(unit % PER) * (32 / G) + lane / G;
  const int64_t item = (int64_t)cdp * P.ns + min(t0, P.ns - 1);
  Kept kept;
  const bool live = t0 < P.ns && kept.load(R, item);
  const int most = __reduce_max_sync(0xffffffffu, live ? kept.total : 0);
  if (!__any_sync(0xffffffffu, live)) return;
  const int64_t e0 = P.ap_off[cdp], e1 = P.ap_off[cdp + 1];
  const int napert = (int)(e1 - e0);
  int64_t zb = 0, ze = 0;
  if (R.z0) {
    const int2 zr = P.z0r[cdp];
    zb = e0 + zr.x;
    ze = zb + zr.y;
  }
  const float T = (float)t0;
  const float T_lo = __fmul_rn(P.dt, (float)td.y), T_hi = __fmul_rn(P.dt, (float)min(td.y + kTB - 1, P.ns - 1));
  const unsigned span = (unsigned)(P.ns - 2 * P.tau - 2);
  float fs[kTopK] = {}, fk[kTopK] = {};
  int fi[kTopK];
#pragma unroll
  for (int q = 0; q < kTopK; ++q) fi[q] = 0x7fffffff;
  for (int r0 = 0; r0 < most; r0 += G) {
    const int slot = live ? kept.at(r0 + lane % G) : -1;
    const float4 cv = __ldg(R.runs + max(slot, 0));
    const int g = max(__float_as_int(cv.w), 0);
    const int ia = g / (R.nc * R.nb), ib = (g / R.nc) % R.nb, ic = g % R.nc;
    const int pass = (int)((((int64_t)ic * R.na + ia) * R.nbp + ib) / P.cpp);
    float pb[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) pb[q] = __ldg(P.pass_bounds + 8 * (int64_t)pass + q);
    FastAcc<W, LAY> fa;
    fa.reset();
    float hi = 0.f, lo = 0.f;                                   // Kahan total and compensation
    float z_n0 = 0.f, z_n1 = 0.f, z_n2 = 0.f, z_den = 0.f;      // the central traces' sums
    int z_m = 0;
    auto traveltime = [&](const float4 gm) {
      const float u0 = fmaf(cv.x, gm.x, T);
      return sqrt_fast(fmaf(cv.y, gm.y, fmaf(u0, u0, cv.z * gm.z)));
    };
    auto add = [&](int tr, int rel, float x) {
      float s[W + 8], d0 = 0.f, d2 = 0.f;
      store_samples<W, true>(P, tr, rel, s, d0, d2);
      if constexpr (LAY == LAY_PD) fa.acc(make_float4(s[0], s[2], d0, d2), x);
      else fa.add_samples(s, x);
      fa.M += 1;
    };
    // the chunk under way: its first entry, staged samples, entries, position in the
    // planner's round of 32 traces
    int64_t c0 = e0;
    int used = 0, nent = 0, rpos = 0;
    bool back = false;
    auto close = [&](int64_t c1) {
      if (back) {   // the partly-in-range traces of entries c0 .. c1-1, last first
        for (int64_t k = c1 - 1; k >= c0; --k) {
          const float4 gm = __ldg(P.ap_geo + k);
          if (k >= zb && k < ze && gm.x == 0.f) continue;
          int wlo, whi;
          bool inr;
          float smin;
          if (!trace_window<METHOD_CRS>(pb, gm, T_lo, T_hi, P.idt, P.tau, P.ns, wlo, whi, inr, smin) || inr) continue;
          const float t = traveltime(gm);   // NaN below 0: out of range
          const float y = __fadd_rz(t, 8388608.0f);
          const int rel = __float_as_int(y) - (0x4B000000 + P.tau);
          if ((unsigned)rel <= span) add(__ldg(P.ap_tr + k), rel, t - (y - 8388608.0f));
        }
      }
      const float yv = fa.take_energy() - lo;
      const float tv = hi + yv;
      lo = (tv - hi) - yv;
      hi = tv;
      c0 = c1;
      used = nent = rpos = 0;
      back = false;
    };
    for (int64_t k = e0; k < e1; ++k) {
      const float4 gm = __ldg(P.ap_geo + k);
      const int tr = __ldg(P.ap_tr + k);
      int wlo = 0, whi = -1;
      bool inr = false, keep = false;
      if (k >= zb && k < ze && gm.x == 0.f) {
        // a central trace: as central_add
        const float t = sqrt_fast(fmaf(T, T, cv.z * gm.z));
        const float y = __fadd_rz(t, 8388608.0f);
        const int rel = __float_as_int(y) - (0x4B000000 + P.tau);
        if ((unsigned)rel <= span) {
          const float x = t - (y - 8388608.0f);
          float s[W + 8], d0 = 0.f, d2 = 0.f;
          store_samples<W, false>(P, tr, rel, s, d0, d2);
          const float w0 = fmaf(d0, x, s[0]), w2 = fmaf(d2, x, s[2]);
          const float s1 = s[0] + d0;
          const float w1 = fmaf(s[2] - s1, x, s1);
          z_n0 += w0;
          z_n1 += w1;
          z_n2 += w2;
          z_den = fmaf(w0, w0, z_den);
          z_den = fmaf(w1, w1, z_den);
          z_den = fmaf(w2, w2, z_den);
          z_m += 1;
        }
      } else {
        float smin;
        keep = trace_window<METHOD_CRS>(pb, gm, T_lo, T_hi, P.idt, P.tau, P.ns, wlo, whi, inr, smin);
      }
      if (keep) {
        const int len = (whi | 7) - (wlo & ~7) + 1;
        if (used + len > P.cap) close(k);
        used += len;
        nent += 1;
        if (inr) {
          const float t = traveltime(gm);
          const float y = __fadd_rz(t, 8388608.0f);
          const int rel = __float_as_int(y) - (0x4B000000 + P.tau);
          add(tr, min(max(rel, 0), (int)span), t - (y - 8388608.0f));
        } else {
          back = true;
        }
      }
      if (++rpos == 32) {
        rpos = 0;
        if (nent + 32 > kMaxChunk) close(k + 1);
      }
    }
    if (c0 < e1) close(e1);
    if constexpr (LAY == LAY_PD) {
      if (R.z0) {
        fa.add_sums(z_n0, z_n1, z_n2);
        fa.M += z_m;
      }
    }
    float acsq, lin;
    fa.sums(acsq, lin);
    const float den = R.z0 ? hi - lo + z_den : hi - lo;
    const float mf = (float)fa.M;
    const bool ok = slot >= 0 && (den > kEpsilonF) && (fa.M > 0) && (napert - fa.M < 2);
    const float sem = ok ? __fdividef(acsq, den * mf) : 0.f;
    const float stk = ok ? __fdividef(lin, (float)W * mf) : 0.f;
    fold_top<kTopK>(sem > 0.f ? sem : 0.f, sem > 0.f ? g : 0x7fffffff, stk, fs, fi, fk);
  }
  const int q = lane % G;
  if (live && q < kTopK) {
    const float os = q == 0 ? fs[0] : q == 1 ? fs[1] : q == 2 ? fs[2] : fs[3];
    const int oi = q == 0 ? fi[0] : q == 1 ? fi[1] : q == 2 ? fi[2] : fi[3];
    const float ok = q == 0 ? fk[0] : q == 1 ? fk[1] : q == 2 ? fk[2] : fk[3];
    P.top_sem[item * kTopK + q] = os;
    P.top_idx[item * kTopK + q] = os > 0.f ? oi : -1;
    P.top_stk[item * kTopK + q] = ok;
  }
}

}  // namespace semb
