// The FP64 re-pick in pairs of FP32 numbers, certified (sm_103a).
//
// GB300's FP64 pipe runs at 1/64 of its FP32 rate, and a near-tie item evaluates up to four
// candidates at some 35 FP64 operations per aperture trace.  Here every number of that
// evaluation is an unevaluated sum of two FP32 numbers (hi + lo, about 48 bits; Dekker 1971,
// Knuth's TwoSum, products split by FMA), some 200 FP32 operations per trace and candidate:
// a tenth of the FP64 time.  The item's results are the pick among the candidates and the
// FP32 roundings of its semblance and stack, and the evaluation says whether it determines
// them: it returns true only where the candidates' semblances differ, and semblance and
// stack lie away from a rounding boundary of FP32, by more than a bound on both evaluations'
// errors, and no traveltime lies within it of the record's ends.  Then the FP64 evaluation
// gives the same pick and the same FP32 values; everywhere else the item takes that
// evaluation.
//
// Error bound, in units of U2 = 2^-48, worst case throughout (rounding errors of repeated
// geometries add up; where the samples cancel, the energy says nothing about the slopes):
//   t^2     (T + a m)^2 + b m^2 + c h: with S = (T + a m)^2 + |b m^2| + |c h|, the three
//           products, the sums and their inputs err by at most 21 S + |a m| (52 |T + a m| +
//           9 |a m|); the square root adds 14 t^2, FP64's own roundings less than 1.
//   t       half of that over t: w / 2 with w = (40 S + ...) / t + 20, the 20 for the
//           interpolation, which errs by |d_j| w / 2 + |v_j| for slope d_j and value v_j
//           (where t is that close to a sample, the slopes on both sides of it).
//   num_j   the traces' sum of that, sum |d_j| w <= sqrt(M sum (d_j w)^2), and (n + 6)^2 + 100
//           times sum |v_j| <= sqrt(M den) for the low parts of n additions per lane and the
//           lanes' (8 n sum |d_j| for the low parts of what is added).
//   den     sum |d_j| ((w + 12) |v_j| + 9 |d_j|), 7 den, and for the additions, normalised
//           after every trace, n (W^2 + 3 W) den, 6 W den and 16 W sum |v_j d_j|.
// Q, the sum of (d_j w)^2 over traces and window samples, is formed beside the numerators;
// sum |d_j| <= sqrt(M Q) / min w and sum |v_j d_j| w <= sqrt(Q den) follow from it.
//
// What bounds it: FP32 issue, and the one or two items in a hundred that the bound sends to
// FP64 (a quarter of the time).  GB300, re-pick alone, FP64 -> certified pairs: 64 CDPs of the
// 500 x 48 line 9.94 -> 1.74 ms, 128 CDPs with apertures of 50 to 2000 traces 17.9 -> 3.96,
// 48 such CDPs with 31 x 31 x 31 candidates 15.6 -> 3.60.
#pragma once

#include "plan_kernels.cuh"

namespace semb {

struct FF {
  float h, l;
};

__device__ __forceinline__ FF two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ FF quick_two_sum(float a, float b) {   // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF mul_ff(FF a, FF b) {   // not renormalised
  const float p = __fmul_rn(a.h, b.h);
  return {p, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -p)))};
}
__device__ __forceinline__ FF add_ff(FF a, FF b) {   // not renormalised
  const FF s = two_sum(a.h, b.h);
  return {s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ FF norm_ff(FF a) { return quick_two_sum(a.h, a.l); }
__device__ __forceinline__ FF div_ff(FF a, FF b) {
  const float q = __fdiv_rn(a.h, b.h);
  const float r = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
  return quick_two_sum(q, __fdiv_rn(r, b.h));
}
__device__ __forceinline__ FF ff_of(double v) {
  const float h = (float)v;
  return {h, (float)(v - (double)h)};
}

// Whether every value within `err` of the normalised a rounds to the FP32 number a.h.
__device__ __forceinline__ bool rounds_to_hi(FF a, float err) {
  const float m = fabsf(a.h);
  if (!(m > 1e-30f)) return false;
  // half the gap to the next FP32 number away from and towards zero
  const float up = 0.5f * (__int_as_float(__float_as_int(m) + 1) - m);
  const float dn = 0.5f * (m - __int_as_float(__float_as_int(m) - 1));
  const float off = a.h < 0.f ? -a.l : a.l;   // away from zero > 0
  return off + err < up && off - err > -dn;
}

constexpr float kU2 = 3.5527137e-15f;   // 2^-48

// The near-tie item's candidates ti[q] >= 0 (re-picked as repick_item does), all lanes of the
// warp.  True: bi, bs, bk are the FP64 evaluation's pick, semblance and stack as FP32 (bi
// 0x7fffffff: no valid candidate).
template <int W>
__device__ bool repick_ff(const RepickParams& R, int64_t e0, int64_t e1, int t0, const int (&ti)[kTopK], int lane, int& bi,
                          float& bs, float& bk) {
  const int napert = (int)(e1 - e0);
  const float T = (float)t0;
  // lane 3 q + d holds parameter d of candidate q in sample units
  FF par = {0.f, 0.f};
  if (lane < 3 * kTopK) {
    const int q = lane / 3, d = lane % 3;
    const int c = q == 0 ? ti[0] : q == 1 ? ti[1] : q == 2 ? ti[2] : ti[3];
    const double s = d == 0 ? R.idt : R.idt * R.idt;
    if (c >= 0) par = ff_of(R.cand64[3 * (int64_t)c + d] * s);
  }
  bool unsure = false;
  // lane q keeps candidate q's results
  FF my_sem = {0.f, 0.f}, my_stk = {0.f, 0.f};
  float my_err = 0.f, my_kerr = 0.f;
#pragma unroll 1
  for (int q = 0; q < kTopK; ++q) {
    const int c = q == 0 ? ti[0] : q == 1 ? ti[1] : q == 2 ? ti[2] : ti[3];
    if (c < 0) continue;
    FF pa, pb, pc;
    pa.h = __shfl_sync(0xffffffffu, par.h, 3 * q);
    pa.l = __shfl_sync(0xffffffffu, par.l, 3 * q);
    pb.h = __shfl_sync(0xffffffffu, par.h, 3 * q + 1);
    pb.l = __shfl_sync(0xffffffffu, par.l, 3 * q + 1);
    pc.h = __shfl_sync(0xffffffffu, par.h, 3 * q + 2);
    pc.l = __shfl_sync(0xffffffffu, par.l, 3 * q + 2);
    FF num[W], den = {0.f, 0.f};
    float Q = 0.f, wmin = 1e30f;   // see the error bound
    int M = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) num[j] = {0.f, 0.f};
    for (int64_t e = e0 + lane; e < e1; e += 32) {
      const float4 ga = __ldg(R.ap_ff + 2 * e), gb = __ldg(R.ap_ff + 2 * e + 1);   // (m, m^2), (h, -)
      const int tr = __ldg(R.ap_tr + e);
      // t^2 = (T + a m)^2 + b m^2 + c h
      const FF am = mul_ff(pa, FF{ga.x, ga.y});
      FF u = two_sum(T, am.h);
      u.l = __fadd_rn(u.l, am.l);
      const float P = __fmul_rn(u.h, u.h);
      const float Pl = __fmaf_rn(__fadd_rn(u.h, u.h), u.l, __fmaf_rn(u.h, u.h, -P));
      const FF bm = mul_ff(pb, FF{ga.z, ga.w}), ch = mul_ff(pc, FF{gb.x, gb.y});
      const FF s1 = two_sum(P, bm.h);
      const FF s2 = two_sum(s1.h, ch.h);
      const float ql = __fadd_rn(__fadd_rn(__fadd_rn(Pl, bm.l), ch.l), __fadd_rn(s1.l, s2.l));
      const float big = fmaxf(P, fmaxf(fabsf(bm.h), fabsf(ch.h)));
      if (!(s2.h * 2.f >= big) || !(s2.h > 1e-6f)) {   // cancelled, or negative: not certified
        unsure = true;
        continue;
      }
      const FF qq = quick_two_sum(s2.h, ql);
      // t = sqrt(q): g the FP32 root, corrected by the residual
      const float y = rsqrtf(qq.h), hy = 0.5f * y;
      float g = __fmul_rn(qq.h, y);
      g = __fmaf_rn(__fmaf_rn(-g, g, qq.h), hy, g);
      const float r = __fadd_rn(__fmaf_rn(-g, g, qq.h), qq.l);
      const float hg = __fmaf_rn(hy, __fmaf_rn(-g, __fadd_rn(hy, hy), 1.0f), hy);   // 1 / (2 g)
      const float corr = __fmul_rn(r, hg);
      const float aa = fabsf(am.h);
      const float w = fmaf(fmaf(40.f, P + fabsf(bm.h) + fabsf(ch.h), aa * fmaf(9.f, aa, 52.f * fabsf(u.h))), y, 20.f);
      // sample index and weight
      const float fy = __fadd_rz(g, 8388608.0f);
      int it = __float_as_int(fy) - 0x4B000000;
      FF x = two_sum(__fsub_rn(g, __fsub_rn(fy, 8388608.0f)), corr);
      if (x.h < 0.f || (x.h == 0.f && x.l < 0.f)) {
        --it;
        const FF z = two_sum(1.0f, x.h);
        x = two_sum(z.h, __fadd_rn(z.l, x.l));
      } else if (x.h > 1.0f || (x.h == 1.0f && x.l >= 0.f)) {
        ++it;
        x = two_sum(__fsub_rn(x.h, 1.0f), x.l);
      }
      // in range as t >= tau && t < ns - tau - 1: 0 <= rel <= last
      const int rel = it - R.tau, last = R.ns - 2 * R.tau - 2;
      if (rel < -1 || rel > last + 1) continue;
      // the error stays below 2^-25; a t that close to a sample may lie on either side of it
      const bool edge = !(x.h >= 6e-8f) || !(x.h <= 0.9999998f);
      if (!(w < 1.6e7f) || (edge && (rel < 1 || rel > last - 1))) {
        unsure = true;
        continue;
      }
      if (rel < 0 || rel > last) continue;
      wmin = fminf(wmin, w);
      const float* s = R.samples + (int64_t)tr * R.pitch + rel;
      if (edge) {   // the neighbouring intervals' slopes count as well
        float sd = 0.f;
#pragma unroll
        for (int j = -1; j <= W; ++j) sd += fabsf(__ldg(s + j + 1) - __ldg(s + j));
        Q = fmaf((float)W * (sd * w), sd * w, Q);
      }
      float sb = __ldg(s);
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float sa = sb;
        sb = __ldg(s + j + 1);
        const FF d = two_sum(sb, -sa);
        FF v = mul_ff(d, x);
        const FF vs = two_sum(sa, v.h);
        v = {vs.h, __fadd_rn(vs.l, v.l)};
        num[j] = add_ff(num[j], v);
        const float p = __fmul_rn(v.h, v.h);
        const FF sq = {p, __fmaf_rn(__fadd_rn(v.h, v.h), v.l, __fmaf_rn(v.h, v.h, -p))};
        den = add_ff(den, sq);
        const float dw = d.h * w;
        Q = fmaf(dw, dw, Q);
      }
      den = norm_ff(den);
      ++M;
    }
#pragma unroll
    for (int j = 0; j < W; ++j) num[j] = two_sum(num[j].h, num[j].l);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int j = 0; j < W; ++j)
        num[j] = add_ff(num[j], FF{__shfl_xor_sync(0xffffffffu, num[j].h, o), __shfl_xor_sync(0xffffffffu, num[j].l, o)});
      den = add_ff(den, FF{__shfl_xor_sync(0xffffffffu, den.h, o), __shfl_xor_sync(0xffffffffu, den.l, o)});
      Q += __shfl_xor_sync(0xffffffffu, Q, o);
      wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, o));
      M += __shfl_xor_sync(0xffffffffu, M, o);
    }
    if (M <= 0 || napert - M >= 2) continue;   // invalid (its results stay 0)
    den = norm_ff(den);
    if (!(den.h > 2e-13f) || !(den.h < 1e28f)) {
      // at or below the validity threshold, or near overflow: FP64 decides
      unsure = true;
      continue;
    }
    FF acsq = {0.f, 0.f}, lin = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const FF n = two_sum(num[j].h, num[j].l);
      acsq = norm_ff(add_ff(acsq, mul_ff(n, n)));
      lin = add_ff(lin, n);
      lin = two_sum(lin.h, lin.l);
    }
    const float mf = (float)M;
    const FF sem = div_ff(acsq, norm_ff(mul_ff(den, FF{mf, 0.f})));
    const FF stk = div_ff(lin, FF{(float)W * mf, 0.f});
    if (M >= (1 << 20) || !(acsq.h > 1e-30f)) unsure = true;   // W * M must be exact
    // the errors of the numerators (their norm, their sum), the energy, semblance and stack
    const float n1 = (float)((napert + 31) / 32) + 6.f;
    const float iw = 1.f / wmin, fw = (float)W;
    const float eq = fmaf(8.f * n1, iw, 0.5f) * sqrtf(mf * Q), ev = fmaf(n1, n1, 100.f) * sqrtf(mf * den.h);
    const float an = kU2 * (eq + sqrtf(fw) * ev) * rsqrtf(acsq.h);
    const float qd = Q / den.h;
    const float rd = kU2 * (fmaf(12.f + 16.f * fw, iw, 1.f) * sqrtf(qd) + 9.f * qd * iw * iw +
                            fmaf(n1, (float)(W * W + 3 * W), 6.f * fw + 107.f));
    if (!(an < 0.01f) || !(rd < 0.01f)) unsure = true;
    const float rel_e = 1.03f * (2.f * an + rd) + 80.f * kU2;
    const float stk_e =
        1.03f * kU2 * (sqrtf(fw) * eq + fw * ev + 40.f * sqrtf(fw * acsq.h)) / (fw * mf) + 1e-38f;
    if (lane == q) {
      my_sem = sem;
      my_stk = stk;
      my_err = sem.h * rel_e;
      my_kerr = stk_e;
    }
  }
  if (__any_sync(0xffffffffu, unsure)) return false;
  // the largest semblance; every other must lie below it by more than both errors
  int bq = -1;
  FF bsem = {0.f, 0.f};
#pragma unroll
  for (int q = 0; q < kTopK; ++q) {
    const FF s = {__shfl_sync(0xffffffffu, my_sem.h, q), __shfl_sync(0xffffffffu, my_sem.l, q)};
    if (s.h > 0.f && (bq < 0 || (s.h - bsem.h) + (s.l - bsem.l) > 0.f)) {   // both normalised
      bq = q;
      bsem = s;
    }
  }
  const float berr = __shfl_sync(0xffffffffu, my_err, max(bq, 0));
  bool tie = false;
#pragma unroll
  for (int q = 0; q < kTopK; ++q) {
    const FF s = {__shfl_sync(0xffffffffu, my_sem.h, q), __shfl_sync(0xffffffffu, my_sem.l, q)};
    const float er = __shfl_sync(0xffffffffu, my_err, q);
    if (q != bq && s.h > 0.f && !((bsem.h - s.h) + (bsem.l - s.l) > er + berr)) tie = true;
  }
  if (bq < 0) {
    bi = 0x7fffffff;
    return true;
  }
  const FF stk = {__shfl_sync(0xffffffffu, my_stk.h, bq), __shfl_sync(0xffffffffu, my_stk.l, bq)};
  const float kerr = __shfl_sync(0xffffffffu, my_kerr, bq);
  if (tie || !rounds_to_hi(bsem, berr) || !rounds_to_hi(stk, kerr)) return false;
  bi = bq == 0 ? ti[0] : bq == 1 ? ti[1] : bq == 2 ? ti[2] : ti[3];
  bs = bsem.h;
  bk = stk.h;
  return true;
}

}  // namespace semb
