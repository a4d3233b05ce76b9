// CRS-DE on the GPU: the differential-evolution search over (A, B, C) of the
// reference's crs-ocl-de (README.md:86-106; its source is not in the reference).
// One warp per (CDP, t0) evolves a population of NP = na * nb * nc individuals
// started on the search grid, for ngen generations of DE/rand/1/bin (F = 0.5,
// CR = 0.9, trial kept when its semblance is >= the target's, parameters clamped
// to the search box), with counter-based random numbers keyed by (CDP, t0,
// generation, individual, slot), so that a run is reproducible and independent of
// the launch shape.  The population lives in shared memory; lane l owns individuals
// l, l + 32, ...  A semblance evaluation is the plain form's single-precision CRS
// operator (CRS/OpenMP/src/main.cpp:209-267 with real = float, no contraction) over
// the CDP's aperture in its order, so the search agrees bit for bit with the oracle's
// restatement of the same definition.
//
// What bounds it: the lanes of a warp read the samples of their own individuals, spread
// over a window of some hundred samples, so the loads conflict.  From global memory a load
// took up to one L1 cycle per 128-byte line of that window, 153 scheduler cycles per (trace,
// individual) in all.  The CTA (8 consecutive t0 of one CDP) therefore stages each trace's
// window over the whole search box by TMA, twice buffered, where a load costs its bank
// conflicts (about three), and the arithmetic goes two individuals per FP32x2 instruction
// with the plain kernel's square root (plain_kernel.cuh).  A CDP whose windows fit one
// buffer is staged once for all generations.  GB300: 8 CDPs x 500 samples, 180 individuals, 20
// generations, 10.95 -> 5.30 ms.
#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"
#include "plain_kernel.cuh"
#include "plan_kernels.cuh"

namespace semb {

constexpr int kDeMaxPop = 256;     // NP limit (8 individuals per lane)
constexpr int kDePerLane = kDeMaxPop / 32;
constexpr int kDeWarps = 8;        // warps (t0 samples of one CDP) per CTA
constexpr int kDeLongWarps = 4;    // warps (items) per CTA of k_crs_de_long


namespace {

__device__ __forceinline__ uint64_t de_mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t de_key(int cdp, int t0, int gen, int i, int slot) {
  uint64_t z = de_mix(((uint64_t)(uint32_t)cdp << 32) | (uint32_t)t0);
  z = de_mix(z ^ (((uint64_t)(uint32_t)gen << 32) | (uint32_t)i));
  return de_mix(z ^ (uint64_t)(uint32_t)slot);
}

// r[0..2]: distinct indices, all != i, drawn in turn among those not yet excluded
__device__ __forceinline__ void de_pick3(int cdp, int t0, int gen, int i, int np, int* r) {
  int ex[4] = {i, 0, 0, 0};
  int nex = 1;
  for (int q = 0; q < 3; ++q) {
    int v = (int)(de_key(cdp, t0, gen, i, q) % (uint64_t)(np - nex));
    int sorted[4] = {ex[0], ex[1], ex[2], ex[3]};
    for (int a = 1; a < nex; ++a)
      for (int b = a; b > 0 && sorted[b - 1] > sorted[b]; --b) {
        const int t = sorted[b];
        sorted[b] = sorted[b - 1];
        sorted[b - 1] = t;
      }
    for (int a = 0; a < nex; ++a)
      if (v >= sorted[a]) ++v;
    r[q] = v;
    ex[nex++] = v;
  }
}

// Shared-memory layout (bytes), shared by host and device: two mbarriers; two chunks'
// metadata and copy descriptors; the populations [kDeWarps][np][5] (a, b, c, sem, stk); two
// staging buffers of cap samples, each followed by a zero block.
struct DeLayout {
  size_t meta, src, pop, buf, buf_stride, total;
};

__host__ __device__ inline DeLayout de_layout(int cap, int np) {
  DeLayout L;
  L.meta = 128;
  L.src = L.meta + 2 * kMetaBytes;
  L.pop = L.src + 2 * (size_t)kMaxChunk * 16;
  L.buf = L.pop + align128((size_t)kDeWarps * np * 5 * 4);
  L.buf_stride = align128(((size_t)cap + kZeroSlots) * 4);
  L.total = L.buf + 2 * L.buf_stride;
  return L;
}

// P: stores, apertures, sampling, status; pass_bounds holds the search box.
template <int W>
__global__ void __launch_bounds__(kDeWarps * 32, 2) k_crs_de(DeParams R, KParams P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const DeLayout L = de_layout(P.cap, R.np);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);   // [2]
  auto meta_at = [&](int i) { return reinterpret_cast<ChunkMeta*>(smem_raw + L.meta + i * kMetaBytes); };
  auto src_at = [&](int i) { return reinterpret_cast<int4*>(smem_raw + L.src) + i * kMaxChunk; };
  auto buf_at = [&](int i) { return reinterpret_cast<float*>(smem_raw + L.buf + i * L.buf_stride); };
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  float (*pop)[5] = reinterpret_cast<float (*)[5]>(smem_raw + L.pop) + (size_t)wl * R.np;

  const int nblk = (R.ns + kDeWarps - 1) / kDeWarps;
  const int cdp = blockIdx.x / nblk, t0s = (blockIdx.x % nblk) * kDeWarps;
  const int t0 = min(t0s + wl, R.ns - 1);   // warps past the record repeat its last sample
  const int64_t e0 = R.ap_off[cdp], e1 = R.ap_off[cdp + 1];
  const int napert = (int)(e1 - e0);
  const float Tsec = __fmul_rn(R.dt, (float)t0);
  const float T_lo = P.dt * (float)t0s, T_hi = P.dt * (float)min(t0s + kDeWarps - 1, R.ns - 1);
  const int np = R.np;
  const int npair = ((np + 31) / 32 + 1) / 2;                           // pairs of individuals per lane
  const int cnt = max(0, min(kDePerLane, (np - lane + 31) / 32));      // individuals of this lane
  const int ngen = np >= 4 ? R.ngen : 0;

  for (int i = 0; i < 2; ++i)
    if (threadIdx.x < kZeroSlots) buf_at(i)[P.cap + threadIdx.x] = 0.f;
  if (threadIdx.x == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  constexpr int RP = kDePerLane / 2;
  const float nz = P.ns < 0 ? 0.0f : -0.0f;   // -0: see mul2
  const float2 k23 = make_float2(8388608.0f, 8388608.0f), km23 = make_float2(-8388608.0f, -8388608.0f);
  const float2 kNeg = make_float2(-1.0f, -1.0f), idt2 = make_float2(P.idt, P.idt), T2 = make_float2(Tsec, Tsec);
  const float tau_lo = (float)P.tau, tau_hi = (float)(P.ns - P.tau - 1);

  // The chunk stream: the aperture once per generation.  Warp 0 plans the chunk after the
  // current one into the other buffer while the warps compute; a chunk that is the whole
  // aperture stays.
  uint32_t phases = 0;   // bit i: parity of full[i]
  int cur = 0;
  bool whole = false;
  int64_t pos = e0;
  if (wl == 0) {
    plan_chunk<METHOD_CRS, FORM_PLAIN>(P, P.pass_bounds, e0, e1, T_lo, T_hi, meta_at(0), src_at(0));
    issue_chunk_copies(P, meta_at(0), src_at(0), buf_at(0), &full[0]);
  }
  __syncthreads();
  bool ready = false;   // the current chunk's copies have been waited for

  float2 pa[RP], pb[RP], pc[RP];   // the lane's trials, individuals lane + 64 p and lane + 64 p + 32
  float sem[kDePerLane], stk[kDePerLane];

  // Semblance and stack of the trials.  False: a copy did not land in time.
  auto eval = [&](bool more) -> bool {
    float2 num[RP][W], den[RP], lin[RP];
    uint32_t miss1 = 0, miss2 = 0;
    int n_tot = 0;
#pragma unroll
    for (int p = 0; p < RP; ++p) {
#pragma unroll
      for (int j = 0; j < W; ++j) num[p][j] = make_float2(0.f, 0.f);
      den[p] = lin[p] = make_float2(0.f, 0.f);
    }
    for (;;) {
      const ChunkMeta* meta = meta_at(cur);
      bool ok = true;
      if (!ready) {
        const uint32_t parity = (phases >> cur) & 1u;
        ok = wait_bar(&full[cur], parity);
        phases ^= 1u << cur;
        if (__syncthreads_or(!ok)) {
          if (threadIdx.x == 0) atomicOr(P.status, ST_TIMEOUT);
          // the late copy still writes this CTA's shared memory: wait for it (bounded); the
          // other buffer has none under way
          wait_bar(&full[cur], parity);
          return false;
        }
      }
      const int64_t next = pos + meta->consumed;
      whole = pos == e0 && next >= e1;
      ready = whole;
      if (wl == 0 && !whole && (next < e1 || more)) {
        const int64_t at = next < e1 ? next : e0;
        plan_chunk<METHOD_CRS, FORM_PLAIN>(P, P.pass_bounds, at, e1, T_lo, T_hi, meta_at(cur ^ 1), src_at(cur ^ 1));
        issue_chunk_copies(P, meta_at(cur ^ 1), src_at(cur ^ 1), buf_at(cur ^ 1), &full[cur ^ 1]);
      }
      const int n = meta->n;
      const uint32_t plane = smem_u32(buf_at(cur)), top = plane + 4u * (uint32_t)P.cap;
      for (int e = 0; e < n; ++e) {
        const float4 g = meta->geo[e];
        const float2 gx = make_float2(g.x, g.x), gy = make_float2(g.y, g.y), gz = make_float2(g.z, g.z);
        const uint32_t base = plane + 4u * (uint32_t)(__float_as_int(g.w) - P.tau) - 4u * 0x4B000000u;
        const bool inr = meta->raw[e] != 0;   // every point of the box in range
#pragma unroll
        for (int p = 0; p < RP; ++p) {
          if (p >= npair) break;
          const float2 u = __fadd2_rn(T2, mul2(pa[p], gx, nz));
          const float2 q = __fadd2_rn(__fadd2_rn(mul2(u, u, nz), mul2(pb[p], gy, nz)), mul2(pc[p], gz, nz));
          float2 x;
          uint32_t ax, ay;
          if (inr) {
            const float2 t = mul2(sqrt2_rn(q, nz), idt2, nz);
            const float2 y = __fadd2_rz(t, k23);
            x = __ffma2_rn(__fadd2_rn(y, km23), kNeg, t);   // t - floor(t), exact
            ax = min(__float_as_uint(y.x) * 4u + base, top);
            ay = min(__float_as_uint(y.y) * 4u + base, top);
          } else {
            // out of range: the zero block with weight 0 adds +0 and does not count
            const float rx = q.x < 0.0f ? -1.0f : __fsqrt_rn(q.x), ry = q.y < 0.0f ? -1.0f : __fsqrt_rn(q.y);
            const float2 t = make_float2(__fmul_rn(rx, P.idt), __fmul_rn(ry, P.idt));
            const bool okx = t.x >= tau_lo && t.x < tau_hi, oky = t.y >= tau_lo && t.y < tau_hi;
            const float2 y = __fadd2_rz(t, k23);
            x.x = okx ? __fsub_rn(t.x, __fsub_rn(y.x, 8388608.0f)) : 0.0f;
            x.y = oky ? __fsub_rn(t.y, __fsub_rn(y.y, 8388608.0f)) : 0.0f;
            ax = okx ? min(__float_as_uint(y.x) * 4u + base, top) : top;
            ay = oky ? min(__float_as_uint(y.y) * 4u + base, top) : top;
            const uint32_t off = (okx ? 0u : 1u << (2 * p)) | (oky ? 0u : 2u << (2 * p));
            miss2 |= miss1 & off;
            miss1 |= off;
          }
          float2 s0 = make_float2(lds32(ax), lds32(ay));
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const float2 s1 = make_float2(lds32(ax + 4u * (j + 1)), lds32(ay + 4u * (j + 1)));
            const float2 d = __ffma2_rn(s0, kNeg, s1);   // s1 - s0, rounded once
            const float2 v = __fadd2_rn(mul2(d, x, nz), s0);
            num[p][j] = __fadd2_rn(num[p][j], v);
            den[p] = __fadd2_rn(den[p], mul2(v, v, nz));
            lin[p] = __fadd2_rn(lin[p], v);
            s0 = s1;
          }
        }
      }
      n_tot += n;
      if (!whole) {
        __syncthreads();   // the buffer is free; the next chunk's metadata visible
        cur ^= 1;
        pos = next < e1 ? next : e0;
      }
      if (next >= e1) break;
    }
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q) {
      const int p = q >> 1;
      auto half = [&](float2 v) { return (q & 1) ? v.y : v.x; };
      float acsq = 0.f;
#pragma unroll
      for (int j = 0; j < W; ++j) acsq = __fadd_rn(acsq, __fmul_rn(half(num[p][j]), half(num[p][j])));
      const int M = n_tot - (int)((miss1 >> q) & 1);   // with a second miss the individual is invalid anyway
      const float mf = (float)M, dn = half(den[p]);
      const bool ok = dn > kEpsilonF && M > 0 && napert - M < 2 && !((miss2 >> q) & 1);
      sem[q] = ok ? __fdiv_rn(acsq, __fmul_rn(dn, mf)) : 0.f;
      stk[q] = ok ? __fdiv_rn(half(lin[p]), __fmul_rn((float)W, mf)) : 0.f;
    }
    return true;
  };
  auto set_par = [&](int q, const float (&v)[3]) {
    if (q & 1) {
      pa[q >> 1].y = v[0];
      pb[q >> 1].y = v[1];
      pc[q >> 1].y = v[2];
    } else {
      pa[q >> 1].x = v[0];
      pb[q >> 1].x = v[1];
      pc[q >> 1].x = v[2];
    }
  };
  auto keep = [&](int q) {
    const int i = lane + 32 * q;
    const int p = q >> 1;
    pop[i][0] = (q & 1) ? pa[p].y : pa[p].x;
    pop[i][1] = (q & 1) ? pb[p].y : pb[p].x;
    pop[i][2] = (q & 1) ? pc[p].y : pc[p].x;
    pop[i][3] = sem[q];
    pop[i][4] = stk[q];
  };

  // generation 0: the grid (a slot without an individual repeats the first)
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q) {
    const int i = q < cnt ? lane + 32 * q : 0;
    const float v[3] = {R.grid[3 * i], R.grid[3 * i + 1], R.grid[3 * i + 2]};
    set_par(q, v);
  }
  if (!eval(ngen > 0)) return;
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q)
    if (q < cnt) keep(q);
  __syncwarp();

  for (int gen = 1; gen <= ngen; ++gen) {
    // trials from the previous generation's population
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q) {
      if (q >= cnt) continue;
      const int i = lane + 32 * q;
      int r[3];
      de_pick3(cdp, t0, gen, i, np, r);
      const int jrand = (int)(de_key(cdp, t0, gen, i, 3) % 3u);
      float tr[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float u = __fmul_rn((float)(de_key(cdp, t0, gen, i, 4 + d) >> 40), 1.0f / 16777216.0f);
        float v = pop[i][d];
        if (u < 0.9f || d == jrand) v = __fadd_rn(pop[r[0]][d], __fmul_rn(0.5f, __fsub_rn(pop[r[1]][d], pop[r[2]][d])));
        tr[d] = v < R.lo[d] ? R.lo[d] : (v > R.hi[d] ? R.hi[d] : v);
      }
      set_par(q, tr);
    }
    if (!eval(gen < ngen)) return;
    __syncwarp();   // every lane has read the population
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q)
      if (q < cnt && sem[q] >= pop[lane + 32 * q][3]) keep(q);
    __syncwarp();
  }

  // the best individual (largest semblance, lowest index on ties)
  float bs = 0.f;
  int bi = 0x7fffffff;
  for (int q = 0; q < cnt; ++q) {
    const int i = lane + 32 * q;
    if (pop[i][3] > bs) {
      bs = pop[i][3];
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float os = __shfl_xor_sync(0xffffffffu, bs, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (os > bs || (os == bs && oi < bi)) {
      bs = os;
      bi = oi;
    }
  }
  if (lane == 0 && t0s + wl < R.ns) {
    const int64_t o = (int64_t)cdp * R.ns + t0;
    if (bi == 0x7fffffff || !(bs > 0.f)) {
      R.a[o] = R.grid[0];
      R.b[o] = R.grid[1];
      R.c[o] = (float)((double)R.grid[2] / 1e6);
      R.str[o] = 0.f;
      R.stk[o] = R.stt00[cdp];
    } else {
      R.a[o] = pop[bi][0];
      R.b[o] = pop[bi][1];
      R.c[o] = (float)((double)pop[bi][2] / 1e6);
      R.str[o] = bs;
      R.stk[o] = pop[bi][4];
    }
  }
}

// Semblance and stack of up to kDePerLane parameter triples of this lane at t0,
// in single precision with the reference's operation order, samples from global memory.
template <int W>
__device__ void de_eval(const DeParams& R, int64_t e0, int64_t e1, float Tsec, const float (*par)[3], int cnt,
                        float* sem, float* stk) {
  float num[kDePerLane][W], den[kDePerLane], lin[kDePerLane];
  int M[kDePerLane], err[kDePerLane];
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q) {
#pragma unroll
    for (int j = 0; j < W; ++j) num[q][j] = 0.f;
    den[q] = 0.f;
    lin[q] = 0.f;
    M[q] = 0;
    err[q] = 0;
  }
  for (int64_t e = e0; e < e1; ++e) {
    const float4 g = __ldg(R.ap_geo + e);
    const float* row = R.samples + (int64_t)__ldg(R.ap_tr + e) * R.pitch;
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q) {
      if (q >= cnt) continue;
      float t = __fadd_rn(Tsec, __fmul_rn(par[q][0], g.x));
      t = __fadd_rn(__fadd_rn(__fmul_rn(t, t), __fmul_rn(par[q][1], g.y)), __fmul_rn(par[q][2], g.z));
      t = (t < 0.0f) ? -1.0f : __fsqrt_rn(t);
      const float ts = __fmul_rn(t, R.idt);
      // (int) truncation; NaN or out of the int range counts as out of range
      const bool fin = ts > -2147483648.0f && ts < 2147483647.0f;
      const int it = fin ? (int)ts : 0;
      const float x = __fsub_rn(ts, (float)it);
      if (fin && it - R.tau >= 0 && it + R.tau + 1 < R.ns) {
        const float* s = row + (it - R.tau);
        float s1 = __ldg(s);
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const float s0 = s1;
          s1 = __ldg(s + j + 1);
          const float v = __fadd_rn(__fmul_rn(__fsub_rn(s1, s0), x), s0);
          num[q][j] = __fadd_rn(num[q][j], v);
          den[q] = __fadd_rn(den[q], __fmul_rn(v, v));
          lin[q] = __fadd_rn(lin[q], v);
        }
        ++M[q];
      } else {
        ++err[q];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q) {
    if (q >= cnt) continue;
    float acsq = 0.f;
#pragma unroll
    for (int j = 0; j < W; ++j) acsq = __fadd_rn(acsq, __fmul_rn(num[q][j], num[q][j]));
    const float mf = (float)M[q];
    const bool ok = (den[q] > kEpsilonF) && (M[q] > 0) && (err[q] < 2);
    sem[q] = ok ? __fdiv_rn(acsq, __fmul_rn(den[q], mf)) : 0.f;
    stk[q] = ok ? __fdiv_rn(lin[q], __fmul_rn((float)W, mf)) : 0.f;
  }
}

// Records too long for the staging buffers (ns above about 23,000): the same search, one warp
// per (CDP, t0), samples from global memory.
template <int W>
__global__ void __launch_bounds__(kDeLongWarps * 32) k_crs_de_long(DeParams R) {
  __shared__ float pop[kDeLongWarps][kDeMaxPop][5];   // a, b, c, sem, stk
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int64_t item = (int64_t)blockIdx.x * kDeLongWarps + wl;
  if (item >= (int64_t)R.ncdps * R.ns) return;
  const int cdp = (int)(item / R.ns);
  const int t0 = (int)(item - (int64_t)cdp * R.ns);
  const int64_t e0 = R.ap_off[cdp], e1 = R.ap_off[cdp + 1];
  const float Tsec = __fmul_rn(R.dt, (float)t0);
  float (*P)[5] = pop[wl];
  const int np = R.np;
  const int cnt = max(0, min(kDePerLane, (np - lane + 31) / 32));   // individuals of this lane
  float par[kDePerLane][3], sem[kDePerLane], stk[kDePerLane];

  // generation 0: the grid
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q) {
    const int i = lane + 32 * q;
#pragma unroll
    for (int d = 0; d < 3; ++d) par[q][d] = q < cnt ? R.grid[3 * i + d] : 0.f;
  }
  de_eval<W>(R, e0, e1, Tsec, par, cnt, sem, stk);
#pragma unroll
  for (int q = 0; q < kDePerLane; ++q) {
    if (q >= cnt) continue;
    const int i = lane + 32 * q;
    P[i][0] = par[q][0];
    P[i][1] = par[q][1];
    P[i][2] = par[q][2];
    P[i][3] = sem[q];
    P[i][4] = stk[q];
  }
  __syncwarp();

  for (int gen = 1; np >= 4 && gen <= R.ngen; ++gen) {
    // trials from the previous generation's population
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q) {
      if (q >= cnt) continue;
      const int i = lane + 32 * q;
      int r[3];
      de_pick3(cdp, t0, gen, i, np, r);
      const int jrand = (int)(de_key(cdp, t0, gen, i, 3) % 3u);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float u = __fmul_rn((float)(de_key(cdp, t0, gen, i, 4 + d) >> 40), 1.0f / 16777216.0f);
        float v = P[i][d];
        if (u < 0.9f || d == jrand) v = __fadd_rn(P[r[0]][d], __fmul_rn(0.5f, __fsub_rn(P[r[1]][d], P[r[2]][d])));
        v = v < R.lo[d] ? R.lo[d] : (v > R.hi[d] ? R.hi[d] : v);
        par[q][d] = v;
      }
    }
    de_eval<W>(R, e0, e1, Tsec, par, cnt, sem, stk);
    __syncwarp();   // every lane has read the population
#pragma unroll
    for (int q = 0; q < kDePerLane; ++q) {
      if (q >= cnt) continue;
      const int i = lane + 32 * q;
      if (sem[q] >= P[i][3]) {
        P[i][0] = par[q][0];
        P[i][1] = par[q][1];
        P[i][2] = par[q][2];
        P[i][3] = sem[q];
        P[i][4] = stk[q];
      }
    }
    __syncwarp();
  }

  // the best individual (largest semblance, lowest index on ties)
  float bs = 0.f;
  int bi = 0x7fffffff;
  for (int q = 0; q < cnt; ++q) {
    const int i = lane + 32 * q;
    if (P[i][3] > bs) {
      bs = P[i][3];
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float os = __shfl_xor_sync(0xffffffffu, bs, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (os > bs || (os == bs && oi < bi)) {
      bs = os;
      bi = oi;
    }
  }
  if (lane == 0) {
    const int64_t o = item;
    if (bi == 0x7fffffff || !(bs > 0.f)) {
      R.a[o] = R.grid[0];
      R.b[o] = R.grid[1];
      R.c[o] = (float)((double)R.grid[2] / 1e6);
      R.str[o] = 0.f;
      R.stk[o] = R.stt00[cdp];
    } else {
      R.a[o] = P[bi][0];
      R.b[o] = P[bi][1];
      R.c[o] = (float)((double)P[bi][2] / 1e6);
      R.str[o] = bs;
      R.stk[o] = P[bi][4];
    }
  }
}

}  // namespace

// P: stores, apertures, sampling and status as for the search kernels, pass_bounds the search
// box; its capacity is set here.
int launch_crs_de(int w, const DeParams& R, KParams P, cudaStream_t st) {
  if (R.np > kDeMaxPop) return fail(SEMB_E_ARG, "CRS-DE population %d above %d", R.np, kDeMaxPop);
  const void* fn = w == 1 ? (const void*)k_crs_de<1> : w == 3 ? (const void*)k_crs_de<3> : (const void*)k_crs_de<5>;
  if (w != 1 && w != 3 && w != 5) return fail(SEMB_E_WINDOW, "no CRS-DE kernel for w = %d", w);
  // buffers for two CTAs per SM; a buffer must hold a whole trace's window
  int cap = 8192;
  while (cap > 64 && de_layout(cap, R.np).total > 112 * 1024) cap -= 64;
  const int min_cap = (int)P.pitch + 16;
  if (cap < min_cap) cap = (min_cap + 63) & ~63;
  const size_t smem = de_layout(cap, R.np).total;
  void* args[] = {const_cast<DeParams*>(&R), &P};
  if (smem > kMaxDynamicSmem) {
    const void* lf = w == 1   ? (const void*)k_crs_de_long<1>
                     : w == 3 ? (const void*)k_crs_de_long<3>
                              : (const void*)k_crs_de_long<5>;
    const int grid = (int)(((int64_t)R.ncdps * R.ns + kDeLongWarps - 1) / kDeLongWarps);
    SEMB_CUDA(cudaLaunchKernel(lf, dim3(grid), dim3(kDeLongWarps * 32), args, 0, st));
    return SEMB_OK;
  }
  P.cap = cap;
  const int grid = (int)((int64_t)R.ncdps * ((R.ns + kDeWarps - 1) / kDeWarps));
  // the most any plan takes: plans of other sizes share the kernel
  SEMB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem));
  SEMB_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(kDeWarps * 32), args, smem, st));
  return SEMB_OK;
}

}  // namespace semb
