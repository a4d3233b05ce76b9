// CRS filter kernel: bounds on the semblance of every candidate, from the moments of
// whole B runs (sm_103a).
//
// A search spends its time evaluating candidates that are far from winning.  This kernel
// bounds every candidate's semblance at about a quarter of the direct kernels' cost and
// keeps, per (CDP, t0), the few whose upper bound reaches the best lower bounds (the
// best one in the plain form, the fourth best in the batched form, which keeps four).
// The refine kernels (refine_kernel.cuh) then evaluate those few with the direct
// kernels' own arithmetic, operation by operation, so the search's results are the
// direct kernels' unless a candidate's rounding lies outside its bounds (see below).
//
// The items of one warp and lane are consecutive B values of one (A, C) pair: one run,
// B_r = B_c + r dB about its centre slot.  On one trace their traveltimes differ by
//
//     t_r - t = dB dm^2 r / (2 t) - (dB dm^2 r)^2 / (8 t^3) + ... = k1 r + k2 r^2,
//
// t the centre's, usually a few hundredths of a sample over the whole run (dm is at most
// the midpoint aperture, and B's range is fixed by the curvatures a CRS search covers).
// As long as no item leaves the centre's sample interval, item r interpolates window
// sample j as v_j + d_j (k1 r + k2 r^2) with the centre's value v_j and slope d_j, so the
// numerators and the energy of *every* item of the run are polynomials in r whose
// coefficients are sums over traces:
//
//     num_j(r) = sum v_j + r sum d_j k1 + r^2 sum d_j k2
//     den(r)   = sum E + 2 r sum k1 G + r^2 sum (k1^2 H + 2 k2 G) + 2 r^3 sum k1 k2 H,
//                E = sum_j v_j^2, G = sum_j v_j d_j, H = sum_j d_j^2
//
// (the r^4 term, k2^2 H, is below 4e-7 of E at the widest run the planner admits).  One
// trace costs a lane about 40 instructions for the whole run, where the direct kernels
// spend about 20 on every item.
//
// Crossings.  Where some item of the run lies across a sample boundary from the centre,
// the piecewise linear interpolation gains, beyond that boundary, the slope change there
// times the distance: v_j += c_j z with c_j the second difference at the boundary
// sample and z >= 0 the item's distance beyond it.  The lane notes such a trace in a bit
// mask; at the end of the chunk every lane takes its next noted trace and adds the
// crossing terms of all items of the run (zero for those not beyond the boundary) into
// per-item sums.  At most half a sample lies between an item and the centre
// (moment_narrow, planned per trace), so at most one boundary is crossed.  Traces that
// are too wide for the expansion take a per-item path with range checks, into the same
// per-item sums, and so do those that may leave the record, on the lanes where the run
// straddles its end.  A pass on which two traces are
// out of the record for every item is left: no item of it is valid (err < 2).
//
// The bounds.  The direct kernels round the traveltime of every (trace, candidate) on
// its own, by about t 2^-24 samples, which moves numerator j by a random sum of rms
// s sqrt(sum d_j^2), s = t 2^-24; the filter's own rounding adds as much.  The bounds
// take `kappa` times that (8 in the batched form; 16 in the plain form, whose
// traveltimes are rounded more often), growing with sqrt(N) for what may not be random,
// and a relative 4e-6 and up for the order of the FP32 sums.  A trace's slopes are the
// steepest of its run: beyond a boundary that an item crosses, or may cross by its
// rounding (`edge`), and of every item of a trace that goes on its own.  Where an energy is
// all rounding, or not finite, or where rounding decides whether a trace is in the record,
// the item is kept.  The bounds are a multiple of an rms, not a worst case (which, some 8 s
// sum |d_j|, would keep ten times the candidates): what the filter leaves out has lost
// unless a rounding lies outside them.
//
// Windows are staged as plain FP32 samples (4 bytes each, a chunk holds up to 128
// traces): straight from the FP32 store by TMA, or, for a 16-bit store, converted once
// per chunk.  The pipeline otherwise follows semb_pipe_kernel: a rotating planner warp,
// mbarrier hand-offs, a work queue, the last warp of a task merging its lists.
//
// What bounds it: the latency of a warp's own chains, at 12 warps of 168 registers per SM.
// ncu on 16 CDPs of the 500 x 48 line: issue 59% of cycles, FMA pipe 34%, ALU 26%,
// shared-memory loads 22%; a warp waits 1.3 cycles per instruction on fixed latencies, 0.65 on
// instruction fetch, 0.6 on shared memory.  By section the main loop (about 40 instructions per
// trace and run) takes 30% of the time, the crossings (about 100 per noted trace of the
// busiest lane) 30%, the traces at the record's ends 10 to 15%, and the rest is the planner's
// and the copies' latency, hidden only in part.  Long runs pay: 21 B values as one run of 22
// slots at 384 threads took 29.5 ms where two runs of 12 slots at 512 threads took 36.2 (32
// CDPs of the line), 31 as one of 32 slots at 256 threads 130 against 147 as two of 16.  The
// second-order terms only where they count (moment_linear) gave 2%, the crossings above
// and below the centre apart (half the slots each) 7%; two noted traces at a time was 10%
// slower, and so was the main loop unrolled by four.  Counting the steepest slopes costs 2 to 3%.
// Measured on GB300, whole pass with the re-pick, with every candidate evaluated and now, in
// turn on the same surveys: 64 CDPs of the line (21 x 21 x 21, FP16) 172.3 -> 55.4 ms; 128 CDPs
// with apertures of 50 to 2000 traces 653 -> 206 ms; 48 such CDPs with 31 x 31 x 31 candidates
// (BF16) 539 -> 178 ms; plain form, 12 CDPs of the line 99.6 -> 9.8 ms.
#pragma once

#include <type_traits>

#include "pipe_kernel.cuh"

namespace semb {

constexpr int kFilterList = 6;     // runs kept per thread
constexpr int kFilterPool = 6;     // output pool: kept runs per (CDP, t0) on average

// rsqrt.approx (ftz), 1/t for the expansion's slopes
__device__ __forceinline__ float rsqrt_fast(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct FilterParams {
  KParams k;               // geometry, queue, candidate runs ([npass * warps][RC]), staging
  int2* head;              // [ncdps][ns]: (first entry, entries) in the pool; entries -1: the
                           // task goes to the direct kernel
  int2* pool;              // entries (run, slot mask)
  int pool_cap;
  unsigned long long* pool_count;
  int2* fb_tasks;          // tasks whose lists overflowed
  int* fb_count;
  unsigned long long* fb_total;   // counts them over all launches of a run
  float edge;              // within this of a sample boundary rounding may lie across it
  float kappa;             // multiple of the rms rounding effect (see above)
};

// Shared-memory layout (bytes), shared by host and device:
//   [0, 128)   mbarriers (full[3], q_full[3], q_empty[3], merge_done) and the merge counter
//   prod       producer state (its `drop` counts the pass's dropped traces)
//   meta[4]    chunk metadata, tag[4] chunk tags
//   src[4]     copy descriptors
//   list       per thread: upper bound, run, slot mask [3][kFilterList][NT]; the KT best
//              lower bounds [KT][NT]; the largest upper bound dropped from the list [NT]
//   plane[3]   staged windows, FP32, each followed by its zero block
//   raw[2]     16-bit windows (TMA destination; 16-bit stores only)
struct FilterLayout {
  size_t prod, meta, tag, src, list, plane, plane_stride, raw, raw_stride, total;
};

__host__ __device__ inline FilterLayout filter_layout(int cap, bool f32, int kt, int nt) {
  FilterLayout L;
  L.prod = 128;
  L.meta = L.prod + align128(sizeof(Producer));
  L.tag = L.meta + kMetaRing * kMetaBytes;
  L.src = L.tag + align128(kMetaRing * sizeof(ChunkTag));
  L.list = L.src + (size_t)kMetaRing * kMaxChunk * 16;
  L.plane = L.list + (size_t)(3 * kFilterList + kt + 1) * nt * 4;
  L.plane_stride = align128(((size_t)cap + kZeroSlots) * 4);
  L.raw = L.plane + kStages * L.plane_stride;
  L.raw_stride = f32 ? 0 : align128((size_t)cap * 2);
  L.total = L.raw + kRawBufs * L.raw_stride;
  return L;
}

// The run's sums over the in-range traces of a pass: window samples in the pairs
// (j, j+2) plus one single, and the energy coefficients.
template <int W>
struct MomentSums {
  static constexpr int NP = (W - 1) / 2;      // pairs: W = 3: (0,2); W = 5: (0,2), (1,3)
  static constexpr int NQ = NP > 0 ? NP : 1;
  static constexpr int JS = W == 3 ? 1 : W - 1;   // the single window sample
  float2 v[NQ], n1[NQ], n2[NQ];
  float vs, n1s, n2s;
  float2 e0;
  float e1, e2, e3, h;

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int i = 0; i < NQ; ++i) v[i] = n1[i] = n2[i] = make_float2(0.f, 0.f);
    vs = n1s = n2s = 0.f;
    e0 = make_float2(0.f, 0.f);
    e1 = e2 = e3 = h = 0.f;
  }
  // one trace: window samples at address a, weight x, expansion k1 and k2n = k1^2 / t
  // (k2 = -k2n / 2; the factor is applied at the end of the pass)
  // QUAD: with the terms of k2n (else they are below the rounding, moment_linear)
  template <bool QUAD>
  __device__ __forceinline__ void add(uint32_t a, float x, float k1, float k2n) {
    float s[W + 1];
#pragma unroll
    for (int j = 0; j <= W; ++j) s[j] = lds32(a + 4u * j);
    const float2 xx = make_float2(x, x), kk1 = make_float2(k1, k1), kk2 = make_float2(k2n, k2n);
    const float ds = s[JS + 1] - s[JS];
    const float ws = fmaf(ds, x, s[JS]);
    vs += ws;
    n1s = fmaf(ds, k1, n1s);
    if (QUAD) n2s = fmaf(ds, k2n, n2s);
    float G = ws * ds, H = ds * ds;
    e0.x = fmaf(ws, ws, e0.x);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const float2 lo = make_float2(s[i], s[i + 2]), up = make_float2(s[i + 1], s[i + 3]);
      const float2 d = __ffma2_rn(lo, make_float2(-1.f, -1.f), up);
      const float2 w = __ffma2_rn(d, xx, lo);
      v[i] = __fadd2_rn(v[i], w);
      n1[i] = __ffma2_rn(d, kk1, n1[i]);
      if (QUAD) n2[i] = __ffma2_rn(d, kk2, n2[i]);
      e0 = __ffma2_rn(w, w, e0);
      G = fmaf(w.x, d.x, fmaf(w.y, d.y, G));
      H = fmaf(d.x, d.x, fmaf(d.y, d.y, H));
    }
    e1 = fmaf(k1, G, e1);
    const float aH = k1 * H;
    e2 = fmaf(aH, k1, e2);
    if (QUAD) {
      e2 = fmaf(-k2n, G, e2);
      e3 = fmaf(k2n, aH, e3);
    }
    h += H;
  }
  // num_j at slot offsets rr
  __device__ __forceinline__ float2 num(int j, float2 rr) const {
    float a, b, c;
    if (j == JS) {
      a = vs;
      b = n1s;
      c = n2s;
    } else {
      const int i = W == 3 ? 0 : (j & 1);
      const bool hi = j >= 2;
      a = hi ? v[i].y : v[i].x;
      b = hi ? n1[i].y : n1[i].x;
      c = hi ? n2[i].y : n2[i].x;
    }
    c *= -0.5f;
    return __ffma2_rn(rr, __ffma2_rn(rr, make_float2(c, c), make_float2(b, b)), make_float2(a, a));
  }
};

// Start the copies of a chunk's windows: straight into the FP32 plane, or the 16-bit
// windows into the raw buffer (window lengths and offsets are multiples of 8 samples).
template <bool F32>
__device__ __forceinline__ void issue_windows(const KParams& P, const ChunkMeta* meta, const int4* src, void* dst,
                                              uint64_t* bar) {
  const int lane = threadIdx.x & 31;
  constexpr uint32_t unit = F32 ? 4u : 2u;
  const int n = meta->n;
  if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)(meta->bytes / 4) * unit);
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    const int4 si = src[entry_slot(meta, i)];
    if (si.z <= 0) continue;
    const int64_t at = (int64_t)si.x * P.pitch + si.y;
    const void* g = F32 ? (const void*)(P.samples + at) : (const void*)(P.samples16 + at);
    bulk_g2s(static_cast<unsigned char*>(dst) + (size_t)si.w * unit, g, (uint32_t)si.z * unit, bar);
  }
}

// 16-bit stores, all warps: the landed windows as FP32 samples.
__device__ __forceinline__ void convert_windows(const KParams& P, const ChunkMeta* meta, const int4* src,
                                                const unsigned char* raw, float* plane, int first_warp) {
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int warp = ((threadIdx.x >> 5) + nwarps - first_warp) % nwarps;
  const int n = meta->n;
  const bool f16 = P.storage == STORE_F16;
  for (int i = warp; i < n; i += nwarps) {
    const int e = entry_slot(meta, i);
    const int4 si = src[e];   // (trace, lo, len, off)
    const float sc = meta->scale[e];
    const uint32_t* r = reinterpret_cast<const uint32_t*>(raw) + si.w / 2;
    float2* d = reinterpret_cast<float2*>(plane + si.w);
    for (int k = lane; k < si.z / 2; k += 32) {
      const uint32_t b = r[k];
      const float v0 = f16 ? half_bits_to_float(b & 0xffffu) : __uint_as_float(b << 16);
      const float v1 = f16 ? half_bits_to_float(b >> 16) : __uint_as_float(b & 0xffff0000u);
      d[k] = make_float2(v0 * sc, v1 * sc);
    }
  }
}

// W: window.  F32: stage the FP32 store (plain form, FP32 batched store).  KT: how many
// best candidates the search keeps per (CDP, t0).  RC: slots per run (even).  NT: threads
// per CTA, one CTA per SM.
template <int W, bool F32, int KT, int RC, int NT>
__global__ void __launch_bounds__(NT, 1) semb_filter_kernel(FilterParams FP) {
  static_assert((W == 1 || W == 3 || W == 5) && RC % 2 == 0 && RC <= 32, "CRS windows; slot pairs and masks");
  constexpr int KL = kFilterList;
  constexpr int RP = RC / 2;
  constexpr int CS = (RC - 1) / 2;   // the centre slot
  const KParams& P = FP.k;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const FilterLayout L = filter_layout(P.cap, F32, KT, NT);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);   // copies landed: [kStages] (F32) or [kRawBufs]
  uint64_t* q_full = full + kStages;                         // [kStages] (16-bit: converted)
  uint64_t* q_empty = q_full + kStages;                      // [kStages]
  uint64_t* merge_done = q_empty + kStages;                  // [1]
  int* merge_cnt = reinterpret_cast<int*>(smem_raw + 96);
  Producer* prod = reinterpret_cast<Producer*>(smem_raw + L.prod);
  auto meta_at = [&](int c) {
    return reinterpret_cast<ChunkMeta*>(smem_raw + L.meta + (size_t)(c % kMetaRing) * kMetaBytes);
  };
  auto tag_at = [&](int c) { return reinterpret_cast<ChunkTag*>(smem_raw + L.tag) + (c % kMetaRing); };
  auto src_at = [&](int c) { return reinterpret_cast<int4*>(smem_raw + L.src) + (c % kMetaRing) * kMaxChunk; };
  auto plane_at = [&](int c) {
    return reinterpret_cast<float*>(smem_raw + L.plane + (size_t)(c % kStages) * L.plane_stride);
  };
  auto raw_at = [&](int c) { return smem_raw + L.raw + (size_t)(c % kRawBufs) * L.raw_stride; };
  auto full_at = [&](int c) { return F32 ? &full[c % kStages] : &full[c % kRawBufs]; };
  auto full_phase = [&](int c) { return (uint32_t)((F32 ? c / kStages : c / kRawBufs) & 1); };
  float* l_up = reinterpret_cast<float*>(smem_raw + L.list);   // [KL][NT]
  int* l_run = reinterpret_cast<int*>(l_up + KL * NT);
  int* l_msk = l_run + KL * NT;
  float* l_low = reinterpret_cast<float*>(l_msk + KL * NT);    // [KT][NT]
  float* l_ev = l_low + KT * NT;                               // [NT]

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;

  for (int s = 0; s < kStages; ++s)
    if (threadIdx.x < kZeroSlots) plane_at(s)[P.cap + threadIdx.x] = 0.f;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&q_full[s], nwarps);
      mbar_init(&q_empty[s], nwarps);
    }
    mbar_init(merge_done, 1);
    *merge_cnt = 0;
    prod->task = -1;
    prod->done = 0;
    prod->next = 0;
    fence_mbar_init();
  }
  __syncthreads();

  int seen = 0;   // chunks whose copies this thread has seen land
  // a bounded wait failed: report it and wait (bounded) for the copies in flight
  auto give_up = [&]() {
    if (lane == 0) atomicOr(P.status, ST_TIMEOUT);
    const int issued = min(prod->next, seen + (F32 ? kStages : kRawBufs));
    for (int c = seen; c < issued; ++c) wait_bar(full_at(c), full_phase(c));
  };

  // the planner warp: plan the next chunk of the stream and start its copies
  auto produce = [&]() -> bool {
    const int c = prod->next;
    // F32: the copies land in the plane the warps computed chunk c - kStages from
    if (F32 && c >= kStages && !wait_bar(&q_empty[c % kStages], (c / kStages - 1) & 1)) return false;
    ChunkMeta* m = meta_at(c);
    ChunkTag* tg = tag_at(c);
    int4* src = src_at(c);
    void* dst = F32 ? (void*)plane_at(c) : (void*)raw_at(c);
    if (prod->task < 0) {
      int t = 0;
      if (lane == 0) t = atomicAdd(P.counter, 1);
      t = __shfl_sync(0xffffffffu, t, 0);
      __syncwarp();
      if (t >= P.ntasks) {
        if (lane == 0) {
          m->n = m->n_in = m->consumed = m->bytes = 0;
          tg->flags = CH_END;
          prod->done = 1;
          prod->next = c + 1;
        }
        __syncwarp();
        issue_windows<F32>(P, m, src, dst, full_at(c));
        return true;
      }
      const int2 td = P.tasks[t];
      if (lane == 0) {
        prod->task = t;
        prod->cdp = td.x;
        prod->t0s = td.y;
        prod->begin = P.ap_off[td.x];
        prod->end = P.ap_off[td.x + 1];
        prod->pos = prod->begin;
        prod->pass = 0;
        prod->drop = 0;
        prod->T_lo = P.dt * (float)td.y;
        prod->T_hi = P.dt * (float)min(td.y + kTB - 1, P.ns - 1);
      }
      __syncwarp();
    }
    const int64_t pos = prod->pos, begin = prod->begin, end = prod->end;
    const int pass = prod->pass;
    plan_chunk<METHOD_CRS, FORM_FAST, true>(P, P.pass_bounds + pass * 8, pos, end, prod->T_lo, prod->T_hi, m, src);
    const int64_t npos = pos + m->consumed;
    const int drop = prod->drop + m->consumed - m->n;
    __syncwarp();
    if (lane == 0) {
      int flags = pos == begin ? CH_PASS_FIRST : 0;
      // two traces out of the record for every item: the pass has no valid item
      const bool dead = drop >= 2;
      if (dead) {
        m->n = m->n_in = m->bytes = 0;
        flags |= CH_DEAD;
      }
      if (npos >= end || dead) {
        flags |= CH_PASS_LAST;
        prod->pos = begin;
        prod->pass = pass + 1;
        prod->drop = 0;
        if (pass + 1 == P.npass) {
          flags |= CH_TASK_LAST;
          prod->task = -1;
        }
      } else {
        prod->pos = npos;
        prod->drop = drop;
      }
      tg->flags = flags;
      tg->cdp = prod->cdp;
      tg->t0s = prod->t0s;
      tg->pass = pass;
      tg->napert = (int)(end - begin);
      prod->next = c + 1;
    }
    __syncwarp();
    issue_windows<F32>(P, m, src, dst, full_at(c));
    return true;
  };

  // wait for chunk c's samples; 16-bit: convert this warp's share of it first
  auto convert_step = [&](int c) -> bool {
    if (!F32 && c >= kStages && !wait_bar(&q_empty[c % kStages], (c / kStages - 1) & 1)) return false;
    if (!wait_bar(full_at(c), full_phase(c))) return false;
    seen = c + 1;
    if constexpr (!F32) {
      convert_windows(P, meta_at(c), src_at(c), raw_at(c), plane_at(c), c % nwarps);
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[c % kStages]);
    }
    return true;
  };

  // chunks 0 and 1 (warp 0; the copies' barrier of chunk 0 orders them for the planner
  // of chunk 2)
  bool alive = true;
  if (warp == 0) {
    alive = produce();
    if (alive && !prod->done) alive = produce();
  }
  if (!alive || !convert_step(0)) {
    give_up();
    return;
  }

  const unsigned span = (unsigned)(P.ns - 2 * P.tau - 2);   // valid iff 0 <= it - tau <= span
  const float q_lo = (float)(P.tau * P.tau), q_hi = (float)(P.ns - P.tau - 1) * (float)(P.ns - P.tau - 1);
  const float hdB = 0.5f * P.dB;
  const float sig = (float)P.ns * 5.9604645e-8f;   // t 2^-24 at the record's end
  float T = 0.f;
  // the warp's run: A, C and the centre's B; the real slots and their widest offset
  float ca = 0.f, cb = 0.f, cc = 0.f, rmax = 0.f;
  unsigned valid = 0;
  MomentSums<W> ms;
  float2 inum[W][RP], iden[RP];   // per-item sums: the per-item path and the crossings
  int n_tot = 0;                  // staged traces of the pass
  uint32_t miss1 = 0, miss2 = 0;  // items out of range on one, on two or more of them
  uint32_t unsure = 0;            // items that may be in or out of range on some trace
  float low[KT];                  // the best lower bounds so far
  int ntask = 0;

  for (int c = 0;; ++c) {
    const ChunkTag tg = *tag_at(c);   // visible: this thread saw chunk c's copies land
    if (tg.flags & CH_END) break;
    // wait for (16-bit: convert) the next chunk; it exists: this one is not the end
    if (!F32 && !convert_step(c + 1)) {
      give_up();
      return;
    }
    if (!F32 && !wait_bar(&q_full[c % kStages], (c / kStages) & 1)) {
      give_up();
      return;
    }
    if (!F32 && warp == (c + 2) % nwarps && !prod->done && !produce()) {
      give_up();
      return;
    }

    const ChunkMeta* meta = meta_at(c);
    const float4* cand = P.cand + (size_t)(tg.pass * nwarps + warp) * RC;
    const int t0 = min(tg.t0s + lane, P.ns - 1);
    if (tg.flags & CH_PASS_FIRST) {
      T = (float)t0;
      const float4 cv = __ldg(cand + CS);
      ca = cv.x;
      cb = cv.y;
      cc = cv.z;
      valid = __ballot_sync(0xffffffffu, lane < RC && __float_as_int(__ldg(&cand[min(lane, RC - 1)].w)) >= 0);
      const int lo = valid ? __ffs(valid) - 1 : CS, hi = valid ? 31 - __clz(valid) : CS;
      // a little more than the widest offset: k2 r^2 is below 0.3% of k1 r
      rmax = 1.003f * (float)max(CS - lo, hi - CS);
      ms.reset();
#pragma unroll
      for (int p = 0; p < RP; ++p) {
#pragma unroll
        for (int j = 0; j < W; ++j) inum[j][p] = make_float2(0.f, 0.f);
        iden[p] = make_float2(0.f, 0.f);
      }
      n_tot = 0;
      miss1 = miss2 = unsure = 0;
    }

    // ---- compute chunk c ----
    const int n = meta->n, n_in = meta->n_in;
    const uint32_t plane = smem_u32(plane_at(c));
    const uint32_t top = plane + 4u * (uint32_t)P.cap;
    const uint32_t base0 = plane - 4u * (0x4B000000u + (uint32_t)P.tau);
    // traces whose run crosses the sample boundary above, below the centre
    uint32_t up_mask[kMaxChunk / 32], dn_mask[kMaxChunk / 32];
    auto front = [&](auto quad) {
      constexpr bool QUAD = decltype(quad)::value;
#pragma unroll
      for (int b = 0; b < kMaxChunk / 32; ++b) {
        uint32_t um = 0, dm = 0;
        const int e1 = min(n_in, 32 * b + 32);
#pragma unroll 2
        for (int e = 32 * b; e < e1; ++e) {
          const float4 g = meta->geo[e];
          const float u = fmaf(ca, g.x, T);
          const float q = fmaf(cb, g.y, fmaf(u, u, cc * g.z));
          const float t = sqrt_fast(q), ti = rsqrt_fast(q);
          const float y = __fadd_rz(t, 8388608.0f);
          const float x = t - (y - 8388608.0f);
          const float k1 = (hdB * g.y) * ti;
          const uint32_t a = min((__float_as_uint(y) + __float_as_uint(g.w)) * 4u + base0, top);
          if constexpr (SEMB_CHECKED) {
            report_window(P.status, __float_as_int(y) - 0x4B000000 - P.tau + __float_as_int(g.w), W, src_at(c)[e],
                          tg.cdp, t0);
          }
          ms.template add<QUAD>(a, x, k1, QUAD ? (k1 * k1) * ti : 0.f);
          const float h = fmaf(k1, rmax, FP.edge);
          if (x + h >= 1.0f) um |= 1u << (e - 32 * b);
          if (x < h) dm |= 1u << (e - 32 * b);
        }
        up_mask[b] = um;
        dn_mask[b] = dm;
      }
    };
    const bool quad = meta->quad != 0;
    if (quad) front(std::true_type{});
    else front(std::false_type{});
    // the other traces.  Wide ones in the record: every item on its own.  A narrow one whose
    // run is well inside the record on this lane joins the moments (and the crossings); one
    // whose run is well outside is a miss for every item; where the run straddles an end,
    // and for the other wide traces, each item goes on its own with range checks: an
    // out-of-range item reads the zero block with weight 0 and does not count
    for (int e = kMaxChunk - (n - n_in); e < kMaxChunk; ++e) {
      const float4 g = meta->geo[e];
      const int soff = __float_as_int(g.w);
      float hm = 0.f;   // the most of its items' sums of squared slopes (padding: no less)
      const float u = fmaf(ca, g.x, T);
      const float q0 = fmaf(u, u, cc * g.z);
      const int kind = meta->raw[e];
      if (kind == 2) {
        // wide, every item in range: items two at a time, no range checks
        const float qc = fmaf(cb, g.y, q0), qs = P.dB * g.y;
        const uint32_t base = base0 + 4u * (uint32_t)soff;
#pragma unroll
        for (int pr = 0; pr < RP; ++pr) {
          const float2 rr = make_float2((float)(2 * pr - CS), (float)(2 * pr + 1 - CS));
          const float2 q = __ffma2_rn(rr, make_float2(qs, qs), make_float2(qc, qc));
          const float2 t = make_float2(sqrt_fast(q.x), sqrt_fast(q.y));
          const float2 y = __fadd2_rz(t, make_float2(8388608.0f, 8388608.0f));
          const float2 x = __ffma2_rn(__fadd2_rn(y, make_float2(-8388608.0f, -8388608.0f)), make_float2(-1.f, -1.f), t);
          // a padding slot's window may not be staged: the address stays in the plane
          const uint32_t ax = max(min(__float_as_uint(y.x) * 4u + base, top), plane);
          const uint32_t ay = max(min(__float_as_uint(y.y) * 4u + base, top), plane);
          if constexpr (SEMB_CHECKED) {
            const int i0 = soff - P.tau - 0x4B000000;
            if ((valid >> (2 * pr)) & 1) report_window(P.status, __float_as_int(y.x) + i0, W, src_at(c)[e], tg.cdp, t0);
            if ((valid >> (2 * pr + 1)) & 1)
              report_window(P.status, __float_as_int(y.y) + i0, W, src_at(c)[e], tg.cdp, t0);
          }
          float2 s0 = make_float2(lds32(ax), lds32(ay)), hs = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const float2 s1 = make_float2(lds32(ax + 4u * (j + 1)), lds32(ay + 4u * (j + 1)));
            const float2 d = __ffma2_rn(s0, make_float2(-1.f, -1.f), s1);
            const float2 v = __ffma2_rn(d, x, s0);
            inum[j][pr] = __fadd2_rn(inum[j][pr], v);
            iden[pr] = __ffma2_rn(v, v, iden[pr]);
            hs = __ffma2_rn(d, d, hs);
            s0 = s1;
          }
          hm = fmaxf(hm, fmaxf(hs.x, hs.y));
        }
        ms.h += hm;
        continue;
      }
      bool single = true;
      if (kind == 1) {   // narrow
        const float q = fmaf(cb, g.y, q0);
        const float t = sqrt_fast(q), ti = rsqrt_fast(q);   // NaN, or infinite: neither in nor out
        const float y = __fadd_rz(t, 8388608.0f);
        const float x = t - (y - 8388608.0f);
        const float k1 = (hdB * g.y) * ti;
        // the run stays within h samples of t, rounding included
        const float h = fmaf(k1, rmax, fmaf(4e-6f, (float)P.ns, 0.01f));
        const bool in = t - h >= (float)P.tau && t + h < (float)(P.ns - P.tau - 1) && h < 0.5f;
        const bool out = t + h < (float)P.tau || t - h >= (float)(P.ns - P.tau - 1);
        single = !in && !out;
        if (__any_sync(0xffffffffu, in)) {
          const uint32_t a = in ? min((__float_as_uint(y) + __float_as_uint(g.w)) * 4u + base0, top) : top;
          ms.template add<true>(a, in ? x : 0.f, in ? k1 : 0.f, in ? (k1 * k1) * ti : 0.f);
        }
        if (in) {
          const float hc = fmaf(k1, rmax, FP.edge);
          const uint32_t up = x + hc >= 1.0f ? 1u << (e & 31) : 0u, dn = x < hc ? 1u << (e & 31) : 0u;
#pragma unroll
          for (int b = 0; b < kMaxChunk / 32; ++b)
            if (e >> 5 == b) {
              up_mask[b] |= up;
              dn_mask[b] |= dn;
            }
        }
        if (out) {
          miss2 |= miss1;
          miss1 = ~0u;
        }
      }
      if (__any_sync(0xffffffffu, single)) {
        // t^2 within dq of the record's ends may be in range or not in the direct
        // kernels' rounding: such an item is kept whatever its sums
        const float dq = 9.5e-7f * fmaf(u, u, fmaf(P.bmax, g.y, fabsf(cc) * g.z));
        const float qc = fmaf(cb, g.y, q0), qs = P.dB * g.y;
        uint32_t off_now = 0, near_end = 0;   // items out of range, items within dq of an end
#pragma unroll
        for (int pr = 0; pr < RP; ++pr) {
          const float2 rr = make_float2((float)(2 * pr - CS), (float)(2 * pr + 1 - CS));
          const float2 q = __ffma2_rn(rr, make_float2(qs, qs), make_float2(qc, qc));
          const float2 t = make_float2(sqrt_fast(q.x), sqrt_fast(q.y));   // NaN below 0: out of range
          const float2 y = __fadd2_rz(t, make_float2(8388608.0f, 8388608.0f));
          float2 x = __ffma2_rn(__fadd2_rn(y, make_float2(-8388608.0f, -8388608.0f)), make_float2(-1.f, -1.f), t);
          const int relx = __float_as_int(y.x) - (0x4B000000 + P.tau);   // it - tau
          const int rely = __float_as_int(y.y) - (0x4B000000 + P.tau);
          const bool okx = single && ((valid >> (2 * pr)) & 1) && (unsigned)relx <= span;
          const bool oky = single && ((valid >> (2 * pr + 1)) & 1) && (unsigned)rely <= span;
          if (!okx) {
            x.x = 0.f;
            off_now |= 1u << (2 * pr);
          }
          if (!oky) {
            x.y = 0.f;
            off_now |= 1u << (2 * pr + 1);
          }
          if (fabsf(q.x - q_lo) <= dq || fabsf(q.x - q_hi) <= dq) near_end |= 1u << (2 * pr);
          if (fabsf(q.y - q_lo) <= dq || fabsf(q.y - q_hi) <= dq) near_end |= 1u << (2 * pr + 1);
          if constexpr (SEMB_CHECKED) {
            if (okx) report_window(P.status, soff + relx, W, src_at(c)[e], tg.cdp, t0);
            if (oky) report_window(P.status, soff + rely, W, src_at(c)[e], tg.cdp, t0);
          }
          const uint32_t ax = okx ? min(plane + 4u * (uint32_t)(soff + relx), top) : top;
          const uint32_t ay = oky ? min(plane + 4u * (uint32_t)(soff + rely), top) : top;
          float2 s0 = make_float2(lds32(ax), lds32(ay)), hs = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const float2 s1 = make_float2(lds32(ax + 4u * (j + 1)), lds32(ay + 4u * (j + 1)));
            const float2 d = __ffma2_rn(s0, make_float2(-1.f, -1.f), s1);
            const float2 v = __ffma2_rn(d, x, s0);
            inum[j][pr] = __fadd2_rn(inum[j][pr], v);
            iden[pr] = __ffma2_rn(v, v, iden[pr]);
            hs = __ffma2_rn(d, d, hs);
            s0 = s1;
          }
          hm = fmaxf(hm, fmaxf(hs.x, hs.y));
        }
        ms.h += hm;
        if (single) {
          unsure |= near_end;
          miss2 |= miss1 & off_now & ~near_end;
          miss1 |= off_now & ~near_end;
        }
      }
    }
    // crossings: each lane takes its next noted trace until none has one, first those above
    // the centre (dB >= 0: items of the higher slots), then those below
    auto crossings = [&](auto quad_c, auto up_c, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
      constexpr bool QUAD = decltype(quad_c)::value, UP = decltype(up_c)::value;
      while (__any_sync(0xffffffffu, (m0 | m1 | m2 | m3) != 0)) {
        const bool have = (m0 | m1 | m2 | m3) != 0;
        int e = 0;
        if (m0) {
          e = __ffs(m0) - 1;
          m0 &= m0 - 1;
        } else if (m1) {
          e = 31 + __ffs(m1);
          m1 &= m1 - 1;
        } else if (m2) {
          e = 63 + __ffs(m2);
          m2 &= m2 - 1;
        } else if (m3) {
          e = 95 + __ffs(m3);
          m3 &= m3 - 1;
        }
        const float4 g = meta->geo[e];
        const float u = fmaf(ca, g.x, T);
        const float q = fmaf(cb, g.y, fmaf(u, u, cc * g.z));
        const float t = sqrt_fast(q), ti = rsqrt_fast(q);
        const float y = __fadd_rz(t, 8388608.0f);
        const float x = t - (y - 8388608.0f);
        const float k1 = (hdB * g.y) * ti;
        // the boundary samples p_1 .. p_W with their neighbours p_0, p_W+1: the window
        // itself for a crossing upwards, one sample earlier for one downwards; without a
        // trace the zero block
        const uint32_t a =
            have ? min((__float_as_uint(y) + __float_as_uint(g.w)) * 4u + base0, top) - (UP ? 0u : 4u) : top;
        if constexpr (SEMB_CHECKED) {
          if (have)
            report_window(P.status, __float_as_int(y) - 0x4B000000 - P.tau + __float_as_int(g.w) - (UP ? 0 : 1), W + 1,
                          src_at(c)[e], tg.cdp, t0);
        }
        float p[W + 2];
#pragma unroll
        for (int j = 0; j < W + 2; ++j) p[j] = lds32(a + 4u * j);
        // distance beyond the boundary z_r = z0 + a1 r + a2 r^2; beyond it sample j is
        // p_j+1 + e_j z + c_j z with e_j the centre interval's slope along z
        const float z0 = have ? (UP ? x - 1.0f : -x) : 0.f;
        const float a1 = have ? (UP ? k1 : -k1) : 0.f;
        const float a2 = QUAD && have ? (UP ? -0.5f : 0.5f) * ((k1 * k1) * ti) : 0.f;
        float cj[W], q1 = 0.f, q2 = 0.f;
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const float dm = p[j + 1] - p[j], dp = p[j + 2] - p[j + 1];
          cj[j] = dp - dm;
          q1 = fmaf(cj[j], p[j + 1], q1);
          q2 = fmaf(cj[j], fmaf(2.f, UP ? dm : -dp, cj[j]), q2);
        }
        // the slopes beyond the boundary, where they are the larger ones: q2 is the difference
        // of the two intervals' sums of squared slopes
        ms.h += fmaxf(q2, 0.f);
        const float2 z02 = make_float2(z0, z0), a12 = make_float2(a1, a1), a22 = make_float2(a2, a2);
        const float2 q12 = make_float2(2.f * q1, 2.f * q1), q22 = make_float2(q2, q2);
        // only the slots on that side of the centre
#pragma unroll
        for (int pr = UP ? (CS + 1) / 2 : 0; pr < (UP ? RP : (CS + 1) / 2); ++pr) {
          const float2 rr = make_float2((float)(2 * pr - CS), (float)(2 * pr + 1 - CS));
          float2 z = __ffma2_rn(rr, QUAD ? __ffma2_rn(rr, a22, a12) : a12, z02);
          z = make_float2(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f));
#pragma unroll
          for (int j = 0; j < W; ++j) inum[j][pr] = __ffma2_rn(make_float2(cj[j], cj[j]), z, inum[j][pr]);
          iden[pr] = __ffma2_rn(z, __ffma2_rn(z, q22, q12), iden[pr]);
        }
      }
    };
    if (quad) {
      crossings(std::true_type{}, std::true_type{}, up_mask[0], up_mask[1], up_mask[2], up_mask[3]);
      crossings(std::true_type{}, std::false_type{}, dn_mask[0], dn_mask[1], dn_mask[2], dn_mask[3]);
    } else {
      crossings(std::false_type{}, std::true_type{}, up_mask[0], up_mask[1], up_mask[2], up_mask[3]);
      crossings(std::false_type{}, std::false_type{}, dn_mask[0], dn_mask[1], dn_mask[2], dn_mask[3]);
    }
    n_tot += n;
    // the plane and metadata of chunk c are no longer read by this warp
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_empty[c % kStages]);

    if (tg.flags & CH_PASS_LAST) {
      if (tg.pass == 0) {
        // the first pass of a task: the previous task's merge must have read the lists
        if (ntask > 0 && !wait_bar(merge_done, (ntask - 1) & 1)) {
          give_up();
          return;
        }
#pragma unroll
        for (int q = 0; q < KL; ++q) l_up[q * NT + threadIdx.x] = 0.f;
        l_ev[threadIdx.x] = 0.f;
#pragma unroll
        for (int q = 0; q < KT; ++q) low[q] = 0.f;
      }
      // ---- bounds of the pass's items ----
      if (!(tg.flags & CH_DEAD) && valid) {
        const float E0 = ms.e0.x + ms.e0.y, E1 = 2.f * ms.e1, E2 = ms.e2, E3 = -ms.e3;   // 2 k2 = -k2n
        const float nap = (float)tg.napert;
        const float sh = sig * sqrtf(ms.h);
        const float dn = (FP.kappa + 0.25f * sqrtf(nap)) * sh;
        const float de = 2.f * sh;                      // den: times sqrt(E0 + den)
        const float eta = 4e-6f + 1e-8f * nap;
        float up[RC];   // upper bounds; 0: not a valid item
#pragma unroll
        for (int p = 0; p < RP; ++p) {
          const float2 rr = make_float2((float)(2 * p - CS), (float)(2 * p + 1 - CS));
          float2 ac = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const float2 nj = __fadd2_rn(ms.num(j, rr), inum[j][p]);
            ac = __ffma2_rn(nj, nj, ac);
          }
          float2 dd = __ffma2_rn(rr, make_float2(E3, E3), make_float2(E2, E2));
          dd = __ffma2_rn(rr, dd, make_float2(E1, E1));
          dd = __fadd2_rn(__ffma2_rn(rr, dd, make_float2(E0, E0)), iden[p]);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const int r = 2 * p + hf;
            const float acsq = hf ? ac.y : ac.x, den = hf ? dd.y : dd.x;
            const int M = n_tot - ((miss1 >> r) & 1);   // with a second miss the item is invalid anyway
            const float es = E0 + fabsf(den);
            const float ed = fmaf(eta, es, de * sqrt_fast(es));
            // (a NaN, or sums near overflow, bound nothing either: es is not below 1e28)
            const bool sure = !((unsure >> r) & 1);
            const bool ok = ((valid & ~miss2) >> r & 1) && M > 0 && tg.napert - M < 2 &&
                            (!sure || !(den + ed <= kEpsilonF));
            const bool sane = sure && es < 1e28f;
            const float rm = __fdividef(1.0f, (float)M);
            const float am = sqrt_fast(acsq);
            // the bounds; an energy that is all rounding bounds nothing
            const float dlo = den - ed;
            const float u = sane && dlo > 0.f ? __fdividef(fmaf(dn, 2.f * am + dn, acsq) * rm, dlo) : 4.f;
            const float al = fmaxf(am - dn, 0.f);
            const float lw = sane && dlo > 2.f * kEpsilonF ? __fdividef(al * al * rm, den + ed) : 0.f;
            up[r] = ok ? u : 0.f;
            if (ok && lw > low[KT - 1]) {   // the KT best lower bounds
              float x = lw;
#pragma unroll
              for (int q = 0; q < KT; ++q) {
                const float b = low[q];
                low[q] = fmaxf(b, x);
                x = fminf(b, x);
              }
            }
          }
        }
        float umax = 0.f;
        uint32_t msk = 0;
#pragma unroll
        for (int r = 0; r < RC; ++r) {
          umax = fmaxf(umax, up[r]);
          if (up[r] > 0.f && up[r] >= low[KT - 1]) msk |= 1u << r;
        }
        if (msk) {
          // sorted insert (descending upper bound); what falls off the end is remembered
          float cu = umax;
          int cr = tg.pass * nwarps + warp, cm = (int)msk;
#pragma unroll
          for (int q = 0; q < KL; ++q) {
            const int o = q * NT + threadIdx.x;
            const float bu = l_up[o];
            if (cu > bu) {
              const int br = l_run[o], bm = l_msk[o];
              l_up[o] = cu;
              l_run[o] = cr;
              l_msk[o] = cm;
              cu = bu;
              cr = br;
              cm = bm;
            }
          }
          l_ev[threadIdx.x] = fmaxf(l_ev[threadIdx.x], cu);
        }
      }
      if (tg.flags & CH_TASK_LAST) {
        // ---- task done for this warp; the last warp to get here merges ----
#pragma unroll
        for (int q = 0; q < KT; ++q) l_low[q * NT + threadIdx.x] = low[q];
        __threadfence_block();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(merge_cnt, 1) == nwarps - 1;
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) {
          __threadfence_block();
          float best[KT], ev = 0.f;
#pragma unroll
          for (int q = 0; q < KT; ++q) best[q] = 0.f;
          for (int w2 = 0; w2 < nwarps; ++w2) {
            ev = fmaxf(ev, l_ev[w2 * 32 + lane]);
            for (int q2 = 0; q2 < KT; ++q2) {
              float x = l_low[q2 * NT + w2 * 32 + lane];
#pragma unroll
              for (int q = 0; q < KT; ++q) {
                const float b = best[q];
                best[q] = fmaxf(b, x);
                x = fminf(b, x);
              }
            }
          }
          const float thr = best[KT - 1];
          const int tt = tg.t0s + lane;
          const bool in = tt < P.ns;
          int cnt = 0;
          for (int w2 = 0; w2 < nwarps; ++w2)
            for (int q2 = 0; q2 < KL; ++q2) {
              const float up = l_up[q2 * NT + w2 * 32 + lane];
              if (in && up > 0.f && up >= thr) ++cnt;
            }
          // the lanes' entries, one after the other in the pool
          int incl = cnt;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
          }
          const int total = __shfl_sync(0xffffffffu, incl, 31);
          int base = 0;
          if (lane == 0) base = (int)min(atomicAdd(FP.pool_count, (unsigned long long)total), 0x7fffffffull);
          base = __shfl_sync(0xffffffffu, base, 0);
          // an overflowing thread list (or pool) sends the task to the direct kernel
          const bool over = (in && ev > 0.f && ev >= thr) || base > FP.pool_cap - total;
          const bool fb = __any_sync(0xffffffffu, over);
          if (in) FP.head[(int64_t)tg.cdp * P.ns + tt] = make_int2(base + incl - cnt, fb ? -1 : cnt);
          if (fb) {
            if (lane == 0) {
              FP.fb_tasks[atomicAdd(FP.fb_count, 1)] = make_int2(tg.cdp, tg.t0s);
              atomicAdd(FP.fb_total, 1ull);
            }
          } else if (cnt > 0) {
            int2* out = FP.pool + base + incl - cnt;
            for (int w2 = 0; w2 < nwarps; ++w2)
              for (int q2 = 0; q2 < KL; ++q2) {
                const int o = q2 * NT + w2 * 32 + lane;
                const float up = l_up[o];
                if (up > 0.f && up >= thr) *out++ = make_int2(l_run[o], l_msk[o]);
              }
          }
          __syncwarp();
          if (lane == 0) {
            *merge_cnt = 0;
            mbar_arrive(merge_done);   // the lists may be reused
          }
        }
        ++ntask;
      }
    }
    if (F32) {
      // the next chunk's copies: its tag is read next, and its planner is done
      if (!convert_step(c + 1)) {
        give_up();
        return;
      }
      if (warp == (c + 2) % nwarps && !prod->done && !produce()) {
        give_up();
        return;
      }
    }
  }
}

}  // namespace semb
