// Plain search kernel with a decoupled staging ring (sm_103a): the plain form of
// semb_search_kernel, its arithmetic bit for bit (the reference's FP32 operations in
// aperture order), for windows up to 5.
//
// What bounds the plain form is FP32 issue: every multiply and add is rounded on its own,
// so a (trace, candidate) takes 29 (CMP) or 34 (CRS) FP32 operations besides its square
// root.  Three things cut the instructions around them:
//
//   * Items two at a time.  A thread's candidates are pairs, and every operation of a pair
//     is one FP32x2 instruction (mul, add and FMA round each half as the scalar
//     instruction does).  Window samples come as scalar loads straight into the halves.
//   * The square root.  Two correctly rounded roots at a time, by Markstein's method, for
//     the range that squared traveltimes have (sqrt2_rn).
//   * No range checks where the planner has shown that every item is in range (nearly all
//     traces); the others take the checked path, in aperture order with them.
//
// and the CTA barriers go: windows land by TMA straight in one of three planes while the
// warps work (the ring of semb_filter_kernel's FP32 form: rotating planner warp, bounded
// mbarrier waits, a work queue, the last warp of a task merging its picks).
//
// What bounds it: the FP32 pipe.  160 CMPs of the uneven-fold line (256 velocities, w = 5)
// take 8.7 ms, 77% of the pipe's rate by operation count, against 11.4 in the two-barrier
// kernel; the 200 x 60 line (101 velocities, w = 3) 1.74 against 2.37, with a seventh of its
// lanes idle (104 slots in 28 warps' time) and 60 traces per pass.  Halving 1/sqrt by an
// integer subtraction instead of a multiply: 1% slower.
#pragma once

#include "filter_kernel.cuh"

namespace semb {

// FP32x2 product rounded on its own.  ptxas contracts a packed product and a following
// packed sum into one FMA (also where both name their rounding, and with -fmad=false),
// and the reference's arithmetic rounds both; as an FMA with a -0 that the compiler cannot
// see through (`nz`, from the launch's parameters) the product stays apart.
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float nz) {
  return __ffma2_rn(a, b, make_float2(nz, nz));
}

// The correctly rounded square roots of two floats in [2^-45, 2^30], after P. Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res.
// Dev. 34 (1990): from y near 1 / sqrt(x), g = x y and h = y / 2 approximate sqrt(x) and
// 1 / (2 sqrt(x)); the FMA gives the residual x - g^2 without error, and g + h (x - g^2) is
// so close to sqrt(x) that its one rounding is the root's.  semb_selftest_sqrt compares it
// with __fsqrt_rn on every float of that range.
__device__ __forceinline__ float2 sqrt2_rn(float2 x, float nz) {
  const float2 y = make_float2(rsqrt_fast(x.x), rsqrt_fast(x.y));
  const float2 g = mul2(x, y, nz);
  const float2 h = __fmul2_rn(y, make_float2(0.5f, 0.5f));
  const float2 r = __ffma2_rn(make_float2(-g.x, -g.y), g, x);
  return __ffma2_rn(r, h, g);
}

// Shared-memory layout (bytes), shared by host and device:
//   [0, 128)   mbarriers (full[3], q_empty[3], merge_done) and the merge counter
//   prod       producer state
//   meta[4]    chunk metadata, tag[4] chunk tags
//   src[4]     copy descriptors
//   pick       per thread: semblance, grid index, stack [3][NT]
//   plane[3]   staged windows, FP32, each followed by its zero block
struct PlainLayout {
  size_t prod, meta, tag, src, pick, plane, plane_stride, total;
};

__host__ __device__ inline PlainLayout plain_layout(int cap, int nt) {
  PlainLayout L;
  L.prod = 128;
  L.meta = L.prod + align128(sizeof(Producer));
  L.tag = L.meta + kMetaRing * kMetaBytes;
  L.src = L.tag + align128(kMetaRing * sizeof(ChunkTag));
  L.pick = L.src + (size_t)kMetaRing * kMaxChunk * 16;
  L.plane = L.pick + align128(3 * (size_t)nt * 4);
  L.plane_stride = align128(((size_t)cap + kZeroSlots) * 4);
  L.total = L.plane + kStages * L.plane_stride;
  return L;
}

// W: window.  RC: candidates per thread (even).  NT: threads per CTA, one CTA per SM.
template <int METHOD, int W, int RC, int NT>
__global__ void __launch_bounds__(NT, 1) semb_plain_kernel(KParams P) {
  static_assert(RC % 2 == 0, "item pairs");
  constexpr int RP = RC / 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const PlainLayout L = plain_layout(P.cap, NT);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);   // [kStages]
  uint64_t* q_empty = full + kStages;                        // [kStages]
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
  float* p_sem = reinterpret_cast<float*>(smem_raw + L.pick);   // [NT]
  int* p_idx = reinterpret_cast<int*>(p_sem + NT);
  float* p_stk = p_sem + 2 * NT;

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;

  for (int s = 0; s < kStages; ++s)
    if (threadIdx.x < kZeroSlots) plane_at(s)[P.cap + threadIdx.x] = 0.f;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
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
    const int issued = min(prod->next, seen + kStages);
    for (int c = seen; c < issued; ++c) wait_bar(&full[c % kStages], (c / kStages) & 1);
  };
  // the planner warp: plan the next chunk of the stream and start its copies
  auto produce = [&]() -> bool {
    const int c = prod->next;
    // the copies land in the plane the warps computed chunk c - kStages from
    if (c >= kStages && !wait_bar(&q_empty[c % kStages], (c / kStages - 1) & 1)) return false;
    ChunkMeta* m = meta_at(c);
    ChunkTag* tg = tag_at(c);
    int4* src = src_at(c);
    if (prod->task < 0) {
      int t = 0;
      if (lane == 0) t = atomicAdd(P.counter, 1);
      t = __shfl_sync(0xffffffffu, t, 0);
      __syncwarp();
      if (t >= (P.ntasks_dev ? *P.ntasks_dev : P.ntasks)) {
        if (lane == 0) {
          m->n = m->n_in = m->consumed = m->bytes = 0;
          tg->flags = CH_END;
          prod->done = 1;
          prod->next = c + 1;
        }
        __syncwarp();
        issue_chunk_copies(P, m, src, plane_at(c), &full[c % kStages]);
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
    plan_chunk<METHOD, FORM_PLAIN>(P, P.pass_bounds + pass * 8, pos, end, prod->T_lo, prod->T_hi, m, src);
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
    issue_chunk_copies(P, m, src, plane_at(c), &full[c % kStages]);
    return true;
  };

  bool alive = true;
  if (warp == 0) {
    alive = produce();
    if (alive && !prod->done) alive = produce();
  }
  if (!alive || !wait_bar(&full[0], 0)) {
    give_up();
    return;
  }
  seen = 1;

  const float2 k23 = make_float2(8388608.0f, 8388608.0f), km23 = make_float2(-8388608.0f, -8388608.0f);
  const float2 kNeg = make_float2(-1.0f, -1.0f), idt2 = make_float2(P.idt, P.idt);
  const float nz = P.ns < 0 ? 0.0f : -0.0f;   // -0: see mul2
  const float tau_lo = (float)P.tau, tau_hi = (float)(P.ns - P.tau - 1);
  constexpr float kSent = (METHOD == METHOD_CMP) ? -1.0f : 0.0f;
  float Tsec = 0.f;
  float2 ca[RP], cb[RP], cc[RP];
  float2 num[RP][W], den[RP], lin[RP];
  int n_tot = 0;                   // staged traces of the pass
  uint32_t miss1 = 0, miss2 = 0;   // items out of range on one, on two or more of them
  float best_s = 0.f, best_k = 0.f;
  int best_i = 0x7fffffff;
  int ntask = 0;

  for (int c = 0;; ++c) {
    const ChunkTag tg = *tag_at(c);   // visible: this thread saw chunk c's copies land
    if (tg.flags & CH_END) break;
    const ChunkMeta* meta = meta_at(c);
    const float4* cand = P.cand + tg.pass * P.cpp + warp * RC;
    const int t0 = min(tg.t0s + lane, P.ns - 1);
    if (tg.flags & CH_PASS_FIRST) {
      Tsec = __fmul_rn(P.dt, (float)t0);
      if (METHOD == METHOD_CMP) Tsec = __fmul_rn(Tsec, Tsec);   // t0^2
#pragma unroll
      for (int p = 0; p < RP; ++p) {
        const float4 c0 = __ldg(cand + 2 * p), c1 = __ldg(cand + 2 * p + 1);
        ca[p] = make_float2(c0.x, c1.x);
        cb[p] = make_float2(c0.y, c1.y);
        cc[p] = make_float2(c0.z, c1.z);
#pragma unroll
        for (int j = 0; j < W; ++j) num[p][j] = make_float2(0.f, 0.f);
        den[p] = lin[p] = make_float2(0.f, 0.f);
      }
      n_tot = 0;
      miss1 = miss2 = 0;
    }

    // ---- compute chunk c, in aperture order ----
    const int n = meta->n;
    const uint32_t plane = smem_u32(plane_at(c));
    const uint32_t top = plane + 4u * (uint32_t)P.cap;
    const float2 T2 = make_float2(Tsec, Tsec);
#pragma unroll 2
    for (int e = 0; e < n; ++e) {
      const float4 g = meta->geo[e];
      const float2 gx = make_float2(g.x, g.x), gy = make_float2(g.y, g.y), gz = make_float2(g.z, g.z);
      const uint32_t base = plane + 4u * (uint32_t)(__float_as_int(g.w) - P.tau) - 4u * 0x4B000000u;
      const bool inr = meta->raw[e] != 0;   // every item in range
#pragma unroll
      for (int p = 0; p < RP; ++p) {
        float2 q;
        if (METHOD == METHOD_CMP) {
          q = __fadd2_rn(T2, mul2(cc[p], gz, nz));
        } else {
          const float2 u = __fadd2_rn(T2, mul2(ca[p], gx, nz));
          q = __fadd2_rn(__fadd2_rn(mul2(u, u, nz), mul2(cb[p], gy, nz)), mul2(cc[p], gz, nz));
        }
        float2 x;
        uint32_t ax, ay;
        if (inr) {
          const float2 t = mul2(sqrt2_rn(q, nz), idt2, nz);
          const float2 y = __fadd2_rz(t, k23);
          x = __ffma2_rn(__fadd2_rn(y, km23), kNeg, t);   // t - floor(t), exact
          ax = min(__float_as_uint(y.x) * 4u + base, top);
          ay = min(__float_as_uint(y.y) * 4u + base, top);
          if constexpr (SEMB_CHECKED) {
            const int i0 = __float_as_int(g.w) - P.tau - 0x4B000000;
            report_window(P.status, __float_as_int(y.x) + i0, W, src_at(c)[e], tg.cdp, t0);
            report_window(P.status, __float_as_int(y.y) + i0, W, src_at(c)[e], tg.cdp, t0);
          }
        } else {
          // each item with its range check; an out-of-range item reads the zero block
          // with weight 0, adds +0 and does not count
          const float rx = q.x < 0.0f ? -1.0f : __fsqrt_rn(q.x), ry = q.y < 0.0f ? -1.0f : __fsqrt_rn(q.y);
          const float2 t = make_float2(__fmul_rn(rx, P.idt), __fmul_rn(ry, P.idt));
          const bool okx = t.x >= tau_lo && t.x < tau_hi, oky = t.y >= tau_lo && t.y < tau_hi;
          const float2 y = __fadd2_rz(t, k23);
          x.x = okx ? __fsub_rn(t.x, __fsub_rn(y.x, 8388608.0f)) : 0.0f;
          x.y = oky ? __fsub_rn(t.y, __fsub_rn(y.y, 8388608.0f)) : 0.0f;
          ax = okx ? min(__float_as_uint(y.x) * 4u + base, top) : top;
          ay = oky ? min(__float_as_uint(y.y) * 4u + base, top) : top;
          if constexpr (SEMB_CHECKED) {
            const int i0 = __float_as_int(g.w) - P.tau - 0x4B000000;
            if (okx) report_window(P.status, __float_as_int(y.x) + i0, W, src_at(c)[e], tg.cdp, t0);
            if (oky) report_window(P.status, __float_as_int(y.y) + i0, W, src_at(c)[e], tg.cdp, t0);
          }
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
    // the plane and metadata of chunk c are no longer read by this warp
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_empty[c % kStages]);

    if (tg.flags & CH_PASS_LAST) {
      if (tg.pass == 0) {
        best_s = best_k = 0.f;
        best_i = 0x7fffffff;
      }
      if (!(tg.flags & CH_DEAD)) {
#pragma unroll
        for (int r = 0; r < RC; ++r) {
          const int p = r >> 1;
          auto half = [&](float2 v) { return (r & 1) ? v.y : v.x; };
          float acsq = 0.f;
#pragma unroll
          for (int j = 0; j < W; ++j) acsq = __fadd_rn(acsq, __fmul_rn(half(num[p][j]), half(num[p][j])));
          const int M = n_tot - (int)((miss1 >> r) & 1);   // with a second miss the item is invalid anyway
          const float mf = (float)M, dn = half(den[p]);
          const bool ok = dn > kEpsilonF && mf > kEpsilonF && tg.napert - M < 2 && !((miss2 >> r) & 1);
          const float sem = ok ? __fdiv_rn(acsq, __fmul_rn(dn, mf)) : kSent;
          const int idx = __float_as_int(__ldg(&cand[r].w));   // -1: padding slot
          if (idx >= 0 && sem > 0.f && better(sem, idx, best_s, best_i)) {
            best_s = sem;
            best_i = idx;
            best_k = __fdiv_rn(half(lin[p]), __fmul_rn((float)W, mf));
          }
        }
      }
      if (tg.flags & CH_TASK_LAST) {
        // ---- task done for this warp; the last warp to get here merges ----
        // the previous task's merge must have read the picks
        if (ntask > 0 && !wait_bar(merge_done, (ntask - 1) & 1)) {
          give_up();
          return;
        }
        p_sem[threadIdx.x] = best_s;
        p_idx[threadIdx.x] = best_i;
        p_stk[threadIdx.x] = best_k;
        __threadfence_block();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(merge_cnt, 1) == nwarps - 1;
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) {
          __threadfence_block();
          float fs = 0.f, fk = 0.f;
          int fi = 0x7fffffff;
          for (int w2 = 0; w2 < nwarps; ++w2) {
            const int o = w2 * 32 + lane;
            if (p_sem[o] > 0.f && better(p_sem[o], p_idx[o], fs, fi)) {
              fs = p_sem[o];
              fi = p_idx[o];
              fk = p_stk[o];
            }
          }
          const int tt = tg.t0s + lane;
          if (tt < P.ns) {
            const int64_t o = (int64_t)tg.cdp * P.ns + tt;
            // no candidate above 0: CMP ctr -1, stack 0 (CMP main.cpp:219-221); CRS ctr 0
            // and the stack of item (t0 = 0, candidate 0) (CRS main.cpp:282-284)
            const bool none = !(fs > 0.f);
            P.ctr[o] = none ? (METHOD == METHOD_CMP ? -1 : 0) : fi;
            P.str[o] = none ? 0.f : fs;
            P.stk[o] = none ? (METHOD == METHOD_CMP ? 0.f : P.stt00[tg.cdp]) : fk;
          }
          __syncwarp();
          if (lane == 0) {
            *merge_cnt = 0;
            mbar_arrive(merge_done);   // the picks may be overwritten
          }
        }
        ++ntask;
      }
    }
    // the next chunk's copies: its tag is read next, and its planner is done
    if (!wait_bar(&full[(c + 1) % kStages], ((c + 1) / kStages) & 1)) {
      give_up();
      return;
    }
    seen = c + 2;
    if (warp == (c + 2) % nwarps && !prod->done && !produce()) {
      give_up();
      return;
    }
  }
}

}  // namespace semb
