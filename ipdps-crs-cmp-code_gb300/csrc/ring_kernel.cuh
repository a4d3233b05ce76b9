// Batched CMP search kernel with item pairs in a staging ring (sm_103a).
//
// The batched arithmetic of semb_search_kernel on item pairs: a thread's candidates go two
// per FP32x2 instruction, and their window samples come as scalar shared-memory loads
// straight into the halves, from planes of plain FP32 samples (4 bytes each instead of
// 16-byte entries: w + 1 wavefronts per item, and a chunk holds up to 128 traces). 16-bit
// stores are converted once per chunk, FP32 stores land by TMA in place. The ring is
// semb_filter_kernel's: rotating planner warp, mbarrier hand-offs, a work queue, the last
// warp of a task merging the top-4 lists.
//
// What bounds it: latency and the FP32 pipe together (w = 5: 25 FP32 operations per
// trace-evaluation on 33 cycles).  256 CMPs of the uneven-fold line (256 velocities, w = 5)
// 10.29 ms in the two-barrier kernel (79% of the shared-memory pipe for its 16-byte entries),
// 9.45 here; w = 11, 90 velocities 0.57 -> 0.46.  The trace loop unrolled by two: 1 to 2%.
// ring_variant() (launch.cu) says where it is used and has both sides.
#pragma once

#include "filter_kernel.cuh"

namespace semb {

// Traces whose energy one FP32 chain sums before it is folded into the Kahan total (almost
// twice as many where a chunk's last in-range traces and the others meet).  A chunk holds up
// to 128; the two-barrier kernel's entries leave room for some 60, in two chains up to w = 5.
// In one chain per chunk the semblance's rms distance from 64 bits was above that kernel's
// with the FP32 store: w = 7, fold 200 2.70e-7 against 2.67e-7 in chains of 64, 2.81e-7 in
// whole chunks, 2.63e-7 so.  It costs 1.4% on the uneven-fold line (9.32 -> 9.45 ms), up to 5%
// with 10 candidates per thread; one copy of the fold for all traces 3.3% and 2%, chunks of
// 32 traces 7%.
constexpr int kRingFold = 32;

// Shared-memory layout (bytes), shared by host and device:
//   [0, 128)   mbarriers (full[3], q_full[3], q_empty[3], merge_done) and the merge counter
//   prod       producer state
//   meta[4]    chunk metadata, tag[4] chunk tags
//   src[4]     copy descriptors
//   tops       running top-4 per thread [3][4][NT]
//   kahan      Kahan totals and compensations [2][RC][NT]
//   plane[3]   staged windows, FP32, each followed by its zero block
//   raw[2]     16-bit windows (TMA destination; 16-bit stores only)
struct RingLayout {
  size_t prod, meta, tag, src, tops, kahan, plane, plane_stride, raw, raw_stride, total;
};

__host__ __device__ inline RingLayout ring_layout(int rc, int cap, int storage, int nt) {
  RingLayout L;
  L.prod = 128;
  L.meta = L.prod + align128(sizeof(Producer));
  L.tag = L.meta + kMetaRing * kMetaBytes;
  L.src = L.tag + align128(kMetaRing * sizeof(ChunkTag));
  L.tops = L.src + (size_t)kMetaRing * kMaxChunk * 16;
  L.kahan = L.tops + align128(3 * (size_t)kTopK * nt * 4);
  L.plane = L.kahan + align128(2 * (size_t)rc * nt * 4);
  L.plane_stride = align128(((size_t)cap + kZeroSlots) * 4);
  L.raw = L.plane + kStages * L.plane_stride;
  L.raw_stride = storage == STORE_F32 ? 0 : align128((size_t)cap * 2);
  L.total = L.raw + kRawBufs * L.raw_stride;
  return L;
}

// W: window.  RC: candidates per thread (even).  NT: threads per CTA.
template <int W, int RC, int NT>
__global__ void __launch_bounds__(NT, 1) semb_ring_kernel(KParams P) {
  static_assert(RC % 2 == 0, "item pairs");
  constexpr int K = kTopK, RP = RC / 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const bool f32 = P.storage == STORE_F32;
  const RingLayout L = ring_layout(RC, P.cap, P.storage, NT);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);   // copies landed: [kStages] (f32) or [kRawBufs]
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
  auto full_at = [&](int c) { return f32 ? &full[c % kStages] : &full[c % kRawBufs]; };
  auto full_phase = [&](int c) { return (uint32_t)((f32 ? c / kStages : c / kRawBufs) & 1); };
  float* top_s = reinterpret_cast<float*>(smem_raw + L.tops);   // [K][NT]
  int* top_i = reinterpret_cast<int*>(top_s + K * NT);
  float* top_k = top_s + 2 * K * NT;
  float* kahan_hi = reinterpret_cast<float*>(smem_raw + L.kahan) + threadIdx.x;   // [RC][NT]
  float* kahan_lo = kahan_hi + RC * NT;

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
    const int issued = min(prod->next, seen + (f32 ? kStages : kRawBufs));
    for (int c = seen; c < issued; ++c) wait_bar(full_at(c), full_phase(c));
  };

  // the planner warp: plan the next chunk of the stream and start its copies
  auto produce = [&]() -> bool {
    const int c = prod->next;
    // F32: the copies land in the plane the warps computed chunk c - kStages from
    if (f32 && c >= kStages && !wait_bar(&q_empty[c % kStages], (c / kStages - 1) & 1)) return false;
    ChunkMeta* m = meta_at(c);
    ChunkTag* tg = tag_at(c);
    int4* src = src_at(c);
    auto issue = [&]() {
      if (f32) issue_windows<true>(P, m, src, plane_at(c), full_at(c));
      else issue_windows<false>(P, m, src, raw_at(c), full_at(c));
    };
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
        issue();
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
    plan_chunk<METHOD_CMP, FORM_FAST>(P, P.pass_bounds + pass * 8, pos, end, prod->T_lo, prod->T_hi, m, src);
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
    issue();
    return true;
  };

  // wait for chunk c's samples; 16-bit: convert this warp's share of it first
  auto convert_step = [&](int c) -> bool {
    if (!f32 && c >= kStages && !wait_bar(&q_empty[c % kStages], (c / kStages - 1) & 1)) return false;
    if (!wait_bar(full_at(c), full_phase(c))) return false;
    seen = c + 1;
    if (!f32) {
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
  const float2 k23 = make_float2(8388608.0f, 8388608.0f), km23 = make_float2(-8388608.0f, -8388608.0f);
  const float2 kNeg = make_float2(-1.0f, -1.0f);
  float T2 = 0.f;
  float2 cc[RP], num[RP][W], den[RP];
  int n_tot = 0;                   // staged traces of the pass
  uint32_t miss1 = 0, miss2 = 0;   // items out of range on one, on two or more of them
  float last_s = 0.f;
  int last_i = 0x7fffffff;
  int ntask = 0;

  for (int c = 0;; ++c) {
    const ChunkTag tg = *tag_at(c);   // visible: this thread saw chunk c's copies land
    if (tg.flags & CH_END) break;
    if (!f32) {
      // convert the next chunk (it exists: this one is not the end), then plan the one
      // after it into the raw buffer that this chunk has left
      if (!convert_step(c + 1) || !wait_bar(&q_full[c % kStages], (c / kStages) & 1) ||
          (warp == (c + 2) % nwarps && !prod->done && !produce())) {
        give_up();
        return;
      }
    }
    const ChunkMeta* meta = meta_at(c);
    const float4* cand = P.cand + tg.pass * P.cpp + warp * RC;
    const int t0 = min(tg.t0s + lane, P.ns - 1);
    if (tg.flags & CH_PASS_FIRST) {
      T2 = (float)t0 * (float)t0;
#pragma unroll
      for (int p = 0; p < RP; ++p) {
        cc[p] = make_float2(__ldg(&cand[2 * p].z), __ldg(&cand[2 * p + 1].z));
#pragma unroll
        for (int j = 0; j < W; ++j) num[p][j] = make_float2(0.f, 0.f);
        den[p] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int r = 0; r < RC; ++r) {
        kahan_hi[r * NT] = 0.f;
        kahan_lo[r * NT] = 0.f;
      }
      n_tot = 0;
      miss1 = miss2 = 0;
    }

    // ---- compute chunk c ----
    const int n = meta->n, n_in = meta->n_in;
    const uint32_t plane = smem_u32(plane_at(c)), top = plane + 4u * (uint32_t)P.cap;
    const float2 T22 = make_float2(T2, T2);
    // one pair's window at sample addresses ax, ay with weights x
    auto window = [&](int p, uint32_t ax, uint32_t ay, float2 x) {
      float2 s0 = make_float2(lds32(ax), lds32(ay));
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float2 s1 = make_float2(lds32(ax + 4u * (j + 1)), lds32(ay + 4u * (j + 1)));
        const float2 v = __ffma2_rn(__ffma2_rn(s0, kNeg, s1), x, s0);
        num[p][j] = __fadd2_rn(num[p][j], v);
        den[p] = __ffma2_rn(v, v, den[p]);
        s0 = s1;
      }
    };
    // Kahan: fold the energy since the last time into the compensated totals
    auto fold = [&]() {
#pragma unroll
      for (int r = 0; r < RC; ++r) {
        const float hi = kahan_hi[r * NT], lo = kahan_lo[r * NT];
        const float yv = ((r & 1) ? den[r >> 1].y : den[r >> 1].x) - lo;
        const float tv = hi + yv;
        kahan_lo[r * NT] = (tv - hi) - yv;
        kahan_hi[r * NT] = tv;
      }
#pragma unroll
      for (int p = 0; p < RP; ++p) den[p] = make_float2(0.f, 0.f);
    };
    for (int e0 = 0; e0 < n_in; e0 += kRingFold) {   // every item in range
      if (e0 > 0) fold();
      const int e1 = min(n_in, e0 + kRingFold);
#pragma unroll 2
      for (int e = e0; e < e1; ++e) {
        const float4 g = meta->geo[e];
        const uint32_t base = plane + 4u * (uint32_t)(__float_as_int(g.w) - P.tau) - 4u * 0x4B000000u;
        const float2 gz = make_float2(g.z, g.z);
#pragma unroll
        for (int p = 0; p < RP; ++p) {
          const float2 q = __ffma2_rn(cc[p], gz, T22);
          const float2 t = make_float2(sqrt_fast(q.x), sqrt_fast(q.y));
          const float2 y = __fadd2_rz(t, k23);
          const float2 x = __ffma2_rn(__fadd2_rn(y, km23), kNeg, t);   // t - floor(t)
          if constexpr (SEMB_CHECKED) {
            const int i0 = __float_as_int(g.w) - P.tau - 0x4B000000;
            report_window(P.status, __float_as_int(y.x) + i0, W, src_at(c)[e], tg.cdp, t0);
            report_window(P.status, __float_as_int(y.y) + i0, W, src_at(c)[e], tg.cdp, t0);
          }
          window(p, min(__float_as_uint(y.x) * 4u + base, top), min(__float_as_uint(y.y) * 4u + base, top), x);
        }
      }
    }
    // the other traces: per-item range checks; an out-of-range item reads the zero block
    // with weight 0 and does not count
    for (int e = kMaxChunk - (n - n_in); e < kMaxChunk; ++e) {
      if ((kMaxChunk - e) % kRingFold == 0) fold();
      const float4 g = meta->geo[e];
      const int soff = __float_as_int(g.w);
#pragma unroll
      for (int p = 0; p < RP; ++p) {
        const float2 q = __ffma2_rn(cc[p], make_float2(g.z, g.z), T22);
        const float2 t = make_float2(sqrt_fast(q.x), sqrt_fast(q.y));   // NaN below 0: out of range
        const float2 y = __fadd2_rz(t, k23);
        const int rx = __float_as_int(y.x) - (0x4B000000 + P.tau), ry = __float_as_int(y.y) - (0x4B000000 + P.tau);
        const bool okx = (unsigned)rx <= span, oky = (unsigned)ry <= span;
        const float2 x = make_float2(okx ? t.x - (y.x - 8388608.0f) : 0.f, oky ? t.y - (y.y - 8388608.0f) : 0.f);
        if constexpr (SEMB_CHECKED) {
          if (okx) report_window(P.status, soff + rx, W, src_at(c)[e], tg.cdp, t0);
          if (oky) report_window(P.status, soff + ry, W, src_at(c)[e], tg.cdp, t0);
        }
        const uint32_t off = (okx ? 0u : 1u << (2 * p)) | (oky ? 0u : 2u << (2 * p));
        miss2 |= miss1 & off;
        miss1 |= off;
        window(p, okx ? min(plane + 4u * (uint32_t)(soff + rx), top) : top,
               oky ? min(plane + 4u * (uint32_t)(soff + ry), top) : top, x);
      }
    }
    n_tot += n;
    // the plane and metadata of chunk c are no longer read by this warp
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_empty[c % kStages]);
    fold();

    if (tg.flags & CH_PASS_LAST) {
      // ---- finalize the pass's items into this thread's top-4 ----
      if (tg.pass == 0) {
        // the first pass of a task: the previous task's merge must have read the lists
        if (ntask > 0 && !wait_bar(merge_done, (ntask - 1) & 1)) {
          give_up();
          return;
        }
#pragma unroll
        for (int q = 0; q < K; ++q) {
          top_s[q * NT + threadIdx.x] = 0.f;
          top_i[q * NT + threadIdx.x] = 0x7fffffff;
          top_k[q * NT + threadIdx.x] = 0.f;
        }
        last_s = 0.f;
        last_i = 0x7fffffff;
      }
      if (!(tg.flags & CH_DEAD)) {
#pragma unroll
        for (int r = 0; r < RC; ++r) {
          const int p = r >> 1;
          auto half = [&](float2 v) { return (r & 1) ? v.y : v.x; };
          float acsq = 0.f, lin = 0.f;
#pragma unroll
          for (int j = 0; j < W; ++j) {
            acsq = fmaf(half(num[p][j]), half(num[p][j]), acsq);
            lin += half(num[p][j]);
          }
          const float dn = kahan_hi[r * NT] - kahan_lo[r * NT];
          const int M = n_tot - (int)((miss1 >> r) & 1);   // with a second miss the item is invalid anyway
          const float mf = (float)M;
          const bool ok = dn > kEpsilonF && M > 0 && tg.napert - M < 2 && !((miss2 >> r) & 1);
          const float sem = ok ? __fdividef(acsq, dn * mf) : 0.f;
          const int idx = __float_as_int(__ldg(&cand[r].w));   // -1: padding slot
          if (idx >= 0 && sem > 0.f && better(sem, idx, last_s, last_i)) {
            // sorted insert (descending semblance, ascending index)
            float cs = sem, ck = __fdividef(lin, (float)W * mf);
            int cidx = idx;
#pragma unroll
            for (int q = 0; q < K; ++q) {
              const int o = q * NT + threadIdx.x;
              const float bs = top_s[o];
              const int bi = top_i[o];
              if (better(cs, cidx, bs, bi)) {
                const float bk = top_k[o];
                top_s[o] = cs;
                top_i[o] = cidx;
                top_k[o] = ck;
                cs = bs;
                cidx = bi;
                ck = bk;
              }
            }
            last_s = top_s[(K - 1) * NT + threadIdx.x];
            last_i = top_i[(K - 1) * NT + threadIdx.x];
          }
        }
      }
      if (tg.flags & CH_TASK_LAST) {
        // ---- task done for this warp; the last warp to get here merges ----
        merge_task<NT>(P, tg, top_s, top_i, top_k, merge_cnt, merge_done);
        ++ntask;
      }
    }
    if (f32) {
      // the next chunk's copies: its tag is read next, and its planner is done
      if (!convert_step(c + 1) || (warp == (c + 2) % nwarps && !prod->done && !produce())) {
        give_up();
        return;
      }
    }
  }
}

}  // namespace semb
