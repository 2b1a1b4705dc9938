// book32.cu — the FP32 production scan of a book (its universe increments: book_gen32.cu).
//
// book_scan32_kernel: persistent, one launch for every trade.  Work items are (path block, trade),
// taken from an atomic counter per underlying count, five underlyings first: the code of a count is
// its own section of the kernel (so each keeps its registers) and a CTA that finds a count's items
// gone moves on to the next, so only the cheapest count has a tail.  A count's items go in
// path-block-major order, longest trades first, so the CTAs in flight read the same block of
// increments.  A CTA is one scenario
// group × one path group per warp: a thread steps two paths (packed FP32x2 arithmetic) of NS
// scenarios, so a warp covers 64 paths and reads each increment once for its NS scenarios.  The
// increments a (path tile, time tile) stage needs are staged in shared memory by TMA,
// double-buffered on mbarriers, and a thread steps the trade's assets in log space —
// x_f += σ_f·ΔW + (r - q_f - σ_f²/2)·dt — from shared memory and runs the Phoenix state machine of
// note.rs:150-218 with the period schedule advanced incrementally.
// What bounds it: issue slots (shared-memory loads, FP32x2 arithmetic and the ALU's minima and
// compares, about equally).  Steps go four at a time: one knock-out test on the maximum of four
// worst-of values serves them all, and the rare path that knocks out in them is settled from the
// four kept values; accruals are counted as floats.  Three-operand minima halve the worst-of.
// Measured: 128 trades × 16 scenarios × 2^14 paths 10.1 ms against 37.8 ms for one path and one
// scenario a thread with a launch per underlying count (45 of 80 TFLOP/s); 64 trades × 2^17 paths
// 38 ms against 193 ms (there the five launches' tails had left most SMs idle).
// Per path the payoff values are FP32; each 32 paths are summed by a fixed butterfly and every sum
// above that is FP64 in a fixed order, so an item's sums do not depend on which CTA ran it.
#include <algorithm>
#include <type_traits>

#include "rg_async.cuh"
#include "rg_internal.h"

namespace rg {

// ------------------------------------------------------------------ TMA-staged scan ----------
// The increments a (trade, path tile) stage needs — for each of the trade's N underlyings, TT
// steps × Pb paths — are one 3-D tensor-map box each (paths innermost), copied into one of two
// shared-memory buffers (cp.async.bulk.tensor, completion counted on that buffer's "full" mbarrier).
// The warp that is the last to be done with a buffer issues the boxes of the stage after next into it,
// so no warp waits for another (with one thread that waited for all the others and then issued, a
// book of 64 trades on 2^17 paths took 58.2 ms, 57.0 without).
// Every wait is bounded: a wait that runs out sets the status word and the kernel returns.

// Bounded wait for the phase of `bar` with the given parity to complete; sets the status word
// when it runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status) {
  if (mbar_wait_bounded(bar, parity)) return true;
  atomicExch(status, KSTAT_TIMEOUT);
  return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// a >= b as 1.0f or 0.0f.
__device__ __forceinline__ float ge_one(float a, float b) {
  float d;
  asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 splat2(float a) { return make_float2(a, a); }
template <int N>
__device__ __forceinline__ float2 worst_of_n(const float2 (&x)[N]) {
  if constexpr (N == 1) return x[0];
  else if constexpr (N == 2) return make_float2(fminf(x[0].x, x[1].x), fminf(x[0].y, x[1].y));
  else if constexpr (N == 3) return make_float2(rg_min3(x[0].x, x[1].x, x[2].x), rg_min3(x[0].y, x[1].y, x[2].y));
  else if constexpr (N == 4)
    return make_float2(rg_min3(fminf(x[0].x, x[1].x), x[2].x, x[3].x), rg_min3(fminf(x[0].y, x[1].y), x[2].y, x[3].y));
  else
    return make_float2(rg_min3(rg_min3(x[0].x, x[1].x, x[2].x), x[3].x, x[4].x),
                       rg_min3(rg_min3(x[0].y, x[1].y, x[2].y), x[3].y, x[4].y));
}

// What a CTA's threads share over the launch.
struct BookScanCta {
  float* bufs;                 // two stage buffers
  uint64_t* full;              // their mbarriers
  int* done;                   // warps done with each buffer
  const CUtensorMap* tmap;     // of this item's underlying count
  int TT;                      // steps per stage of this item
  int* status;
  int* item;    // the item the CTA is on
  double* red;  // [warp][scenario][lane] sums of the item
};

// floor(a·b / c) for non-negative a, b and positive c.
__device__ __forceinline__ int muldiv(int a, int b, int c) {
  const uint64_t p = (uint64_t)(uint32_t)a * (uint32_t)b;
  return (p >> 32) == 0 ? (int)((uint32_t)p / (uint32_t)c) : (int)(p / (uint32_t)c);
}

// One item: trade j under the warp's scenarios s0 .. s0 + NS - 1 on paths [p_lo, p_hi), PB per tile
// of which this thread steps pl and pl + 1.  acc[i]: this lane's quantity (lane & 15) of the warp's
// 32-path half (lane >> 4), summed over the tiles.
template <int N, int NS, int PB>
__device__ __forceinline__ bool book_scan32(const BookDev& bk, const BookTradeDev& tr, int j, int s0, int pl,
                                            uint64_t p_lo, uint64_t p_hi, const BookScanCta& cta, uint32_t& G,
                                            double (&acc)[NS]) {
  const int lane = threadIdx.x & 31, tid = threadIdx.x;
  float drift[NS][N], sig[NS][N], x0[NS][N], dfm[NS];
  const float* df[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const size_t pair = (size_t)j * bk.S + (s0 + i < bk.S ? s0 + i : 0);
    const BookPair32& pc = bk.pair32[pair];
#pragma unroll
    for (int f = 0; f < N; ++f) {
      drift[i][f] = __ldg(&pc.drift[f]);
      sig[i][f] = __ldg(&pc.sig[f]);
      x0[i][f] = __ldg(&pc.x0[f]);
    }
    df[i] = bk.df_f + (size_t)__ldg(&pc.dfrow) * bk.TU;
    dfm[i] = __ldg(bk.dfm_f + pair);
  }
  const int T = tr.T, PER = tr.periods, TT = cta.TT, call_start = tr.call_start;
  const float ln_cb = tr.ln_cb, coupon = tr.coupon_f;
  const int ntiles = (int)((p_hi - p_lo + PB - 1) / PB);
  const int ntt = (T + TT - 1) / TT;
  const int nst = ntiles * ntt;
  const uint32_t stage_floats = (uint32_t)(N * TT * PB);
  // stage st of this item into buffer g & 1, which no warp uses
  auto produce = [&](uint32_t g, int st) {
    const uint32_t b = g & 1u;
    const int tile = st / ntt, k = st % ntt;
    mbar_expect_tx(&cta.full[b], stage_floats * 4u);
    float* dst = cta.bufs + b * stage_floats;
#pragma unroll
    for (int f = 0; f < N; ++f)
      tma_load_3d(dst + f * TT * PB, cta.tmap, &cta.full[b], (int)(p_lo + (uint64_t)tile * PB), tr.idx[f], k * TT);
  };
  if (tid == 0) {
    produce(G, 0);
    if (nst > 1) produce(G + 1, 1);
  }
  // path state, [scenario][path of the pair]; a path that knocked out has a NaN threshold
  float2 x[NS][N], qual[NS], worst[NS];
  float ko_th[NS][2], unpaid[NS][2], cpv[NS][2], mpv[NS][2];
  int ko_step[NS][2];
  uint32_t received = 0;
  int per = 0, pend = 0, lo = 0, tile = 0, k = 0;
  float inc = 0.0f, cbt = 0.0f;
  bool fixed = false;
  // the schedule at period q, whose first step is floor(T·q / PER) = lo for the next one: its last
  // step and the coupon increment coupon_rate / max(1, steps)
  auto open_period = [&](int q) {
    per = q;
    const int a = muldiv(T, q + 1, PER);
    const bool whole = (uint64_t)(uint32_t)a * (uint32_t)PER == (uint64_t)(uint32_t)T * (uint32_t)(q + 1);
    pend = q == PER - 1 ? T - 1 : (whole ? a - 1 : a);
    inc = a - lo <= tr.ps_a ? tr.inc_a : tr.inc_b;
    lo = a;
  };
  for (int st = 0; st < nst; ++st, ++G) {
    if (k == 0) {
      // a new path tile: fresh path state
      received = 0;
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        qual[i] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int f = 0; f < N; ++f) x[i][f] = splat2(x0[i][f]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ko_th[i][h] = tr.ln_ko;
          unpaid[i][h] = cpv[i][h] = mpv[i][h] = 0.0f;
          ko_step[i][h] = -1;
        }
      }
      lo = 0;
      open_period(0);
      fixed = tr.fixed_first != 0;
      cbt = fixed ? INFINITY : ln_cb;  // the fixed first period accrues nothing
    }
    const uint32_t b = G & 1u;
    if (!mbar_wait(&cta.full[b], (G >> 1) & 1u, cta.status)) return false;
    const float* buf = cta.bufs + b * stage_floats + pl;
    const int t0 = k * TT, tn = min(TT, T - t0);
    // one step of every scenario's pair of paths: log-space Euler on the staged increments
    auto advance = [&](int tt, float2 (&w)[NS]) {
#pragma unroll
      for (int f = 0; f < N; ++f) {
        const float2 d = *reinterpret_cast<const float2*>(buf + (f * TT + tt) * PB);
#pragma unroll
        for (int i = 0; i < NS; ++i)
          x[i][f] = __fadd2_rn(__ffma2_rn(splat2(sig[i][f]), d, x[i][f]), splat2(drift[i][f]));
      }
#pragma unroll
      for (int i = 0; i < NS; ++i) w[i] = worst_of_n<N>(x[i]);
    };
    auto accrue = [&](int i, float2 w) {
      qual[i] = __fadd2_rn(qual[i], make_float2(ge_one(w.x, cbt), ge_one(w.y, cbt)));
    };
    // a path knocks out after step t with `q` accruals in the period
    auto knock_out = [&](int i, int h, int t, float q) {
      ko_th[i][h] = __int_as_float(0x7fffffff);
      ko_step[i][h] = t;
      const float due = fixed ? coupon : q * inc;
      const float carry = due > 0.0f ? unpaid[i][h] * coupon : 0.0f;
      if (due + carry > 0.0f) {
        const float d = __ldg(df[i] + t);
        cpv[i][h] = fmaf(due, d, cpv[i][h]);
        mpv[i][h] = fmaf(carry, d, mpv[i][h]);
        received |= 1u << (2 * i + h);
      }
    };
    auto half = [](float2 v, int h) { return h ? v.y : v.x; };
    // K plain steps (no period end) from tt; KO: the trade can be called in them
    auto plain_steps = [&](auto kc, auto ko, int tt) {
      constexpr int K = decltype(kc)::value;
      float2 w[K][NS];
#pragma unroll
      for (int u = 0; u < K; ++u) advance(tt + u, w[u]);
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        worst[i] = w[K - 1][i];
        if constexpr (decltype(ko)::value) {
          float2 m = w[0][i];
          if constexpr (K == 4) {
            asm("max.f32 %0, %1, %2, %3;" : "=f"(m.x) : "f"(w[0][i].x), "f"(w[1][i].x), "f"(w[2][i].x));
            asm("max.f32 %0, %1, %2, %3;" : "=f"(m.y) : "f"(w[0][i].y), "f"(w[1][i].y), "f"(w[2][i].y));
            m = make_float2(fmaxf(m.x, w[3][i].x), fmaxf(m.y, w[3][i].y));
          }
          if (m.x >= ko_th[i][0] || m.y >= ko_th[i][1]) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (half(m, h) >= ko_th[i][h]) {
                float q = half(qual[i], h);
                int at = K - 1;
#pragma unroll
                for (int u = K - 1; u >= 0; --u)
                  if (half(w[u][i], h) >= ko_th[i][h]) at = u;
#pragma unroll
                for (int u = 0; u < K; ++u)
                  if (u <= at) q += ge_one(half(w[u][i], h), cbt);
                knock_out(i, h, t0 + tt + at, q);
              }
          }
        }
#pragma unroll
        for (int u = 0; u < K; ++u) accrue(i, w[u][i]);
      }
    };
    auto plain_run = [&](auto ko, int tt, int end) {
      for (; tt + 4 <= end; tt += 4) plain_steps(std::integral_constant<int, 4>{}, ko, tt);
      for (; tt < end; ++tt) plain_steps(std::integral_constant<int, 1>{}, ko, tt);
    };
    // The schedule is the trade's, the same for every thread: the stage splits into runs of plain
    // steps before and after the call start, and the period-end step, which alone pays coupons and
    // moves to the next period.
    int tt = 0;
    while (tt < tn) {
      const int seg = min(tn, pend - t0 + 1);            // through the next period end, or the stage end
      const int plain = pend - t0 < tn ? seg - 1 : seg;  // steps [tt, plain) are not a period end
      const int ko_from = max(tt, min(plain, call_start - t0));
      plain_run(std::false_type{}, tt, ko_from);
      plain_run(std::true_type{}, ko_from, plain);
      tt = max(tt, plain);
      if (tt < seg) {
        // the period-end step (note.rs:150-218 at a period boundary)
        const int t = t0 + tt;
        float2 w[NS];
        advance(tt, w);
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          worst[i] = w[i];
          accrue(i, w[i]);
          const float d = __ldg(df[i] + t);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float q = half(qual[i], h);
            if (t >= call_start && half(w[i], h) >= ko_th[i][h]) {
              knock_out(i, h, t, q);
            } else if (ko_step[i][h] < 0) {
              const float due = fixed ? coupon : q * inc;
              if (due > 0.0f) {
                cpv[i][h] = fmaf(due, d, cpv[i][h]);
                mpv[i][h] = fmaf(unpaid[i][h] * coupon, d, mpv[i][h]);
                unpaid[i][h] = 0.0f;
                received |= 1u << (2 * i + h);
              } else if (tr.memory) {
                unpaid[i][h] += 1.0f;
              }
            }
          }
          qual[i] = make_float2(0.0f, 0.0f);
        }
        if (t + 1 < T) {
          // with at least as many steps as periods the next period is the next index
          int q = per + 1;
          if (PER > T) {
            q = min(muldiv(t + 1, PER, T), PER - 1);
            lo = muldiv(T, q, PER);
          }
          open_period(q);
          fixed = false;
          cbt = ln_cb;
        }
        ++tt;
      }
    }
    // this warp is done with the buffer; the last one refills it
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      if (atomicAdd(&cta.done[b], 1) == (int)(blockDim.x >> 5) - 1) {
        cta.done[b] = 0;  // the next count starts after the refill has landed
        __threadfence_block();
        fence_proxy_async_smem();
        if (st + 2 < nst) produce(G + 2, st + 2);
      }
    }
    if (++k == ntt) {
      // path close (note.rs:221-258) in FP32.  Each quantity is summed over the 32 paths of a half
      // warp by the butterfly over path offsets 16, 8, 4, 2, 1, the last one the thread's own pair;
      // at each offset a lane keeps the half of the quantities its lane bit names and hands over
      // the other half, so lane l ends with quantity l & 15 (the same pairs are added as when every
      // lane sums every quantity).
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        float v[2][RG_ACC];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const bool ok = s0 + i < bk.S && p_lo + (uint64_t)tile * PB + pl + h < p_hi;
          const float wf = half(worst[i], h);
          const bool ko = ko_step[i][h] >= 0;
          const float funding = ok ? (ko ? __ldg(df[i] + ko_step[i][h]) : dfm[i]) : 0.0f;
          const bool hit_ki = ok && wf <= tr.ln_ki;
          const bool put_ok = hit_ki && !ko;
          const float put = put_ok ? fmaxf(tr.strike_f - expf(wf), 0.0f) * dfm[i] : 0.0f;
          const float cn = cpv[i][h] + mpv[i][h];
          const float pv1 = ok ? (funding - 1.0f) + cn - put : 0.0f;
          const bool kof = ok && ko, rec = ok && ((received >> (2 * i + h)) & 1u);
          float* o = v[h];
          o[ACC_PV] = pv1;
          o[ACC_PV2] = pv1 * pv1;
          o[ACC_KOF] = kof ? funding - 1.0f : 0.0f;
          o[ACC_KOF2] = kof ? (funding - 1.0f) * (funding - 1.0f) : 0.0f;
          o[ACC_KIPUT] = hit_ki ? put : 0.0f;
          o[ACC_KIPUT2] = hit_ki ? put * put : 0.0f;
          o[ACC_CPN] = rec ? cn : 0.0f;
          o[ACC_CPN2] = rec ? cn * cn : 0.0f;
          o[ACC_PUT] = put;
          o[ACC_FUND] = funding;
          o[ACC_CQ] = ok ? cpv[i][h] * 10.0f : 0.0f;
          o[ACC_MQ] = ok ? mpv[i][h] * 10.0f : 0.0f;
          o[ACC_NKO] = kof ? 1.0f : 0.0f;
          o[ACC_NKI] = hit_ki ? 1.0f : 0.0f;
          o[ACC_NPUT] = put_ok ? 1.0f : 0.0f;
          o[ACC_NCPN] = rec ? 1.0f : 0.0f;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int off = 8; off > 0; off >>= 1) {
            const bool up = (lane & off) != 0;
#pragma unroll
            for (int q = 0; q < off; ++q) {
              const float mine = up ? v[h][q + off] : v[h][q], other = up ? v[h][q] : v[h][q + off];
              v[h][q] = mine + __shfl_xor_sync(0xffffffffu, other, off);
            }
          }
        acc[i] += (double)(v[0][0] + v[1][0]);
      }
      k = 0;
      ++tile;
    }
  }
  return true;
}

struct BookMaps {
  CUtensorMap m[RG_NMAX];  // per underlying count n: boxes of PB paths × 1 asset × book_stage_steps(n) steps
};

struct BookGroups {
  int lo[RG_NMAX], n[RG_NMAX];  // trades order[lo[k], lo[k] + n[k]) have k + 1 underlyings
};

// The items of the trades on N underlyings; false when a bounded wait ran out.
template <int N, int NS, int PB>
__device__ __forceinline__ bool book_scan32_group(const BookMaps& maps, const BookGroups& groups, const BookDev& bk,
                                                  uint64_t npaths, uint64_t block0, int blk_paths, int base_tt,
                                                  BookScanCta& cta, uint32_t& G, double* __restrict__ partial,
                                                  int32_t* __restrict__ counter) {
  int& s_item = *cta.item;
  auto s_red = reinterpret_cast<double(*)[NS][32]>(cta.red);
  constexpr int PG = PB / 64;  // path groups: warps that share a scenario group
  // the warp's number by a shuffle: warp-uniform to the compiler, whose loop state then needs no vector
  // registers (276 bytes of spills gone, the book 57.0 -> 53.5 ms)
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int s0 = warp / PG * NS, pl = (warp % PG) * 64 + 2 * lane;
  const int ng = groups.n[N - 1];
  const int64_t n_items = (int64_t)((npaths + blk_paths - 1) / blk_paths) * ng;
  cta.TT = book_stage_steps(N, base_tt);
  cta.tmap = &maps.m[N - 1];
  for (;;) {
    if (tid == 0) s_item = n_items > 0 ? atomicAdd(counter + N - 1, 1) : 0;
    __syncthreads();
    const int64_t item = s_item;
    __syncthreads();
    if (item >= n_items) return true;
    if (*(volatile int*)cta.status != 0) return false;
    const int64_t b = item / ng;
    const int j = bk.order[groups.lo[N - 1] + item % ng];
    const uint64_t p_lo = (uint64_t)b * blk_paths;
    const uint64_t p_hi = p_lo + blk_paths < npaths ? p_lo + blk_paths : npaths;
    double acc[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) acc[i] = 0.0;
    if (!book_scan32<N, NS, PB>(bk, bk.trades[j], j, s0, pl, p_lo, p_hi, cta, G, acc)) return false;
    // the scenario's 32-path columns in path order
#pragma unroll
    for (int i = 0; i < NS; ++i) s_red[warp][i][lane] = acc[i];
    __syncthreads();
    for (int o = tid; o < bk.S * RG_ACC; o += blockDim.x) {
      const int sc = o / RG_ACC, kk = o % RG_ACC;
      double v = 0.0;
      for (int p = 0; p < PG; ++p)
        for (int h = 0; h < 2; ++h) v += s_red[sc / NS * PG + p][sc % NS][h * 16 + kk];
      partial[(((size_t)(block0 + b) * bk.n_trades + j) * bk.S + sc) * RG_ACC + kk] = v;
    }
  }
}

template <int NS, int PB>
__global__ void __launch_bounds__(512, 1) book_scan32_kernel(const __grid_constant__ BookMaps maps,
                                                             const __grid_constant__ BookGroups groups, BookDev bk,
                                                             uint64_t npaths, uint64_t block0, int blk_paths, int base_tt,
                                                             double* __restrict__ partial, int32_t* __restrict__ counter,
                                                             int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ uint64_t s_bars[2];
  __shared__ int s_done[2];
  __shared__ int s_item;
  __shared__ double s_red[16 * NS * 32];
  BookScanCta cta;
  cta.item = &s_item;
  cta.red = s_red;
  cta.bufs = reinterpret_cast<float*>(smem_raw);
  cta.full = s_bars;
  cta.done = s_done;
  cta.status = status;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&cta.full[b], 1);
      s_done[b] = 0;
    }
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t G = 0;
  // a wait that ran out has set the status: nothing more is issued
  if (!book_scan32_group<5, NS, PB>(maps, groups, bk, npaths, block0, blk_paths, base_tt, cta, G, partial, counter)) return;
  if (!book_scan32_group<4, NS, PB>(maps, groups, bk, npaths, block0, blk_paths, base_tt, cta, G, partial, counter)) return;
  if (!book_scan32_group<3, NS, PB>(maps, groups, bk, npaths, block0, blk_paths, base_tt, cta, G, partial, counter)) return;
  if (!book_scan32_group<2, NS, PB>(maps, groups, bk, npaths, block0, blk_paths, base_tt, cta, G, partial, counter)) return;
  book_scan32_group<1, NS, PB>(maps, groups, bk, npaths, block0, blk_paths, base_tt, cta, G, partial, counter);
}

// The launch shape (all shapes add the same 32-path sums): NS scenarios a thread (two, or one for a single scenario), a scenario group per
// ceil(S / NS), as many path groups of 64 as fit 16 warps and a 256-path box.  One CTA per SM (the
// stage buffers take most of its shared memory), so a grid of fewer CTAs leaves whole SMs free.
Book32Shape book32_shape(int S, int sm_count, uint64_t paths, int n_trades) {
  Book32Shape sh{};
  if (S > 32) raise(RG_ERR_INVALID_ARGUMENT, "at most 32 scenarios per book launch");
  sh.ns = S > 1 ? 2 : 1;
  const int groups = (S + sh.ns - 1) / sh.ns;
  int pg = 4;
  while (pg * groups > 16) pg >>= 1;
  sh.Pb = 64 * pg;
  sh.threads = 32 * groups * pg;
  // stage depth for five underlyings: as many steps as two stage buffers of 168 KB hold
  sh.TT = 64;
  while (book32_smem(sh.TT, sh.Pb) > 168 * 1024) sh.TT >>= 1;
  sh.grid = sm_count;
  // a work item is one trade over a block of at most 2048 paths; a small book (few paths or trades)
  // takes smaller blocks, so that the persistent CTAs still have 16 items each and end together
  sh.blk_paths = 2048;
  const uint64_t nt = (uint64_t)(n_trades > 0 ? n_trades : 1);
  while (sh.blk_paths > sh.Pb &&
         (paths + (uint64_t)sh.blk_paths - 1) / (uint64_t)sh.blk_paths * nt < 16 * (uint64_t)sm_count)
    sh.blk_paths >>= 1;
  return sh;
}

void launch_book_trade32(const BookDev& bk, const Book32Shape& sh, const CUtensorMap* maps, uint64_t npaths,
                         uint64_t block0, const int* group_lo, const int* group_n, double* partial,
                         int32_t* counter, int* status, cudaStream_t s) {
  BookMaps bm;
  BookGroups gr;
  for (int n = 0; n < RG_NMAX; ++n) {
    gr.lo[n] = group_lo[n];
    gr.n[n] = group_n[n];
  }
  for (int n = 0; n < RG_NMAX; ++n) bm.m[n] = maps[n];
  const int smem = book32_smem(sh.TT, sh.Pb);
  if (smem > 168 * 1024) raise(RG_ERR_GPU_ERROR, "book stage buffers exceed the shared-memory limit");
  auto go = [&](auto kernel) {
    // process-wide attribute: always the same value, so concurrent engines never lower it
    cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 168 * 1024), "book smem attribute");
    cuda_check(cudaMemsetAsync(counter, 0, sizeof(int32_t) * RG_NMAX, s), "book counter reset");
    kernel<<<sh.grid, sh.threads, smem, s>>>(bm, gr, bk, npaths, block0, sh.blk_paths, sh.TT, partial, counter, status);
    cuda_check(cudaGetLastError(), "book_scan32_kernel launch");
  };
  if (sh.ns == 1) go(book_scan32_kernel<1, 256>);
  else if (sh.Pb == 256) go(book_scan32_kernel<2, 256>);
  else if (sh.Pb == 128) go(book_scan32_kernel<2, 128>);
  else go(book_scan32_kernel<2, 64>);
}

// out[pair][k] = Σ_b partial[b·stride_b + pair·stride_pair + k], b in order.
__global__ void book_reduce_kernel(const double* __restrict__ partial, int64_t blocks, int64_t stride_b,
                                   int64_t stride_pair, int pairs, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs * RG_ACC) return;
  const int pair = i / RG_ACC, k = i % RG_ACC;
  double v = 0.0;
  for (int64_t b = 0; b < blocks; ++b) v += partial[b * stride_b + (int64_t)pair * stride_pair + k];
  out[i] = v;
}

void launch_book_reduce_strided(const double* partial, int64_t blocks, int64_t stride_b, int64_t stride_pair,
                                int pairs, double* out, cudaStream_t s) {
  const int n = pairs * RG_ACC;
  book_reduce_kernel<<<(n + 255) / 256, 256, 0, s>>>(partial, blocks, stride_b, stride_pair, pairs, out);
  cuda_check(cudaGetLastError(), "book_reduce_kernel launch");
}

}  // namespace rg
