// phoenix32d.cu — the FP32 kernel for single-scenario launches: one or two paths per thread, everything
// in registers, no shared-memory time tiles and no CTA barriers.
//
// The tiled kernel (phoenix32.cu) stages a tile's normals and Brownian increments in shared
// memory so that the scenarios of a path share one generation; with one scenario there is nothing
// to share and the staging only costs occupancy; the tiled kernel wins with two or more scenarios, and
// on few paths, where one path per thread leaves too few warps to hide the per-step latency
// (p32_direct, rg_internal.h, has the line and both sides).  Here a warp walks 32 or 64 consecutive
// paths through time, a thread one path or the two that are 32 apart (p32_direct_ppt has that line):
//   * Sobol points from consumption-order tables staged for the launch (sobol_lut_kernel,
//     book_gen32.cu): the warp's points lie in two or three aligned 32-point blocks, and
//     Gray codes are linear over XOR, so a point is the block's high-bit term X(gray(a)) — one
//     coalesced row of transposed directions per set bit of gray(a), for a batch of the next
//     32 / N nodes' dimensions at once, kept in shared memory — XOR the lane's low-bit term, one
//     coalesced 128-byte row per dimension, the same for a thread's two paths; without the tables
//     (another offset within a block), by warp cooperation: x(n) for the warp's first point as a
//     shuffle reduction over the set bits of its Gray code, and the Gray recurrence
//     x(n) = x(n-1) ^ v[ctz(n)] as an XOR scan over the lanes;
//   * the digital shift (or Owen scramble) and the FP32 inverse normals of a node together
//     (rg_packed.cuh);
//   * the streamed Brownian bridge per factor, the top of its anchor stack in registers and the rest
//     laid out [depth][factor][lane] so that a warp's accesses (the depth is warp-uniform) hit 32 banks;
//   * the correlation with the scenario's Cholesky factor, the log-space GBM / Dupire step and the
//     Phoenix state machine.
// Two paths a thread share the node, the schedule and the constants, and step in packed FP32x2
// arithmetic: 5 assets take 279 instructions per step of 32 paths against 370.  What bounds it is issue
// (65% of the slots used, the rest waiting for the gathers and dependent arithmetic of 16 warps an SM).
// 2^21 paths × 1260 steps of 5 assets under local vol: 40 ms at one path a thread; 35.0 with the stack's
// top in registers, a step's local-vol rows adjacent and the warp number, and so the loops, uniform to
// the compiler; 34.4 at two paths; 28.5 with the deep stack outside shared memory and the kernel free of
// the other lanes' generation code; 27.3 with the cells' addresses by one multiply-add.  The lanes
// without tables have a kernel of their own, whose long generation wants the registers: 2^20 paths on
// Halton points 92.7 ms in one kernel for all lanes, 97.8 with the lookup's constants in registers, 70.8
// with them in shared memory.
// Every operation of the per-path arithmetic is the one phoenix32.cu performs, in the same order,
// so a path's FP32 payoff values are identical in both kernels.  Each 32 consecutive paths are one
// chunk of the sums, added by the same FP32 shuffle butterfly and written as FP64 to
// partial[chunk] as the tiled kernel writes them, so both kernels — and every launch
// shape of either — give the same sums.
#include "p32_path.cuh"
#include "rg_internal.h"

namespace rg {

#define P32D_THREADS 256
#define P32D_WARPS (P32D_THREADS / 32)
// CTAs per SM, and with them the registers: at one path a thread 64 up to three assets and 80 for four or
// five; at two 80 up to three (2^20 paths of 3 assets × 252 steps 1.65 ms against 1.82 at 112) and 128.
__host__ __device__ constexpr int p32d_min_ctas(int n, int ppt) { return ppt == 2 ? (n <= 3 ? 3 : 2) : (n <= 3 ? 4 : 3); }
// The anchor stack below its top: a step's nodes lie at the end of the stack, and slot d counted from the
// deepest stack's end is used every 2^d steps, so the last kFastSlots slots are in shared memory,
// [slot][factor][lane], and at two paths a thread the others in local memory: all of them in shared
// memory left 28 KB of L1 for the local-vol rows of 5 assets, and 37% of the gathers hit instead of 90%.
constexpr int kFastSlots = 5, kSlowSlots = 20;
// Bytes of dynamic shared memory per warp: the stack's fast slots, and the high-bit Sobol terms of a batch of nodes, one row for each 32-point block that the warp's points lie in.
__host__ __device__ constexpr int p32d_slow(int ppt, int stack_max) {
  return ppt == 2 && stack_max - 1 > kFastSlots ? stack_max - 1 - kFastSlots : 0;
}
__host__ __device__ constexpr int p32d_slots(int ppt, int stack_max) {
  return stack_max > 2 ? stack_max - 1 - p32d_slow(ppt, stack_max) : 1;
}
__host__ __device__ constexpr int p32d_hi_row(int n) { return 32 / n * n < 32 ? 31 : 33; }  // odd: other banks
__host__ __device__ constexpr uint32_t p32d_warp_bytes(int n, int ppt, int stack_max) {
  return (uint32_t)(p32d_slots(ppt, stack_max) * n * ppt * 128 + ((ppt + 1) * p32d_hi_row(n) * 4 + 15) / 16 * 16);
}

// Bytes of dynamic shared memory per CTA: its warps', and at one path a thread the lookup's constants.
__host__ __device__ constexpr uint32_t p32d_smem(int n, int ppt, int stack_max) {
  return p32d_warp_bytes(n, ppt, stack_max) * P32D_WARPS + (ppt == 1 ? (uint32_t)n * 16u : 0u);
}

// LUT: Sobol points from the staged consumption-order tables, built for this launch's offset within a
// 32-point block; else, at one path a thread, any lane, Sobol points by the warp cooperation of
// rg_warp_sobol.
template <int N, bool LV, bool REC, int PPT, bool LUT>
__global__ void __launch_bounds__(P32D_THREADS, p32d_min_ctas(N, PPT)) phoenix32d_kernel(
    DevTrade tr, DevTables tb, const DevScen32* __restrict__ scen32, int stack_max, int n_surf, float ln_ko, float ln_cb,
    float ln_ki, uint64_t path0, uint64_t npaths, double* __restrict__ partial, int32_t* __restrict__ ko_steps,
    rg_path_record* __restrict__ records) {
  using V = PVec<PPT>;
  extern __shared__ __align__(16) unsigned char s_raw[];
  // the warp's number by a shuffle, which makes it, and the loops that it bounds, warp-uniform to the
  // compiler: schedule words, row pointers and loop counters then live in uniform registers
  const int lane = threadIdx.x & 31, wib = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int T = (int)tr.steps;
  const int gx = tr.gx;
  const V gxm1 = V::splat((float)(gx - 1));
  const V two23 = V::splat(8388608.0f);
  const V nhdt = V::splat(tr.neg_half_dt_f);
  unsigned char* const wmem = s_raw + (size_t)wib * p32d_warp_bytes(N, PPT, stack_max);
  V* const stk = reinterpret_cast<V*>(wmem) + lane;  // fast slot d, factor f at stk[(d * N + f) * 32]
  uint32_t* const s_hi = reinterpret_cast<uint32_t*>(wmem + p32d_slots(PPT, stack_max) * N * PPT * 128);
  // the scenario's constants: Cholesky factor, drifts, flat vols or local-vol lookup
  V Lf[N * (N + 1) / 2], mu[N], sig[N];
  float lva[N], lvb[N];
  int32_t lvo[N];
  // at one path a thread, where registers are short, the lookup's constants are in shared memory
  float4* const s_lv = reinterpret_cast<float4*>(s_raw + (size_t)P32D_WARPS * p32d_warp_bytes(N, PPT, stack_max));
  {
    const float inv_gxm1 = 1.0f / (float)(gx - 1);
    int q = 0;
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b) Lf[q++] = V::splat(scen32->L[a * N + b]);
#pragma unroll
    for (int f = 0; f < N; ++f) {
      mu[f] = V::splat(scen32->mu_dt[f]);
      sig[f] = V::splat(scen32->sig[f]);
      lva[f] = scen32->a_u[f] * inv_gxm1;
      lvb[f] = scen32->inv_h[f] * inv_gxm1;
      lvo[f] = scen32->surf_off[f] - 0x4B000000;  // less the bias of the grid index
      if (PPT == 1 && threadIdx.x == 0) s_lv[f] = make_float4(lva[f], lvb[f], __int_as_float(lvo[f]), 0.0f);
    }
    if (PPT == 1) __syncthreads();
  }
  V deep[PPT == 2 ? kSlowSlots : 1][N];
  const int slow = PPT == 2 ? p32d_slow(PPT, stack_max) : 0;
  const int row_step = n_surf * gx;
  const uint64_t groups = (npaths + 32 * PPT - 1) / (32 * PPT);
  constexpr int kNb = 32 / N;  // nodes per batch of high-bit terms
  constexpr int kRow = p32d_hi_row(N);
  const int upper = (uint32_t)tb.sob_lut_o + (uint32_t)lane >= 32u ? kRow : 0;  // point in the next 32-block
  for (uint64_t grp = (uint64_t)blockIdx.x * P32D_WARPS + wib; grp < groups; grp += (uint64_t)gridDim.x * P32D_WARPS) {
    const uint64_t n1 = path0 + grp * (32 * PPT) + 1;  // Sobol point of the warp's first path
    const uint32_t ga = (uint32_t)((n1 & ~(uint64_t)31) ^ ((n1 & ~(uint64_t)31) >> 1));  // gray(a)
    // the directions that the term of the next block and of the one after it add: the lowest set bit of
    // their number, and 5; and 4
    uint32_t cw[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) cw[j] = min(__ffsll((long long)((n1 >> 5) + 1 + j)) - 1 + 5, 31);
    int cb = -kNb;  // first node of the batch in s_hi
    // the lanes' low-bit terms of the next node, loaded a node ahead so that their latency
    // overlaps the current step; both paths of a thread have the same (their points are 32 apart)
    uint32_t lnext[N];
#pragma unroll
    for (int f = 0; f < N; ++f) lnext[f] = LUT ? __ldg(tb.sob_lut + (size_t)f * 32 + lane) : 0u;
    V x[N], wcur[N], top[N];  // `top`: the anchor stack's top; W(0) = 0 before the first node
#pragma unroll
    for (int f = 0; f < N; ++f) {
      x[f] = V::splat(scen32->x0[f]);
      wcur[f] = top[f] = V::splat(0.0f);
    }
    int sp = -1;  // slots of the stack below `top`, less the value before the first node
    auto push = [&](int d) {
      if (PPT == 2 && d < slow) {
#pragma unroll
        for (int f = 0; f < N; ++f) deep[max(d, 0)][f] = top[f];
      } else {
        V* slot = stk + max(d - slow, 0) * (N * 32);
#pragma unroll
        for (int f = 0; f < N; ++f) slot[f * 32] = top[f];
      }
    };
    auto pop = [&](int d) {
      if (PPT == 2 && d < slow) {
#pragma unroll
        for (int f = 0; f < N; ++f) top[f] = deep[max(d, 0)][f];
      } else {
        const V* slot = stk + max(d - slow, 0) * (N * 32);
#pragma unroll
        for (int f = 0; f < N; ++f) top[f] = slot[f * 32];
      }
    };
    P32Phoenix ph[PPT];
#pragma unroll
    for (int j = 0; j < PPT; ++j) ph[j].alive = grp * (32 * PPT) + 32 * j + lane < npaths;
    const float2* rows = tb.lv_rows;
    int c = 0;
    for (int t = 0; t < T; ++t) {
      // bridge nodes consumed at this step: normals, then the streamed bridge (qmc.rs:158-191)
      const int c1 = __ldg(tb.node_off + t + 1);
      for (; c < c1; ++c) {
        const V cf = V::splat(__ldg(tb.node_cf + c));
        push(sp++);
        // the node's value of factor f, from its normal
        auto node = [&](int f, V z) { top[f] = V::fma(z, cf, V::mul(V::splat(0.5f), V::add(wcur[f], top[f]))); };
        if constexpr (LUT) {
          if (c >= cb + kNb) {
            // the high-bit terms X(gray(a)) of q = c·N .. (c + kNb)·N - 1, lane l holding q0 + l:
            // one coalesced row of transposed directions per set bit of gray(a)
            cb = c;
            __syncwarp();  // every lane has read the previous batch
            const int q = c * N + lane;
            if (lane < kNb * N && q < tb.sob_nq) {
              uint32_t h = 0;
              for (uint32_t g = ga; g; g &= g - 1u) h ^= __ldg(tb.sob_t + (size_t)(__ffs(g) - 1) * tb.sob_nq + q);
              const uint32_t v4 = __ldg(tb.sob_t + (size_t)4 * tb.sob_nq + q);
              s_hi[lane] = h;
#pragma unroll
              for (int j = 0; j < PPT; ++j) {
                h ^= v4 ^ __ldg(tb.sob_t + (size_t)cw[j] * tb.sob_nq + q);
                s_hi[(j + 1) * kRow + lane] = h;
              }
            }
            __syncwarp();
          }
          const uint32_t* hb = s_hi + (c - cb) * N + upper;
          uint32_t xs[PPT][N];
#pragma unroll
          for (int f = 0; f < N; ++f)
#pragma unroll
            for (int j = 0; j < PPT; ++j) {
              xs[j][f] = hb[f + kRow * j] ^ lnext[f];
              if (PPT == 1 && tr.scrambler != RG_SCRAMBLE_DIGITAL_SHIFT)
                xs[j][f] = rg_owen(xs[j][f], (uint64_t)__ldg(tb.node_k + c) * N + f, tr.seed);
            }
          if ((c + 1) * N < tb.sob_nq) {
            const uint32_t* low = tb.sob_lut + (size_t)(c + 1) * (N * 32) + lane;
#pragma unroll
            for (int f = 0; f < N; ++f) lnext[f] = __ldg(low + f * 32);
          }
          // the inverse normals in packed pairs: of both paths, or of two factors
          constexpr int kP = PPT == 2 ? N : (N + 1) / 2;
          uint32_t xa[kP], xb[kP];
          float2 z[kP];
#pragma unroll
          for (int i = 0; i < kP; ++i) {
            xa[i] = PPT == 2 ? xs[0][i] : xs[0][2 * i];
            xb[i] = PPT == 2 ? xs[PPT - 1][i] : xs[0][min(2 * i + 1, N - 1)];
          }
          rg_probit32x2(xa, xb, z);
#pragma unroll
          for (int f = 0; f < N; ++f) {
            if constexpr (PPT == 2) node(f, V::from(z[f]));
            else node(f, V::splat(f % 2 ? z[f / 2].y : z[f / 2].x));
          }
        } else if (tr.vr == RG_VR_SOBOL) {
#pragma unroll
          for (int f = 0; f < N; ++f) {
            const uint32_t xs = rg_warp_sobol(tb.sobol + 32 * (size_t)__ldg(tb.nf_row + c * N + f), n1, lane);
            node(f, V::splat(rg_probit32(tr.scrambler == RG_SCRAMBLE_DIGITAL_SHIFT
                                             ? xs ^ __ldg(tb.nf_shift + c * N + f)
                                             : rg_owen(xs, (uint64_t)__ldg(tb.node_k + c) * N + f, tr.seed))));
          }
        } else {
#pragma unroll
          for (int f = 0; f < N; ++f)
            node(f, V::splat(rg_qmc_normal32(tr, tb, path0 + grp * 32 + lane, (uint64_t)__ldg(tb.node_k + c) * N + f)));
        }
      }
      V d[N], y[N];
#pragma unroll
      for (int f = 0; f < N; ++f) {
        d[f] = V::fma(wcur[f], V::splat(-1.0f), top[f]);
        wcur[f] = top[f];
      }
      --sp;
      pop(sp);
      int q = 0;
#pragma unroll
      for (int a = 0; a < N; ++a) {
        y[a] = V::splat(0.0f);
#pragma unroll
        for (int b = 0; b <= a; ++b) y[a] = V::fma(Lf[q++], d[b], y[a]);
      }
#pragma unroll
      for (int f = 0; f < N; ++f) {
        V sg;
        if (LV) {
          // the saturating grid lookup of the tiled kernel: u01 clamped by the FMA's saturation, the
          // grid index from a round-down FMA's bit pattern (its bias folded into lvo), one gather of
          // the cell's line (c, d) and sigma = c + u01·d
          const float4 c4 = PPT == 1 ? s_lv[f] : make_float4(lva[f], lvb[f], __int_as_float(lvo[f]), 0.0f);
          V u01;
#pragma unroll
          for (int j = 0; j < PPT; ++j) u01.v[j] = __saturatef(fmaf(x[f].v[j], c4.y, c4.x));
          const V fl = V::fma_rd(u01, gxm1, two23);
          const float2* row = p32_at(rows, __float_as_int(c4.z));
#pragma unroll
          for (int j = 0; j < PPT; ++j) {
            const float2 r = __ldg(p32_at(row, __float_as_int(fl.v[j])));
            sg.v[j] = fmaf(u01.v[j], r.y, r.x);
          }
        } else {
          sg = sig[f];
        }
        x[f] = V::add(V::fma(sg, V::fma(nhdt, sg, y[f]), x[f]), mu[f]);
      }
      rows += row_step;
      float wmin[PPT];
#pragma unroll
      for (int j = 0; j < PPT; ++j) {
        wmin[j] = x[0].v[j];
        if constexpr (N == 2) wmin[j] = fminf(wmin[j], x[1].v[j]);
        if constexpr (N >= 3) wmin[j] = rg_min3(wmin[j], x[1].v[j], x[2].v[j]);
        if constexpr (N == 4) wmin[j] = fminf(wmin[j], x[3].v[j]);
        if constexpr (N == 5) wmin[j] = rg_min3(wmin[j], x[3].v[j], x[4].v[j]);
      }
      // Phoenix state machine (note.rs:150-218): in full where a coupon period resets or ends; on other
      // steps a path accrues and tests the knock-out branch-free (a dead path's count is not read again)
      const uint32_t fl = __ldg(tb.step_flags + t);
      if (fl & (STEP_PERIOD_RESET | STEP_PERIOD_END)) {
#pragma unroll
        for (int j = 0; j < PPT; ++j)
          if (ph[j].alive)
            p32_phoenix_step<REC>(ph[j], fl, t, wmin[j], ln_cb, ln_ko, tr, tb, tb.df_f,
                                  [&] { return __ldg(tb.step_period + t); });
      } else {
        if (fl & STEP_ACCRUE) {
#pragma unroll
          for (int j = 0; j < PPT; ++j) {
            if (wmin[j] >= ln_cb) ++ph[j].qual;
            if (REC && ph[j].alive && wmin[j] >= ln_cb) ++ph[j].qualified;
          }
        }
        if (fl & STEP_CALL_ACTIVE) {
          bool any = false;
#pragma unroll
          for (int j = 0; j < PPT; ++j) any |= ph[j].alive & (wmin[j] >= ln_ko);
          if (__any_sync(0xffffffffu, any)) {
#pragma unroll
            for (int j = 0; j < PPT; ++j)
              if (ph[j].alive & (wmin[j] >= ln_ko))
                p32_knock_out<REC>(ph[j], fl, t, tr, tb, tb.df_f, __ldg(tb.step_period + t));
          }
        }
      }
    }
    // path close (note.rs:221-258), and per 32 paths the same FP32 butterfly (one chunk) as phoenix32.cu;
    // then lane k writes the chunk's quantity k as FP64 to partial[chunk]
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
      const uint64_t gi = grp * (32 * PPT) + 32 * j + lane;
      float worst = x[0].v[j];
#pragma unroll
      for (int f = 1; f < N; ++f) worst = fminf(worst, x[f].v[j]);
      float out[RG_ACC];
      p32_close_path<REC>(tr, tb, 0, T, gi < npaths, true, path0, gi, ph[j].ko_step, worst, ln_ki, ph[j].cpv,
                          ph[j].mpv, ph[j].received, ph[j].qualified, ph[j].paid, ko_steps, records, out);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < RG_ACC; ++k) out[k] += __shfl_xor_sync(0xffffffffu, out[k], off);
      float mine = 0.0f;
#pragma unroll
      for (int k = 0; k < RG_ACC; ++k) mine = lane == k ? out[k] : mine;
      const uint64_t chunk = grp * PPT + j;
      if (lane < RG_ACC && chunk * 32 < npaths) partial[(size_t)chunk * RG_ACC + lane] = (double)mine;
    }
  }
}

template <int N, int PPT, bool LUT>
static const void* kernel_of(bool lv, bool rec) {
  if (lv) return rec ? reinterpret_cast<const void*>(&phoenix32d_kernel<N, true, true, PPT, LUT>)
                     : reinterpret_cast<const void*>(&phoenix32d_kernel<N, true, false, PPT, LUT>);
  return rec ? reinterpret_cast<const void*>(&phoenix32d_kernel<N, false, true, PPT, LUT>)
             : reinterpret_cast<const void*>(&phoenix32d_kernel<N, false, false, PPT, LUT>);
}
template <int N>
static const void* kernel_ptr(bool lv, bool rec, int ppt, bool lut) {
  return ppt == 2 ? kernel_of<N, 2, true>(lv, rec) : (lut ? kernel_of<N, 1, true>(lv, rec) : kernel_of<N, 1, false>(lv, rec));
}

static const void* select_kernel(int n, bool lv, bool rec, int ppt, bool lut) {
  switch (n) {
    case 1: return kernel_ptr<1>(lv, rec, ppt, lut);
    case 2: return kernel_ptr<2>(lv, rec, ppt, lut);
    case 3: return kernel_ptr<3>(lv, rec, ppt, lut);
    case 4: return kernel_ptr<4>(lv, rec, ppt, lut);
    case 5: return kernel_ptr<5>(lv, rec, ppt, lut);
    default: raise(RG_ERR_INVALID_MARKET_SHAPE, "unsupported asset count");
  }
}

// Paths per thread and grid of the direct kernel: a warp for every path group, up to four waves of
// resident CTAs.
void phoenix32d_shape(const Prepared& P, uint64_t npaths, bool lut, int sm_count, Fp32Shape& sh) {
  // function attributes are process-wide: raise every instantiation's dynamic shared-memory limit
  // to the device maximum once, so concurrent engines never lower it under each other
  {
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(mu);
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    if (!done[dev]) {
      int optin = 0;
      cuda_check(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "smem opt-in");
      for (int ppt = 0; ppt <= 2; ++ppt)  // 0: one path a thread without the tables
        for (int n = 1; n <= RG_NMAX; ++n)
          for (int lv = 0; lv < 2; ++lv)
            for (int rec = 0; rec < 2; ++rec)
              cuda_check(cudaFuncSetAttribute(select_kernel(n, lv != 0, rec != 0, std::max(ppt, 1), ppt != 0),
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, optin),
                         "phoenix32d smem attribute");
      done[dev] = 1;
    }
  }
  const int ppt = p32_direct_ppt(P, npaths, lut);
  sh.direct = 1;
  sh.ppt = ppt;
  sh.threads = P32D_THREADS;
  sh.smem = (int)p32d_smem(P.n, ppt, P.stack_max);
  int per_sm = 0;
  cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                 &per_sm, select_kernel(P.n, P.trade.has_lv != 0, false, ppt, lut), P32D_THREADS, sh.smem),
             "phoenix32d occupancy");
  if (per_sm < 1 || p32d_slow(ppt, P.stack_max) > kSlowSlots) raise(RG_ERR_GPU_ERROR, "phoenix32d: launch shape does not fit on an SM");
  const uint64_t warps = (npaths + 32 * ppt - 1) / (32 * ppt);
  const uint64_t ctas = (warps + P32D_WARPS - 1) / P32D_WARPS, cap = (uint64_t)sm_count * per_sm * 4;
  sh.grid = (int)std::max<uint64_t>(std::min(ctas, cap), 1);
}

void launch_phoenix32d(const Prepared& P, const DevTables& tb, const DevScen32* scen32, uint64_t path0,
                       uint64_t npaths, const Fp32Shape& sh, const LaunchOut& out, cudaStream_t st) {
  const bool lut = P.trade.vr == RG_VR_SOBOL && tb.sob_lut && (int32_t)((path0 + 1) & 31) == tb.sob_lut_o;
  const void* k = select_kernel(P.n, P.trade.has_lv != 0, out.records != nullptr, sh.ppt, lut);
  if (P.n_scen != 1 || (sh.ppt == 2 && !lut) || sh.threads != P32D_THREADS ||
      sh.smem < (int)p32d_smem(P.n, sh.ppt, P.stack_max))
    raise(RG_ERR_GPU_ERROR, "phoenix32d: invalid launch shape");
  DevTrade tr = P.trade;
  DevTables tables = tb;
  int stack_max = P.stack_max, n_surf = P.n_surf;
  float ln_ko = (float)P.ln_ko, ln_cb = (float)P.ln_cb, ln_ki = (float)P.ln_ki;
  double* partial = out.partial;
  int32_t* ko_steps = out.ko_steps;
  rg_path_record* records = out.records;
  void* args[] = {&tr, &tables, &scen32, &stack_max, &n_surf, &ln_ko, &ln_cb, &ln_ki, &path0, &npaths, &partial, &ko_steps, &records};
  cuda_check(cudaLaunchKernel(k, dim3(sh.grid), dim3(sh.threads), args, sh.smem, st), "phoenix32d_kernel launch");
}

}  // namespace rg
