// path64.cu — the FP64 parity kernels of an engine: normals, then stepping and payoff.
//
// The reference's arithmetic (crates/riga-engine/src/note.rs:81-259) in its own operation order,
// product by product, as phoenix64.cu performs it in one kernel; here the work is split where its
// shape changes, through a buffer of a chunk of paths and, where schedules are long, a window of steps:
//   * normals64_kernel — correlated normals y = L·z of every bridge node, y[node][asset][path].  A
//     CTA forms the normals of 256 paths × a few nodes; the 5% that fall into the inverse normal's
//     tails (a logarithm, a square root and a division) are queued in shared memory and taken 32 at
//     a time, where a warp of one path a lane would enter the tail for 54% of its normals on either
//     side.  correlate64_kernel does the same from the pseudo-random lane's stream.
//   * step64_kernel — a lane per (path, asset): the streamed bridge, the GBM / Dupire step, and the
//     Phoenix state machine replicated over a path's lanes, which agree on the barriers by a vote.
//     Barriers compare spots against the smallest spot whose ratio reaches the barrier (found on the
//     host by rounding the ratio both ways), so no division and no FP64 comparison runs per step,
//     and a period's accruals are counted and looked up.
// What bounds it: the FP64 pipe (rg_fp64.cuh): per (path, step, asset) about 37 operations in the
// normals, 34 in a flat step and 88 in a local-vol one; and, below about four warps an SM, the
// latency of a step's dependent operations, which a lane per asset halves or better.
// Measured: 3 assets flat, 2^16 paths × 756 steps 21.9 ms (normals 10.2, stepping 11.6, the FP64 pipe 83%
// busy in both) against 77.2 ms in one kernel; 2 assets local vol, 30,000 paths × 501 steps of the
// pseudo-random lane 6.3 against 11.1 ms; a replay of 4096 Owen-scrambled paths 2.4 against 13.8 ms.
// Compiled with -fmad=false: products and sums round separately, as in the reference.
#include <algorithm>

#include "rg_fp64.cuh"
#include "rg_internal.h"

namespace rg {

namespace {

constexpr int kNormPaths = 256;                                            // paths (threads) per CTA
__host__ __device__ constexpr int norm_nodes(int n) { return n <= 3 ? 4 : 2; }  // nodes per CTA

template <int N>
__global__ void __launch_bounds__(kNormPaths) normals64_kernel(DevTrade tr, DevTables tb,
                                                               const DevScenario* __restrict__ scen, uint64_t path0,
                                                               uint64_t npaths, uint64_t stride, int path_blocks,
                                                               int node0, int node1, double* __restrict__ y) {
  constexpr int KN = norm_nodes(N);
  __shared__ double zs[KN * N][kNormPaths];
  __shared__ uint16_t queue[KN * N * kNormPaths];
  __shared__ int queued;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t p = (uint64_t)(blockIdx.x % path_blocks) * kNormPaths + tid;
  const int c0 = node0 + (int)(blockIdx.x / path_blocks) * KN, nn = min(KN, node1 - c0);
  if (tid == 0) queued = 0;
  __syncthreads();
  if (tr.vr == RG_VR_SOBOL) {
    const uint64_t n1 = path0 + p - lane + 1;  // Sobol point of the warp's first path
#pragma unroll
    for (int j = 0; j < KN * N; ++j) {
      if (j >= nn * N) break;
      const int i = c0 * N + j;
      const uint32_t g = rg_warp_sobol(tb.sobol + 32 * (size_t)__ldg(tb.nf_row + i), n1, lane);
      const uint32_t x = tr.scrambler == RG_SCRAMBLE_DIGITAL_SHIFT
                             ? g ^ __ldg(tb.nf_shift + i)
                             : rg_owen(g, (uint64_t)__ldg(tb.node_k + c0 + j / N) * N + j % N, tr.seed);
      if (probit64_is_tail(x)) {
        zs[j][tid] = __longlong_as_double((long long)x);
        queue[atomicAdd(&queued, 1)] = (uint16_t)(j * kNormPaths + tid);
      } else {
        zs[j][tid] = probit64_central(x);
      }
    }
    __syncthreads();
    for (int q = tid; q < queued; q += kNormPaths) {
      double& z = (&zs[0][0])[queue[q]];
      z = probit64_tail((uint32_t)__double_as_longlong(z));
    }
    __syncthreads();
  } else {
    for (int j = 0; j < nn * N; ++j)
      zs[j][tid] = rg_qmc_normal64(tr, tb, path0 + p, (uint64_t)__ldg(tb.node_k + c0 + j / N) * N + j % N);
  }
  if (p >= npaths) return;
  const DevScenario& sc = scen[0];
  for (int j = 0; j < nn; ++j) {
    // Cholesky::apply_into (correlation.rs:196-206)
    double z[N];
#pragma unroll
    for (int f = 0; f < N; ++f) z[f] = zs[j * N + f][tid];
#pragma unroll
    for (int a = 0; a < N; ++a) {
      double s = sc.L[a * N] * z[0];
#pragma unroll
      for (int b = 1; b <= a; ++b) s += sc.L[a * N + b] * z[b];
      y[((uint64_t)(c0 - node0 + j) * N + a) * stride + p] = s;
    }
  }
}

// The pseudo-random lane (note.rs:123-127): y = L·z of the stream's draws z[path][step][asset], read
// along a path's row and written along paths.
constexpr int kCorPaths = 32, kCorSteps = 16;
template <int N>
__global__ void __launch_bounds__(kCorPaths * 8) correlate64_kernel(const DevScenario* __restrict__ scen,
                                                                   const double* __restrict__ z, int64_t T,
                                                                   uint64_t npaths, uint64_t stride, int path_blocks,
                                                                   int64_t step0, int64_t step1, double* __restrict__ y) {
  __shared__ double zs[kCorPaths][kCorSteps * N + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t p0 = (uint64_t)(blockIdx.x % path_blocks) * kCorPaths;
  const int64_t t0 = step0 + (int64_t)(blockIdx.x / path_blocks) * kCorSteps;
  const int nt = (int)min((int64_t)kCorSteps, step1 - t0);
  for (int r = warp; r < kCorPaths; r += 8)
    if (p0 + r < npaths)
      for (int i = lane; i < nt * N; i += 32) zs[r][i] = z[((p0 + r) * (uint64_t)T + t0) * N + i];
  __syncthreads();
  const uint64_t p = p0 + lane;
  if (p >= npaths) return;
  const DevScenario& sc = scen[0];
  for (int j = warp; j < nt; j += 8)
#pragma unroll
    for (int a = 0; a < N; ++a) {
      double s = sc.L[a * N] * zs[lane][j * N];
#pragma unroll
      for (int b = 1; b <= a; ++b) s += sc.L[a * N + b] * zs[lane][j * N + b];
      y[((uint64_t)(t0 - step0 + j) * N + a) * stride + p] = s;
    }
}

// Per surface, the widths of the log-strike axis's cells and their reciprocals (rounded).
__global__ void axis64_kernel(const double* __restrict__ logs, int gx, int n, double2* __restrict__ axis) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double d = i % gx + 1 < gx ? logs[i + 1] - logs[i] : 1.0;
  axis[i] = make_double2(d, 1.0 / d);
}

// DupireLocalVol::sigma (riga-market/src/lib.rs:305-343) at a step's tenor rows.
__device__ __forceinline__ double sigma64(const double* __restrict__ v, const double* __restrict__ ls,
                                          const double2* __restrict__ axis, int gx, float l0, float inv, int2 ti,
                                          double wt, double spot) {
  // max(spot, 1e-12); the logarithm's fast form takes positive normals
  const uint32_t h = (uint32_t)hi_word(spot);
  const double x = h - 0x3d719800u < 0x7ff00000u - 0x3d719800u ? fast_log64(spot) : general_log64(spot > 1e-12 ? spot : 1e-12);
  const long long kx = order_key(x);
  int lo, hi;
  double wx = 0.0;
  if (kx <= order_key(__ldg(ls))) {
    lo = hi = 0;
  } else if (!(kx < order_key(__ldg(ls + gx - 1)))) {
    lo = hi = gx - 1;
  } else {
    // first j with x <= ls[j+1], from an estimate on the uniform axis
    int j = (int)(((float)x - l0) * inv);
    j = j < 0 ? 0 : (j > gx - 2 ? gx - 2 : j);
    while (j > 0 && kx <= order_key(__ldg(ls + j))) --j;
    while (j + 1 < gx - 1 && kx > order_key(__ldg(ls + j + 1))) ++j;
    lo = j;
    hi = j + 1;
    const double2 a = __ldg(axis + j);
    wx = divide_by(x - __ldg(ls + j), a.x, a.y);
  }
  const double ox = 1.0 - wx;
  const double v0 = ox * __ldg(v + ti.x * gx + lo) + wx * __ldg(v + ti.x * gx + hi);
  const double v1 = ox * __ldg(v + ti.y * gx + lo) + wx * __ldg(v + ti.y * gx + hi);
  return (1.0 - wt) * v0 + wt * v1;
}

constexpr int kStepWarps = 2;
constexpr int kCtaThreads = 32 * kStepWarps;
// Words of a lane's state between two windows of steps, beside its bridge stack.
constexpr int kStateWords = 7;

struct Step64Args {
  DevTrade tr;
  DevTables tb;
  const DevScenario* scen;
  const double* y;      // [node or step of the window][asset][stride]
  const double2* axis;  // [surface][gx]
  uint64_t stride, path0, first, npaths;  // global index of path 0; the chunk's first path; its paths
  int64_t t0, t1;       // the window's steps
  int node0, node1;     // and the bridge nodes they consume
  double* state;        // [word][thread of the chunk] between windows (unused when one covers all steps)
  uint64_t state_row;
  double* partial;      // row of the chunk's first CTA
  int32_t* ko_steps;
  rg_path_record* records;
  float* cube;
};

template <int N, bool LV, bool MC>
__global__ void __launch_bounds__(kCtaThreads) step64_kernel(const __grid_constant__ Step64Args A) {
  constexpr int G = 32 / N;  // paths per warp, a lane per asset
  extern __shared__ double stk_mem[];  // [depth][thread] bridge anchors
  __shared__ double red[kStepWarps * G][RG_ACC];
  const DevTrade& tr = A.tr;
  const DevTables& tb = A.tb;
  const DevScenario& sc = A.scen[0];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = min(lane / N, G - 1), f = lane < G * N ? lane % N : 0;
  const uint32_t mates = ((1u << N) - 1u) << (g * N);  // this path's lanes
  const int slot = warp * G + g;                      // path within the CTA
  const uint64_t p = (uint64_t)blockIdx.x * (kStepWarps * G) + slot;
  const bool live = lane < G * N && p < A.npaths;
  const uint64_t pl = min(p, A.npaths - 1);  // idle lanes follow the last path
  const int64_t T = tr.steps;
  const double init = tr.init[f], dt = tr.dt, sqrt_dt = tr.sqrt_dt, inv_sqrt_dt = tr.inv_sqrt_dt;
  const double rq = sc.rate - sc.q[f], vol = sc.vols[f];
  const double flat_drift = (rq - 0.5 * vol * vol) * dt, flat_vs = vol * sqrt_dt;
  const long long cb_at = __double_as_longlong(tr.cb_spot[f]), ko_at = __double_as_longlong(tr.ko_spot[f]);
  const double* v = LV ? tb.lv_v + sc.surf_off[f] : nullptr;
  const double* ls = LV ? tb.lv_logs + sc.surf[f] * tr.gx : nullptr;
  const double2* axis = LV ? A.axis + sc.surf[f] * tr.gx : nullptr;
  float l0 = 0.0f, inv = 0.0f;
  if (LV) {
    l0 = (float)ls[0];
    inv = (float)(tr.gx - 1) / (float)(ls[tr.gx - 1] - ls[0]);
  }
  const int2* ti = tb.lv_ti + f * T;
  const double* tw = tb.lv_tw + f * T;
  const double* yp = A.y + f * A.stride + pl;  // this lane's value of node c at yp[c·N·stride]
  const uint64_t ystep = (uint64_t)N * A.stride;
  float* cube = A.cube ? A.cube + (A.first + pl) * (uint64_t)T * N + f : nullptr;
  double* stk = stk_mem + tid;
  double spot = sc.spots[f], wcur = 0.0, top = 0.0;
  int sp = 0, c = A.node0;
  int qual = 0, ko_step = -1, qualified = 0, paid = 0;
  bool ko = false, received = false;
  double unpaid = 0.0, cpv = 0.0, mpv = 0.0;
  double* const state = A.state + (uint64_t)blockIdx.x * kCtaThreads + tid;
  if (A.t0 > 0) {  // what the window before left
    spot = state[0];
    wcur = state[A.state_row];
    unpaid = state[2 * A.state_row];
    cpv = state[3 * A.state_row];
    mpv = state[4 * A.state_row];
    qual = __double2loint(state[5 * A.state_row]);
    ko_step = __double2hiint(state[5 * A.state_row]);
    qualified = __double2loint(state[6 * A.state_row]);
    paid = __double2hiint(state[6 * A.state_row]);
    ko = ko_step >= 0;
    received = paid > 0;
    if (!MC) {
      sp = A.node0 - (int)A.t0;
      for (int i = 0; i < sp; ++i) stk[i * kCtaThreads] = state[(kStateWords + i) * A.state_row];
      if (sp > 0) top = stk[(sp - 1) * kCtaThreads];
    }
  }
  double ynext = __ldg(yp);
  for (int64_t t = A.t0; t < A.t1; ++t) {
    double shock;
    if (MC) {
      shock = ynext;
      if (t + 1 < A.t1) ynext = __ldg(yp + (uint64_t)(t + 1 - A.t0) * ystep);
    } else {
      // bridge nodes consumed at this step (note.rs:89-105 and qmc.rs:158-191)
      const int c1 = __ldg(tb.node_off + t + 1);
      for (; c < c1; ++c) {
        const double yc = ynext * __ldg(tb.node_c + c);
        if (c + 1 < A.node1) ynext = __ldg(yp + (uint64_t)(c + 1 - A.node0) * ystep);
        top = c == 0 ? yc : halve(wcur + top) + yc;
        stk[sp * kCtaThreads] = top;
        ++sp;
      }
      --sp;
      shock = (top - wcur) * inv_sqrt_dt;
      wcur = top;
      if (sp > 0) top = stk[(sp - 1) * kCtaThreads];
    }
    // GBM / Dupire step (note.rs:133-142)
    if (LV) {
      const double s = sigma64(v, ls, axis, tr.gx, l0, inv, __ldg(ti + t), __ldg(tw + t), spot);
      spot *= fast_exp64((rq - halve(s) * s) * dt + s * sqrt_dt * shock);
    } else {
      spot *= fast_exp64(flat_drift + flat_vs * shock);
    }
    if (cube && live) cube[(uint64_t)t * N] = (float)spot;
    // Phoenix state machine (note.rs:150-218)
    const uint32_t fl = __ldg(tb.step_flags + t);
    const long long sb = __double_as_longlong(spot);
    bool above, up;
    if (__any_sync(0xffffffffu, (uint32_t)(sb >> 32) >= 0x7ff00000u)) {
      // an infinite or NaN spot in the warp: the ratios as they are
      const double ratio = spot / init;
      double worst = __shfl_sync(0xffffffffu, ratio, g * N);
#pragma unroll
      for (int a = 1; a < N; ++a) worst = fmin(worst, __shfl_sync(0xffffffffu, ratio, g * N + a));
      above = worst >= tr.coupon_barrier;
      up = (__ballot_sync(0xffffffffu, ratio >= tr.call_barrier) & mates) == mates;
    } else {
      above = (__ballot_sync(0xffffffffu, sb >= cb_at) & mates) == mates;
      up = (__ballot_sync(0xffffffffu, sb >= ko_at) & mates) == mates;
    }
    if (ko) continue;
    if (fl & STEP_PERIOD_RESET) qual = 0;
    if ((fl & STEP_ACCRUE) && above) {
      ++qual;
      ++qualified;
    }
    auto due_now = [&] {
      return (fl & STEP_FIXED_DUE) ? tr.coupon_rate : __ldg(tb.accr_sum + __ldg(tb.accr_at + __ldg(tb.step_period + t)) + qual);
    };
    if ((fl & STEP_CALL_ACTIVE) && up) {
      ko = true;
      ko_step = (int)t;
      const double due = due_now();
      const double carry = due > 0.0 ? unpaid : 0.0;
      if (due + carry > 0.0) {
        const double df = __ldg(tb.df + t);
        cpv += due * df;
        mpv += carry * df;
        received = true;
        ++paid;
      }
      continue;
    }
    if (fl & STEP_PERIOD_END) {
      const double due = due_now();
      if (due > 0.0) {
        const double df = __ldg(tb.df + t);
        cpv += due * df;
        mpv += unpaid * df;
        received = true;
        unpaid = 0.0;
        ++paid;
      } else if (tr.memory) {
        unpaid += tr.coupon_rate;
      }
    }
  }
  if (A.t1 < T) {
    state[0] = spot;
    state[A.state_row] = wcur;
    state[2 * A.state_row] = unpaid;
    state[3 * A.state_row] = cpv;
    state[4 * A.state_row] = mpv;
    state[5 * A.state_row] = __hiloint2double(ko_step, qual);
    state[6 * A.state_row] = __hiloint2double(paid, qualified);
    if (!MC)
      for (int i = 0; i < sp; ++i) state[(kStateWords + i) * A.state_row] = stk[i * kCtaThreads];
    return;
  }
  // path close (note.rs:221-258) on the path's first lane
  const double ratio = spot / init;
  double worst = __shfl_sync(0xffffffffu, ratio, g * N);
#pragma unroll
  for (int a = 1; a < N; ++a) worst = fmin(worst, __shfl_sync(0xffffffffu, ratio, g * N + a));
  if (lane < G * N && f == 0) {
    double out[RG_ACC];
#pragma unroll
    for (int k = 0; k < RG_ACC; ++k) out[k] = 0.0;
    if (live) {
      const double dfm = __ldg(tb.df_mat);
      const double funding = ko ? __ldg(tb.df + ko_step) : dfm;
      const bool hit_ki = worst <= tr.ki, put_ok = hit_ki && !ko;
      const double put = put_ok ? fmax(tr.strike - worst, 0.0) * dfm : 0.0;
      const double cn = cpv + mpv;
      const double pv = funding + cn - put;
      out[ACC_PV] = pv - 1.0;
      out[ACC_PV2] = (pv - 1.0) * (pv - 1.0);
      if (ko) {
        out[ACC_KOF] = funding - 1.0;
        out[ACC_KOF2] = (funding - 1.0) * (funding - 1.0);
        out[ACC_NKO] = 1.0;
      }
      if (hit_ki) {
        out[ACC_KIPUT] = put;
        out[ACC_KIPUT2] = put * put;
        out[ACC_NKI] = 1.0;
      }
      if (received) {
        out[ACC_CPN] = cn;
        out[ACC_CPN2] = cn * cn;
        out[ACC_NCPN] = 1.0;
      }
      out[ACC_PUT] = put;
      out[ACC_FUND] = funding;
      out[ACC_CQ] = cn * 10.0 - mpv * 10.0;
      out[ACC_MQ] = mpv * 10.0;
      out[ACC_NPUT] = put_ok ? 1.0 : 0.0;
      const uint64_t i = A.first + p;
      if (A.ko_steps) A.ko_steps[i] = ko_step;
      if (A.records) {
        rg_path_record r;
        r.path_id = A.path0 + i;
        r.rng_seed = tr.seed;
        r.sobol_index = MC ? 0 : A.path0 + i + 1;
        r.worst_final = worst;
        r.knocked_out = ko;
        r.ko_step = ko_step;
        r.ko_time = ko ? (double)(ko_step + 1) * dt : __longlong_as_double(0x7ff8000000000000LL);
        r.ki_hit = hit_ki;
        r.qualified_steps = qualified;
        r.paid_periods = paid;
        r.put_payoff = put;
        r.coupon_pv = cn;
        r.memory_coupon_pv = mpv;
        r.funding = funding;
        r.pv = pv;
        A.records[i] = r;
      }
    }
#pragma unroll
    for (int k = 0; k < RG_ACC; ++k) red[slot][k] = out[k];
  }
  __syncthreads();
  if (tid < RG_ACC) {
    double s = 0.0;
    for (int i = 0; i < kStepWarps * G; ++i) s += red[i][tid];
    A.partial[(size_t)blockIdx.x * RG_ACC + tid] = s;
  }
}

// Paths of one step64 CTA.
uint64_t cta_paths(int n) { return (uint64_t)kStepWarps * (32 / n); }

// Deepest bridge stack of T steps.
int stack_bound(int64_t T) {
  int bits = 0;
  while (T >> bits) ++bits;
  return std::min(bits + 1, RG_STACK_MAX);
}

// How a launch passes through the buffer: `chunk` paths (whole CTAs) at a time, `window` steps at a time.
struct Path64Plan {
  uint64_t chunk;
  int64_t window;
  size_t y_bytes, state_bytes, axis_bytes;
  size_t bytes() const { return axis_bytes + state_bytes + y_bytes; }
};
// Whole schedules of all paths where `limit` bytes hold them, else of chunks of about equal path counts
// as long as a chunk has kFillCtas CTAs.  Long schedules, whose chunks would leave SMs without work, pass
// all paths (up to twice that many CTAs) through windows of steps instead, the state of each path carried
// from one to the next; a limit too small for windows of kMinWindow steps takes fewer paths.
// Measured, 3 assets flat, 2^16 paths, a GiB, chunks against windows: 2000 steps (chunks of 1,093 CTAs)
// 58.9 and 57.4 ms, 5000 (437) 158 and 143, 15,000 (149) 742 and 430, 50,000 (44) 6,839 and 1,434, where
// one kernel took 5,096; 1000 paths x 200,000 steps 1,638 and 362.
constexpr uint64_t kFillCtas = 152 * 8;
constexpr int64_t kMinWindow = 16;
Path64Plan path64_plan(int n, int64_t T, uint64_t npaths, size_t axis_bytes, size_t limit) {
  limit -= std::min(limit, axis_bytes);
  const uint64_t unit = cta_paths(n), ctas = (npaths + unit - 1) / unit;
  const uint64_t row = unit * n * sizeof(double);  // a CTA's normals of one node
  const uint64_t fit = limit / (row * (uint64_t)T);
  auto even = [&](uint64_t cap) {
    const uint64_t chunks = (ctas + cap - 1) / cap;
    return (ctas + chunks - 1) / chunks;
  };
  if (fit >= std::min(ctas, kFillCtas)) {
    const uint64_t per = even(fit);
    return {per * unit, T, (size_t)(per * row * (uint64_t)T), 0, axis_bytes};
  }
  const uint64_t depth = (uint64_t)stack_bound(T), state = (kStateWords + depth) * kCtaThreads * sizeof(double);
  const uint64_t shortest = std::min<uint64_t>(kMinWindow, (uint64_t)T);
  const uint64_t per = even(std::max<uint64_t>(std::min(2 * kFillCtas, limit / (state + row * (shortest + depth))), 1));
  // a window's steps consume at most `depth` nodes more than it has steps
  const uint64_t nodes = per * state < limit ? (limit - per * state) / (per * row) : 0;
  const uint64_t window = std::min<uint64_t>(std::max<uint64_t>(nodes, depth + 1) - depth, (uint64_t)T);
  return {per * unit, (int64_t)window, (size_t)(per * row * (window + depth)), (size_t)(per * state), axis_bytes};
}

template <int N>
Path64Launch run(Workspace& W, const Prepared& P, const DevTables& tb, const DevScenario* scen, uint64_t path0,
                 uint64_t npaths, const LaunchOut& out, cudaStream_t st) {
  const int64_t T = P.T;
  const bool lv = P.trade.has_lv != 0;
  const size_t axis_bytes = lv ? (size_t)P.n_surf * P.trade.gx * sizeof(double2) : 0;
  const Path64Plan plan = path64_plan(N, T, npaths, axis_bytes, W.limits.normals64);
  const uint64_t chunk = plan.chunk, unit = cta_paths(N);
  if (P.stack_max > stack_bound(T)) raise(RG_ERR_INVALID_SCHEDULE, "path64: the bridge stack is too deep");
  uint8_t* buf = static_cast<uint8_t*>(W.device(WS_NORMALS64, plan.bytes()));
  double* state = reinterpret_cast<double*>(buf + axis_bytes);
  double* y = reinterpret_cast<double*>(buf + axis_bytes + plan.state_bytes);
  Step64Args a{P.trade, tb, scen, y, reinterpret_cast<const double2*>(buf), chunk, path0, 0, 0, 0, 0, 0, 0, state,
               chunk / unit * kCtaThreads, out.partial, out.ko_steps, out.records, out.cube};
  if (lv) {
    const int n = P.n_surf * P.trade.gx;
    axis64_kernel<<<(n + 127) / 128, 128, 0, st>>>(tb.lv_logs, P.trade.gx, n, reinterpret_cast<double2*>(buf));
    cuda_check(cudaGetLastError(), "axis64_kernel launch");
  }
  Path64Launch done{lv ? 1 : 0, 0, kCtaThreads, 0};
  const size_t smem = out.mcz ? 0 : (size_t)P.stack_max * kCtaThreads * sizeof(double);
  for (a.first = 0; a.first < npaths; a.first += chunk) {
    a.npaths = std::min(chunk, npaths - a.first);
    const unsigned blocks = (unsigned)((a.npaths + unit - 1) / unit);
    for (a.t0 = 0; a.t0 < T; a.t0 = a.t1) {
      a.t1 = std::min(a.t0 + plan.window, T);
      a.node0 = P.node_off[a.t0];
      a.node1 = P.node_off[a.t1];
      if (out.mcz) {
        const int pb = (int)((a.npaths + kCorPaths - 1) / kCorPaths);
        const int64_t tiles = (a.t1 - a.t0 + kCorSteps - 1) / kCorSteps;
        correlate64_kernel<N><<<(unsigned)(pb * tiles), kCorPaths * 8, 0, st>>>(
            scen, out.mcz + a.first * (uint64_t)T * N, T, a.npaths, chunk, pb, a.t0, a.t1, y);
      } else if (a.node1 > a.node0) {
        const int pb = (int)((a.npaths + kNormPaths - 1) / kNormPaths);
        const int64_t tiles = (a.node1 - a.node0 + norm_nodes(N) - 1) / norm_nodes(N);
        normals64_kernel<N><<<(unsigned)(pb * tiles), kNormPaths, 0, st>>>(P.trade, tb, scen, path0 + a.first, a.npaths,
                                                                           chunk, pb, a.node0, a.node1, y);
      }
      done.kernels += out.mcz || a.node1 > a.node0 ? 2 : 1;
      if (done.grid == 0) {
        done.grid = (int)blocks;
        done.smem = (int)smem;
      }
      cuda_check(cudaGetLastError(), "normals64 launch");
      if (lv) {
        if (out.mcz) step64_kernel<N, true, true><<<blocks, kCtaThreads, smem, st>>>(a);
        else step64_kernel<N, true, false><<<blocks, kCtaThreads, smem, st>>>(a);
      } else {
        if (out.mcz) step64_kernel<N, false, true><<<blocks, kCtaThreads, smem, st>>>(a);
        else step64_kernel<N, false, false><<<blocks, kCtaThreads, smem, st>>>(a);
      }
      cuda_check(cudaGetLastError(), "step64_kernel launch");
    }
    a.partial += (size_t)blocks * RG_ACC;
  }
  return done;
}

}  // namespace

uint64_t path64_rows(int n, uint64_t npaths) { return (npaths + cta_paths(n) - 1) / cta_paths(n); }

size_t path64_bytes(int n, int64_t T, uint64_t npaths, size_t axis_bytes, size_t limit) {
  return path64_plan(n, T, npaths, axis_bytes, limit).bytes();
}

Path64Launch launch_path64(Workspace& W, const Prepared& P, const DevTables& tb, const DevScenario* scen,
                           uint64_t path0, uint64_t npaths, const LaunchOut& out, cudaStream_t st) {
  switch (P.n) {
    case 1: return run<1>(W, P, tb, scen, path0, npaths, out, st);
    case 2: return run<2>(W, P, tb, scen, path0, npaths, out, st);
    case 3: return run<3>(W, P, tb, scen, path0, npaths, out, st);
    case 4: return run<4>(W, P, tb, scen, path0, npaths, out, st);
    case 5: return run<5>(W, P, tb, scen, path0, npaths, out, st);
    default: raise(RG_ERR_INVALID_MARKET_SHAPE, "unsupported asset count");
  }
}

}  // namespace rg
