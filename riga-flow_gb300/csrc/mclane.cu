// mclane.cu — the reference's pseudo-random lane on the device: ChaCha8Rng::seed_from_u64(seed)
// feeding rand_distr's StandardNormal (rand_chacha 0.9.0, rand_core 0.9.5, rand_distr 0.5.1; the
// reference draws it in crates/riga-engine/src/note.rs:58,123-127 and pathcube.rs:37-66).
//
// The stream is sequential: a normal consumes one 64-bit word, or more when the ziggurat rejects,
// so where the k-th normal starts depends on every earlier draw.  The device reproduces it exactly
// by a parallel parse.  A draw that starts at a word is a function of the words from there on, and
// 98.8% of words are accepted as they stand, so only the others ("slow" words, about 25 per 2048)
// decide where draws start:
//   1. keystream — ChaCha8 is counter-based: one thread per 64-byte block writes its 8 words
//      (next_u64 = low word | high word << 32 of consecutive output words);
//   2. transfer — a CTA per segment of 2048 words finds its slow words with an integer test (below),
//      one thread each runs a slow word's draw to its length, and the 32 lanes of a warp walk the
//      slow words in order, lane e for the entry offset e (where the previous segment's last normal
//      may end): the exit offset and the number of draws for every entry;
//   3. chain — a CTA composes the maps of 128 consecutive segments (lane = entry, two shuffles per
//      segment, 4 segments a warp, then the 32 warps' maps), one CTA chains the groups' maps from
//      word 0, and each group walks its segments again from the entry that gives: every segment's
//      entry and first draw index;
//   4. emit — a CTA per segment marks its draws' start words, ranks them by popcounts and writes the
//      normals whose global index falls in the requested range, consecutive lanes to consecutive
//      normals.
// What bounds it: passes over the words (8 bytes each, read in 2 and 4, written in 1) and the FP64
// pipe, which the product of an emitted normal needs once per word.  The accepted words' test
// |u·x_i| < x_{i+1} runs on integers: the product is monotone in |u| = |2m - 2^52| / 2^52, so it is
// |2m - 2^52| < T_i with T_i found on the host by bisection over the rounded products.
// Measured on 30,000 paths x 501 steps x 2 factors (30 M normals): 0.56 ms —
// keystream 0.12, transfer 0.12, chain 0.02, emit 0.30 — against 34.4 ms when one thread per
// (segment, entry) ran every draw of the segment and one thread chained the segments.
// The ziggurat is Doornik's ZIGNOR with 256 layers (R = 3.6541528853610088, V = 0.00492867323399);
// its tables are regenerated from that recurrence and rounded to the 18 decimals of the crate's
// table literals.  Compiled with -fmad=false so every product and sum rounds as on the host; the
// wedge test's exp and the tail's log are CUDA's (an accept/reject decision could differ from the
// host's libm only for a value within an ulp of the threshold).
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "rg_internal.h"

namespace rg {

namespace {

constexpr double kZigR = 3.6541528853610088;
constexpr int kSegWords = 2048;  // B
constexpr int kEntries = 32;     // E: a normal spans at most E words past a segment end
constexpr int kTailIters = 64;   // tail-loop bound (each pass succeeds with probability > 0.9)

constexpr int kGroupSegs = 128;  // segments one CTA composes, four a warp
constexpr int kSegThreads = 256;

struct ZigTables {
  double x[257], f[257];
  uint64_t accept[256];  // T_i: the word's draw is its first product iff |2m - 2^52| < T_i
};

double round18(double v) {
  char b[64];
  snprintf(b, sizeof b, "%.18f", v);
  return strtod(b, nullptr);
}

const ZigTables& zig_tables() {
  static ZigTables t;
  static std::once_flag once;
  std::call_once(once, [] {
    const double r = kZigR, v = 0.00492867323399;
    double x[257];
    x[0] = v / std::exp(-r * r / 2.0);
    x[1] = r;
    for (int i = 2; i < 256; ++i) {
      const double last = x[i - 1];
      x[i] = std::sqrt(-2.0 * std::log(v / last + std::exp(-last * last / 2.0)));
    }
    x[256] = 0.0;
    for (int i = 0; i < 257; ++i) {
      t.x[i] = round18(x[i]);
      t.f[i] = round18(std::exp(-x[i] * x[i] / 2.0));
    }
    for (int i = 0; i < 256; ++i) {
      // the smallest d in [0, 2^52] with (d / 2^52)·x_i >= x_{i+1} as FP64 rounds the product
      uint64_t lo = 0, hi = (uint64_t(1) << 52) + 1;
      while (lo < hi) {
        const uint64_t mid = (lo + hi) / 2;
        if (std::ldexp((double)mid, -52) * t.x[i] < t.x[i + 1]) lo = mid + 1;
        else hi = mid;
      }
      t.accept[i] = lo;
    }
  });
  return t;
}

struct ChaKey {
  uint32_t k[8];
};

// seed_from_u64: eight PCG32 (XSH-RR) outputs of the seed state (rand_core 0.9.5).
ChaKey chacha_key(uint64_t state) {
  ChaKey key;
  for (int i = 0; i < 8; ++i) {
    state = state * 6364136223846793005ULL + 11634580027462260723ULL;
    const uint32_t xs = (uint32_t)(((state >> 18) ^ state) >> 27);
    const uint32_t rot = (uint32_t)(state >> 59);
    key.k[i] = (xs >> rot) | (xs << ((32 - rot) & 31));
  }
  return key;
}

__device__ __forceinline__ uint32_t rotl(uint32_t v, int c) { return (v << c) | (v >> (32 - c)); }

#define RG_QR(a, b, c, d)               \
  x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 16); \
  x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 12); \
  x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 8);  \
  x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 7);

// ChaCha with 8 rounds, 64-bit block counter in words 12-13, stream 0 in words 14-15.
__global__ void chacha8_stream_kernel(ChaKey key, uint64_t nblocks, uint64_t* __restrict__ out) {
  const uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nblocks) return;
  uint32_t s[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u};
#pragma unroll
  for (int i = 0; i < 8; ++i) s[4 + i] = key.k[i];
  s[12] = (uint32_t)b;
  s[13] = (uint32_t)(b >> 32);
  s[14] = 0;
  s[15] = 0;
  uint32_t x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = s[i];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    RG_QR(0, 4, 8, 12) RG_QR(1, 5, 9, 13) RG_QR(2, 6, 10, 14) RG_QR(3, 7, 11, 15)
    RG_QR(0, 5, 10, 15) RG_QR(1, 6, 11, 12) RG_QR(2, 7, 8, 13) RG_QR(3, 4, 9, 14)
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    out[b * 8 + i] = (uint64_t)(x[2 * i] + s[2 * i]) | ((uint64_t)(x[2 * i + 1] + s[2 * i + 1]) << 32);
}
#undef RG_QR

__device__ __forceinline__ double from_bits(uint64_t frac52, int e) {
  return __longlong_as_double((long long)(frac52 | ((uint64_t)(1023 + e) << 52)));
}

// One StandardNormal draw starting at word `pos`: returns the words consumed (0 if the stream or
// the tail-loop bound ran out) and the value.
__device__ int zig_draw(const uint64_t* __restrict__ U, uint64_t pos, uint64_t limit,
                        const double* __restrict__ zx, const double* __restrict__ zf, double* value) {
  uint64_t p = pos;
  for (int attempt = 0; attempt < kTailIters; ++attempt) {
    if (p >= limit) return 0;
    const uint64_t bits = U[p++];
    const int i = (int)(bits & 0xff);
    const double u = from_bits(bits >> 12, 1) - 3.0;
    const double x = u * zx[i];
    if (fabs(x) < zx[i + 1]) {
      *value = x;
      return (int)(p - pos);
    }
    if (i == 0) {
      double xx = 1.0, y = 0.0;
      int it = 0;
      while (-2.0 * y < xx * xx) {
        if (p + 2 > limit || ++it > kTailIters) return 0;
        const double x_ = from_bits(U[p++] >> 12, 0) - (1.0 - 2.220446049250313e-16 / 2.0);
        const double y_ = from_bits(U[p++] >> 12, 0) - (1.0 - 2.220446049250313e-16 / 2.0);
        xx = log(x_) / kZigR;
        y = log(y_);
      }
      *value = u < 0.0 ? xx - kZigR : kZigR - xx;
      return (int)(p - pos);
    }
    if (p >= limit) return 0;
    const double uu = (double)(U[p++] >> 11) * (1.0 / 9007199254740992.0);
    if (zf[i + 1] + (zf[i] - zf[i + 1]) * uu < exp(-x * x / 2.0)) {
      *value = x;
      return (int)(p - pos);
    }
  }
  return 0;
}

// The slow words of a segment: a bit per word, their list (in no order) and, after slow_draws, the
// length of the draw that starts at each (0: the stream or the tail-loop bound ran out).
struct SlowWords {
  uint32_t mask[kSegWords / 32];
  uint16_t list[kSegWords];
  uint16_t used[kSegWords];  // by word
  int count;
};

// Whether the draw that starts at this word is the word's own product (accepted at once).
__device__ __forceinline__ bool zig_fast(uint64_t bits, const uint64_t* accept) {
  const int64_t d = (int64_t)((bits >> 12) << 1) - ((int64_t)1 << 52);
  return (uint64_t)(d < 0 ? -d : d) < accept[bits & 0xff];
}

// Marks the slow words of the segment (every thread of the CTA; synchronises).
__device__ __forceinline__ void find_slow(const uint64_t* __restrict__ seg, const uint64_t* accept, SlowWords& sw) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) sw.count = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSegWords / kSegThreads; ++j) {
    const int w = j * kSegThreads + tid;
    const bool slow = !zig_fast(__ldg(seg + w), accept);
    const uint32_t m = __ballot_sync(0xffffffffu, slow);
    if (lane == 0) sw.mask[w >> 5] = m;
    if (slow) sw.list[atomicAdd(&sw.count, 1)] = (uint16_t)w;
  }
  __syncthreads();
}

// A CTA per segment: exit offset and draw count for every entry offset.
__global__ void __launch_bounds__(kSegThreads) zig_transfer_kernel(
    const uint64_t* __restrict__ U, uint64_t limit, const double* __restrict__ zt, const uint64_t* __restrict__ zaccept,
    int32_t* __restrict__ exit_off, int32_t* __restrict__ count, int* __restrict__ status) {
  __shared__ SlowWords sw;
  __shared__ uint64_t s_accept[256];
  const int tid = threadIdx.x;
  const uint64_t g = blockIdx.x, at = g * kSegWords;
  s_accept[tid] = zaccept[tid];
  find_slow(U + at, s_accept, sw);
  for (int i = tid; i < sw.count; i += kSegThreads) {
    double v;
    const int w = sw.list[i], used = zig_draw(U, at + w, limit, zt, zt + 257, &v);
    sw.used[w] = (uint16_t)used;
  }
  __syncthreads();
  if (tid < kEntries) {
    // lane e walks the draws from word e: between slow words every word is a draw
    int pos = tid, lost = tid;  // words that start no draw
    bool bad = false;
    for (int k = 0; k < kSegWords / 32; ++k)
      for (uint32_t m = sw.mask[k]; m; m &= m - 1) {
        const int r = k * 32 + __ffs(m) - 1;
        if (r < pos) continue;
        const int used = sw.used[r];
        bad |= used == 0;
        pos = r + max(used, 1);
        lost += min(pos, kSegWords) - r - 1;
      }
    const int ex = max(pos - kSegWords, 0);
    if (bad) atomicExch(status, 1);
    else if (ex >= kEntries) atomicExch(status, 2);
    exit_off[g * kEntries + tid] = min(ex, kEntries - 1);
    count[g * kEntries + tid] = kSegWords - lost;
  }
}

// A warp walks the maps of rows [r0, r1) (exit offset and draws of every entry offset) from entry
// offset e and draw index k, either per lane (composing the rows' maps) or the same in every lane
// (then `entry` and `base` receive what each row starts from).
template <class Count>
__device__ __forceinline__ void zig_walk(const int32_t* __restrict__ exit_off, const Count* __restrict__ count,
                                         uint64_t r0, uint64_t r1, int& e, uint64_t& k, int32_t* entry,
                                         uint64_t* base) {
  const int lane = threadIdx.x & 31;
  constexpr int kAhead = 4;  // rows loaded ahead of the dependent shuffles
  for (uint64_t r = r0; r < r1; r += kAhead) {
    int32_t ex[kAhead];
    Count ct[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const uint64_t row = min(r + j, r1 - 1) * kEntries + lane;
      ex[j] = __ldg(exit_off + row);
      ct[j] = __ldg(count + row);
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (r + j >= r1) break;
      if (entry && lane == 0) {
        entry[r + j] = e;
        base[r + j] = k;
      }
      k += (uint64_t)__shfl_sync(0xffffffffu, ct[j], e);
      e = __shfl_sync(0xffffffffu, ex[j], e);
    }
  }
}

// 32 warps over rows [r0, r1), a 32nd each: every warp composes its rows' maps, then warp 0 chains
// the 32 maps from (e, k) — per lane, so it composes them, or one value — and leaves in (s_e, s_k)
// what each warp's rows start from.  Returns the end of the chain in warp 0's e and k.
struct ZigBlock {
  int32_t exit[32][kEntries], e[32];
  uint64_t count[32][kEntries], k[32];
};
template <class Count>
__device__ __forceinline__ void zig_block(const int32_t* exit_off, const Count* count, uint64_t r0, uint64_t r1,
                                          ZigBlock& sh, int& e, uint64_t& k, int32_t* entry, uint64_t* base) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t per = (r1 - r0 + 31) / 32;
  const uint64_t a = min(r1, r0 + warp * per), b = min(r1, a + per);
  int we = lane;
  uint64_t wk = 0;
  zig_walk(exit_off, count, a, b, we, wk, nullptr, nullptr);
  sh.exit[warp][lane] = we;
  sh.count[warp][lane] = wk;
  __syncthreads();
  if (warp == 0)
    for (int w = 0; w < 32; ++w) {
      if (lane == 0) {
        sh.e[w] = e;
        sh.k[w] = k;
      }
      k += sh.count[w][e];
      e = sh.exit[w][e];
    }
  if (!entry) return;
  __syncthreads();
  we = sh.e[warp];
  wk = sh.k[warp];
  zig_walk(exit_off, count, a, b, we, wk, entry, base);
}

// A CTA per group of kGroupSegs segments: without `g_entry` the group's composed map, with it the
// entry offset and the global index of the first draw of each of the group's segments.
__global__ void __launch_bounds__(1024) zig_group_kernel(
    const int32_t* __restrict__ exit_off, const int32_t* __restrict__ count, uint64_t segs,
    int32_t* __restrict__ g_exit, uint64_t* __restrict__ g_count, const int32_t* __restrict__ g_entry,
    const uint64_t* __restrict__ g_base, int32_t* __restrict__ entry, uint64_t* __restrict__ base) {
  __shared__ ZigBlock sh;
  const uint64_t gr = blockIdx.x, s0 = gr * kGroupSegs, s1 = min(segs, s0 + kGroupSegs);
  int e = g_entry ? g_entry[gr] : (int)(threadIdx.x & 31);
  uint64_t k = g_entry ? g_base[gr] : 0;
  zig_block(exit_off, count, s0, s1, sh, e, k, entry, base);
  if (!g_entry && threadIdx.x < 32) {
    g_exit[gr * kEntries + threadIdx.x] = e;
    g_count[gr * kEntries + threadIdx.x] = k;
  }
}

// One CTA chains the groups from word 0: each group's entry and first draw index, and the total.
__global__ void __launch_bounds__(1024) zig_chain_kernel(const int32_t* __restrict__ g_exit,
                                                         const uint64_t* __restrict__ g_count, uint64_t groups,
                                                         int32_t* __restrict__ g_entry, uint64_t* __restrict__ g_base,
                                                         uint64_t* __restrict__ total) {
  __shared__ ZigBlock sh;
  int e = 0;
  uint64_t k = 0;
  zig_block(g_exit, reinterpret_cast<const unsigned long long*>(g_count), 0, groups, sh, e, k, g_entry, g_base);
  if (threadIdx.x == 0) *total = k;
}

// A CTA per segment: the normals of its draws with global index in
// [first, first + n).
__global__ void __launch_bounds__(kSegThreads) zig_emit_kernel(
    const uint64_t* __restrict__ U, uint64_t limit, uint64_t segs, const double* __restrict__ zt,
    const uint64_t* __restrict__ zaccept, const int32_t* __restrict__ entry, const uint64_t* __restrict__ base,
    uint64_t first, uint64_t n, double* __restrict__ out, int* __restrict__ status) {
  __shared__ SlowWords sw;
  __shared__ uint64_t s_accept[256];
  __shared__ double s_x[256], s_val[kSegWords];  // s_val: by list entry
  __shared__ uint32_t s_start[kSegWords / 32];   // words that start a draw
  __shared__ uint32_t s_rank[kSegWords / 32];    // draws before each 32 words
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t g = blockIdx.x, at = g * kSegWords;
  const uint64_t k0 = base[g];
  // the segment's draws lie in [base[g], base[g + 1])
  if (k0 >= first + n || (g + 1 < segs && base[g + 1] <= first)) return;
  s_accept[tid] = zaccept[tid];
  s_x[tid] = zt[tid];
  find_slow(U + at, s_accept, sw);
  for (int i = tid; i < sw.count; i += kSegThreads) {
    double v = 0.0;
    const int w = sw.list[i], used = zig_draw(U, at + w, limit, zt, zt + 257, &v);
    sw.used[w] = (uint16_t)used;
    s_val[i] = v;
  }
  if (tid < kSegWords / 32) s_start[tid] = 0xffffffffu;
  __syncthreads();
  if (tid == 0) {
    auto clear = [&](int a, int b) {  // words [a, b) start no draw
      for (int w = a; w < b; ++w) s_start[w >> 5] &= ~(1u << (w & 31));
    };
    int pos = entry[g];
    clear(0, pos);
    for (int k = 0; k < kSegWords / 32; ++k)
      for (uint32_t m = sw.mask[k]; m; m &= m - 1) {
        const int r = k * 32 + __ffs(m) - 1;
        if (r < pos) continue;
        const int used = sw.used[r];
        if (used == 0) atomicExch(status, 1);
        pos = r + max(used, 1);
        clear(r + 1, min(pos, kSegWords));
      }
  }
  __syncthreads();
  if (tid < 32) {
    // two mask words a lane: exclusive prefix of their popcounts
    const uint32_t a = __popc(s_start[2 * lane]), b = __popc(s_start[2 * lane + 1]);
    uint32_t sum = a + b;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, sum, off);
      if (lane >= off) sum += v;
    }
    s_rank[2 * lane] = sum - a - b;
    s_rank[2 * lane + 1] = sum - b;
  }
  __syncthreads();
  auto rank = [&](int w) { return s_rank[w >> 5] + __popc(s_start[w >> 5] & ((1u << (w & 31)) - 1u)); };
#pragma unroll
  for (int j = 0; j < kSegWords / kSegThreads; ++j) {
    const int w = j * kSegThreads + tid;
    const uint32_t bit = 1u << lane;
    if ((s_start[w >> 5] & ~sw.mask[w >> 5] & bit) == 0) continue;
    const uint64_t bits = __ldg(U + at + w), k = k0 + rank(w);
    if (k >= first && k < first + n) out[k - first] = (from_bits(bits >> 12, 1) - 3.0) * s_x[bits & 0xff];
  }
  for (int i = tid; i < sw.count; i += kSegThreads) {
    const int w = sw.list[i];
    if (!((s_start[w >> 5] >> (w & 31)) & 1u)) continue;
    const uint64_t k = k0 + rank(w);
    if (k >= first && k < first + n) out[k - first] = s_val[i];
  }
}

}  // namespace

void mc_normals(uint64_t seed, uint64_t first, uint64_t count, double* d_out, Workspace& W) {
  if (count == 0) return;
  const ZigTables& zt = zig_tables();
  const ChaKey key = chacha_key(seed);
  cudaStream_t s = W.stream;
  // words: a normal takes about 1.02 words on average (ziggurat acceptance); grow until they fit
  uint64_t need = first + count;
  uint64_t words = need + need / 32 + 8192;
  for (int attempt = 0; attempt < 4; ++attempt) {
    const uint64_t segs = (words + kSegWords - 1) / kSegWords;
    const uint64_t groups = (segs + kGroupSegs - 1) / kGroupSegs;
    const uint64_t blocks = (segs * kSegWords + 8 * 64 + 7) / 8;  // keystream padding past the last segment
    const uint64_t limit = blocks * 8;
    // status and total; tables; per segment its maps, entry and first index; the same per group
    struct Head {
      int status;
      uint64_t total;
    };
    const size_t o_tab = 256, o_seg64 = o_tab + sizeof(ZigTables),
                 o_seg32 = o_seg64 + 8 * (segs + groups * (kEntries + 1)),
                 bytes = o_seg32 + 4 * (segs * (2 * kEntries + 1) + groups * (kEntries + 1));
    uint8_t* aux = static_cast<uint8_t*>(W.device(WS_MCAUX, bytes));
    uint64_t* U = static_cast<uint64_t*>(W.device(WS_MCKEYS, limit * sizeof(uint64_t)));
    Head* head = reinterpret_cast<Head*>(aux);
    double* d_zt = reinterpret_cast<double*>(aux + o_tab);
    const uint64_t* d_accept = reinterpret_cast<const uint64_t*>(aux + o_tab + offsetof(ZigTables, accept));
    uint64_t* base = reinterpret_cast<uint64_t*>(aux + o_seg64);
    uint64_t *g_count = base + segs, *g_base = g_count + groups * kEntries;
    int32_t* exit_off = reinterpret_cast<int32_t*>(aux + o_seg32);
    int32_t *cnt = exit_off + segs * kEntries, *entry = cnt + segs * kEntries;
    int32_t *g_exit = entry + segs, *g_entry = g_exit + groups * kEntries;
    cuda_check(cudaMemsetAsync(aux, 0, sizeof(Head), s), "mc status");
    cuda_check(cudaMemcpyAsync(d_zt, &zt, sizeof zt, cudaMemcpyHostToDevice, s), "mc tables");
    chacha8_stream_kernel<<<(unsigned)((blocks + 127) / 128), 128, 0, s>>>(key, blocks, U);
    cuda_check(cudaGetLastError(), "chacha8_stream_kernel launch");
    zig_transfer_kernel<<<(unsigned)segs, kSegThreads, 0, s>>>(U, limit, d_zt, d_accept, exit_off, cnt, &head->status);
    cuda_check(cudaGetLastError(), "zig_transfer_kernel launch");
    zig_group_kernel<<<(unsigned)groups, 1024, 0, s>>>(exit_off, cnt, segs, g_exit, g_count, nullptr, nullptr, nullptr, nullptr);
    cuda_check(cudaGetLastError(), "zig_group_kernel launch");
    zig_chain_kernel<<<1, 1024, 0, s>>>(g_exit, g_count, groups, g_entry, g_base, &head->total);
    cuda_check(cudaGetLastError(), "zig_chain_kernel launch");
    zig_group_kernel<<<(unsigned)groups, 1024, 0, s>>>(exit_off, cnt, segs, nullptr, nullptr, g_entry, g_base, entry, base);
    cuda_check(cudaGetLastError(), "zig_group_kernel launch");
    // emits what there is; a stream that came out short is parsed again from more words
    zig_emit_kernel<<<(unsigned)segs, kSegThreads, 0, s>>>(U, limit, segs, d_zt, d_accept, entry, base, first, count, d_out,
                                                           &head->status);
    cuda_check(cudaGetLastError(), "zig_emit_kernel launch");
    if (W.timing) W.timing->kernel_launches += 6;
    Head h{};
    cuda_check(cudaMemcpyAsync(&h, head, sizeof h, cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "mc parse");
    if (h.status) raise(RG_ERR_GPU_ERROR, "ChaCha8 normal stream: ziggurat parse overflow");
    if (h.total >= need) return;
    words = words * 2;
  }
  raise(RG_ERR_GPU_ERROR, "ChaCha8 normal stream: could not size the keystream");
}

// ------------------------------------------------------------------ PathCube (pathcube.rs) ----
namespace {

// y = L·z per (path, time) in the reference's order (Cholesky::apply_into), stored as f32.
__global__ void correlate_block_kernel(const double* __restrict__ z, const double* __restrict__ L, int F,
                                       uint64_t cells, float* __restrict__ out) {
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cells) return;
  const double* zc = z + c * F;
  for (int i = 0; i < F; ++i) {
    double acc = 0.0;
    for (int j = 0; j <= i; ++j) acc += L[i * F + j] * zc[j];
    out[c * F + i] = (float)acc;
  }
}

// gbm_evolve (pathcube.rs:146-187): one thread per (path, factor), log-space FP64, f32 output.
__global__ void gbm_evolve_kernel(const double* __restrict__ s0, const double* __restrict__ vols, double rate,
                                  const double* __restrict__ q, int F, double dt, double sqrt_dt,
                                  const float* __restrict__ block, uint64_t paths, uint64_t times,
                                  float* __restrict__ out) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= paths * (uint64_t)F) return;
  const uint64_t p = t / F;
  const int f = (int)(t % F);
  double log_s = log(s0[f]);
  const double drift = (rate - q[f] - 0.5 * vols[f] * vols[f]) * dt;
  const double diffusion = vols[f] * sqrt_dt;
  for (uint64_t i = 0; i < times; ++i) {
    const uint64_t at = (p * times + i) * F + f;
    log_s += drift + diffusion * (double)block[at];
    out[at] = (float)exp(log_s);
  }
}

// Scratch for the engine-less entry points: plain device allocations freed on exit.
struct TempWorkspace : Workspace {
  DevBuf bufs[WS_NSLOTS];
  TempWorkspace() { sm_count = device_sm_count(); }
  void* device(int slot, size_t bytes) override {
    bufs[slot].ensure(bytes);
    return bufs[slot].ptr;
  }
  void* host(size_t) override { raise(RG_ERR_INVALID_ARGUMENT, "no host sums here"); }
};

}  // namespace

}  // namespace rg

using namespace rg;

extern "C" int32_t rg_chacha8_normals(uint64_t seed, uint64_t first, uint64_t count, double* out) {
  RG_TRY({
    int32_t g = rg_guard_device();
    if (g) return g;
    if (!out && count) raise(RG_ERR_INVALID_ARGUMENT, "null output");
    if (count > (uint64_t(1) << 31) || first > (uint64_t(1) << 40))
      raise(RG_ERR_INVALID_ARGUMENT, "at most 2^31 normals per call");
    TempWorkspace W;
    double* d = static_cast<double*>(W.device(WS_MCZ, sizeof(double) * (count ? count : 1)));
    mc_normals(seed, first, count, d, W);
    if (count) cuda_check(cudaMemcpy(out, d, sizeof(double) * count, cudaMemcpyDeviceToHost), "D2H normals");
  })
}

extern "C" int32_t rg_generate_correlated_block(uint64_t seed, int64_t paths, int64_t times, int32_t factors,
                                                const double* chol, float* out) {
  RG_TRY({
    int32_t g = rg_guard_device();
    if (g) return g;
    if (paths < 0 || times < 0 || factors < 1 || factors > RG_BOOK_MAX_UNIVERSE || !chol || (!out && paths && times))
      raise(RG_ERR_SHAPE_MISMATCH, "paths and times must be non-negative, 1..32 factors, non-null buffers");
    const uint64_t cells = (uint64_t)paths * (uint64_t)times, n = cells * (uint64_t)factors;
    if (n == 0) return RG_OK;
    if (n > (uint64_t(1) << 31)) raise(RG_ERR_INVALID_ARGUMENT, "at most 2^31 normals per block");
    TempWorkspace W;
    double* z = static_cast<double*>(W.device(WS_MCZ, sizeof(double) * n));
    mc_normals(seed, 0, n, z, W);
    DevBuf dl, dout;
    dl.ensure(sizeof(double) * factors * factors);
    dout.ensure(sizeof(float) * n);
    cuda_check(cudaMemcpy(dl.ptr, chol, sizeof(double) * factors * factors, cudaMemcpyHostToDevice), "H2D");
    correlate_block_kernel<<<(unsigned)((cells + 127) / 128), 128>>>(z, static_cast<double*>(dl.ptr), factors, cells,
                                                                    static_cast<float*>(dout.ptr));
    cuda_check(cudaGetLastError(), "correlate_block_kernel launch");
    cuda_check(cudaMemcpy(out, dout.ptr, sizeof(float) * n, cudaMemcpyDeviceToHost), "D2H block");
  })
}

extern "C" int32_t rg_gbm_evolve(const double* s0, const double* vols, double rate, const double* dividend_yields,
                                 int32_t factors, double dt, const float* block, int64_t paths, int64_t times,
                                 float* out) {
  RG_TRY({
    int32_t g = rg_guard_device();
    if (g) return g;
    if (factors < 1 || !s0 || !vols || !dividend_yields)
      raise(RG_ERR_SHAPE_MISMATCH, "s0, vols and dividend_yields must have equal length");
    if (paths < 0 || times < 0 || ((paths && times) && (!block || !out)))
      raise(RG_ERR_SHAPE_MISMATCH, "Brownian block factor count must match the spot count");
    const uint64_t n = (uint64_t)paths * (uint64_t)times * (uint64_t)factors;
    if (n == 0) return RG_OK;
    DevBuf ds, dv, dq, db, dout;
    ds.ensure(sizeof(double) * factors);
    dv.ensure(sizeof(double) * factors);
    dq.ensure(sizeof(double) * factors);
    db.ensure(sizeof(float) * n);
    dout.ensure(sizeof(float) * n);
    cuda_check(cudaMemcpy(ds.ptr, s0, sizeof(double) * factors, cudaMemcpyHostToDevice), "H2D");
    cuda_check(cudaMemcpy(dv.ptr, vols, sizeof(double) * factors, cudaMemcpyHostToDevice), "H2D");
    cuda_check(cudaMemcpy(dq.ptr, dividend_yields, sizeof(double) * factors, cudaMemcpyHostToDevice), "H2D");
    cuda_check(cudaMemcpy(db.ptr, block, sizeof(float) * n, cudaMemcpyHostToDevice), "H2D");
    const uint64_t threads = (uint64_t)paths * factors;
    gbm_evolve_kernel<<<(unsigned)((threads + 127) / 128), 128>>>(
        static_cast<double*>(ds.ptr), static_cast<double*>(dv.ptr), rate, static_cast<double*>(dq.ptr), factors, dt,
        std::sqrt(dt), static_cast<float*>(db.ptr), (uint64_t)paths, (uint64_t)times, static_cast<float*>(dout.ptr));
    cuda_check(cudaGetLastError(), "gbm_evolve_kernel launch");
    cuda_check(cudaMemcpy(out, dout.ptr, sizeof(float) * n, cudaMemcpyDeviceToHost), "D2H cube");
  })
}
