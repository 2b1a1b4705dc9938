// book_gen32.cu — FP32 universe increments of a book.
//
// incr[t][u][p] = ΔW (variance dt) of every (step, universe asset, path) of a chunk of paths,
// written once to HBM and read by every trade.  A CTA owns 64 consecutive paths and walks the
// bridge nodes in consumption order in tiles of B nodes, each in three phases between barriers:
//   G. normals — warp items (node, asset): lane l draws paths l and l + 32, whose Sobol integers
//      share one load of the consumption-order low-bit table and differ in the high-bit term of
//      their 32-point block (staged for 2·B nodes at a time); the two inverse normals run packed;
//   C. correlation — a warp takes a node: lane l holds the pair of paths 2l, 2l + 1 of all assets
//      and forms y_u = Σ_{b<=u} L[u][b]·z_b from the last asset down, in place;
//   B. bridge — a warp takes the assets u = warp, warp + 8, ...: the streamed bridge
//      (note.rs:89-106, qmc.rs:158-191) of each pair with the busy end of its anchor stack in shared
//      memory [depth][asset][path], and the increments of every step that completes.
// What bounds it: issue (54% active) and the waits at the phases' barriers: 132 instructions per (node, asset,
// 64 paths): two packed inverse normals, half of the 21 multiply-adds an asset's row of the factor averages,
// the bridge and the stores.  Up to 20 assets three CTAs fit an SM since the deep stack slots left shared
// memory (two with all of the stack there: a book of 64 trades on 2^17 paths 53.6 ms against 52.1).
// Measured on 20 assets × 1260 steps: 2.22 ms per 29,184 paths (one wave of three CTAs an SM; 1.66 per 19,456
// at two), against 11.0 ms per 19,456 for one thread per (path, asset) that formed every Sobol point from its
// own Gray code; 2^17 paths in three chunks 15.6 ms against 74 (two CTAs an SM, one pair of normals at a time).
// Every normal, correlation and bridge value is formed by the same operations in the same order as
// one thread per (path, asset) forms them.
#include <type_traits>

#include "rg_internal.h"
#include "rg_packed.cuh"

namespace rg {

constexpr int kGenPaths = 64;
constexpr int kGenWarps = 8;
constexpr int kGenTile = 8;  // nodes per tile where the shared memory holds them

// The bridge stack's last slots, which nearly every node uses (slot d from the end every 2^d steps), are in
// shared memory; the others in local memory.
constexpr int kGenFast = 5, kGenSlow = 20;

struct BookGenArgs {
  DevTrade gen;
  DevTables tb;
  const float* L32;
  int U, depth, nodes;  // nodes per tile
  uint64_t path0, npaths, rowlen;
  float* incr;
};

// Byte offsets of the dynamic shared memory, for the host's sizing and the kernel's carve-up alike.
struct BookGenLayout {
  uint32_t z, stk, hi, L, node, total;
};
__host__ __device__ inline BookGenLayout book_gen_layout(int U, int depth, int nodes) {
  BookGenLayout l;
  const uint32_t up = (uint32_t)(U + 3) / 4u * 4u, row = up * kGenPaths * 4u;
  l.z = 0;
  l.stk = l.z + (uint32_t)nodes * row;
  l.hi = l.stk + (uint32_t)(depth < kGenFast ? depth : kGenFast) * row;
  l.L = l.hi + 2u * (uint32_t)nodes * up * 16u;
  l.node = l.L + up * up * 8u;
  l.total = l.node + 8u * kGenTile;
  return l;
}

// UP: the universe's assets rounded up to four.  The loops over assets run to UP without a guard on
// what they read: entries past U hold whatever the memory did, and nothing below U depends on them.
template <int UP>
__global__ void __launch_bounds__(32 * kGenWarps, UP <= 20 ? 3 : 2) book_gen32_kernel(const __grid_constant__ BookGenArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int KA = (UP + kGenWarps - 1) / kGenWarps;  // assets per warp of the bridge
  constexpr int kRow = UP * kGenPaths;                  // floats per stack entry
  const DevTables& tb = A.tb;
  const int U = A.U, B = A.nodes, T = (int)A.gen.steps;
  // the warp's number by a shuffle: warp-uniform to the compiler
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const BookGenLayout lay = book_gen_layout(U, A.depth, B);
  float* z = reinterpret_cast<float*>(smem_raw + lay.z);      // [node][asset][path]
  float* stk = reinterpret_cast<float*>(smem_raw + lay.stk);  // [depth][asset][path]
  // high-bit terms of (node, asset) for paths 0-31 and 32-63: for lanes whose points lie in their
  // group's first 32-point block, then for lanes in the next
  uint2* hi = reinterpret_cast<uint2*>(smem_raw + lay.hi);
  float2* Ls = reinterpret_cast<float2*>(smem_raw + lay.L);  // [asset][asset] factor, each entry twice
  float* s_cf = reinterpret_cast<float*>(smem_raw + lay.node);  // the tile's nodes: standard deviation,
  int* s_done = reinterpret_cast<int*>(s_cf + kGenTile);        // and steps complete once it is on the stack
  const uint64_t p0 = (uint64_t)blockIdx.x * kGenPaths;
  for (int i = tid; i < U * U; i += blockDim.x) {
    const float v = __ldg(A.L32 + i);
    Ls[i / U * UP + i % U] = make_float2(v, v);
  }
  // Sobol points from the consumption-order tables when they were built for this launch's offset
  // within a 32-point block (else every point by itself)
  const uint64_t n1 = A.path0 + p0 + 1;  // Sobol point of the CTA's first path
  const bool lut = tb.sob_lut != nullptr && (int32_t)(n1 & 31) == tb.sob_lut_o;
  const bool upper = (uint32_t)tb.sob_lut_o + (uint32_t)lane >= 32u;  // point in the next 32-block
  const bool shift = A.gen.scrambler == RG_SCRAMBLE_DIGITAL_SHIFT;
  const int hi_n = 2 * B * U;  // entries of each of hi's halves
  // per pair of this warp's assets: the bridge's value at the current time and its next right anchor
  // (the stack's top)
  float2 wcur[KA], top[KA];
#pragma unroll
  for (int k = 0; k < KA; ++k) wcur[k] = top[k] = make_float2(0.0f, 0.0f);
  float* out = A.incr + (uint64_t)warp * A.rowlen + p0 + 2 * lane;  // this warp's first asset at step t
  const uint64_t out_asset = kGenWarps * A.rowlen, out_step = (uint64_t)U * A.rowlen;
  int t = 0, hi0 = 0;
  float* const sp = stk + warp * kGenPaths + 2 * lane;  // this warp's first asset in the first fast slot
  float2 deep[kGenSlow][KA];
  const int slow = max(A.depth - kGenFast, 0);
  int d = 0;  // stack entries
  auto slot = [&](int e, int k) -> float2& {
    return *reinterpret_cast<float2*>(sp + (e - slow) * kRow + k * kGenWarps * kGenPaths);
  };
  for (int c0 = 0; c0 < T; c0 += B) {
    const int nb = min(B, T - c0);
    if (lut && (c0 == 0 || c0 >= hi0 + 2 * B)) {
      // X(gray(a)) of the blocks of paths 0-31 and 32-63 and of the block after each, for the
      // dimensions of the next 2·B nodes: XORs of transposed direction rows
      hi0 = c0;
      const uint64_t blk = n1 >> 5;
      auto gray = [](uint64_t b) { return (uint32_t)((b << 5) ^ (b << 4)); };
      auto next_row = [](uint64_t b) { return min(__ffsll((long long)(b + 1)) - 1 + 5, 31); };
      const uint32_t ga = gray(blk), gb = gray(blk + 1);
      const int ra = next_row(blk), rb = next_row(blk + 1);
      const int nq = min(2 * B, T - c0) * U;
      for (int i = tid; i < nq; i += blockDim.x) {
        const uint32_t* col = tb.sob_t + (size_t)c0 * U + i;
        uint32_t a = 0, b = 0;
        for (uint32_t g = ga & gb; g; g &= g - 1u) a ^= __ldg(col + (size_t)(__ffs(g) - 1) * tb.sob_nq);
        b = a;
        for (uint32_t g = ga & ~gb; g; g &= g - 1u) a ^= __ldg(col + (size_t)(__ffs(g) - 1) * tb.sob_nq);
        for (uint32_t g = gb & ~ga; g; g &= g - 1u) b ^= __ldg(col + (size_t)(__ffs(g) - 1) * tb.sob_nq);
        hi[i] = make_uint2(a, b);
        const uint32_t v4 = __ldg(col + (size_t)4 * tb.sob_nq);
        hi[hi_n + i] = make_uint2(a ^ v4 ^ __ldg(col + (size_t)ra * tb.sob_nq), b ^ v4 ^ __ldg(col + (size_t)rb * tb.sob_nq));
      }
    }
    if (tid < nb) {
      s_cf[tid] = __ldg(tb.node_cf + c0 + tid);
      // the last step whose nodes all come no later than this one (node_off is sorted, and a node is
      // consumed at or before the step of its own index)
      int d = min(c0 + tid + 1, T);
      while (d > 0 && __ldg(tb.node_off + d) > c0 + tid + 1) --d;
      s_done[tid] = d;
    }
    __syncthreads();
    // ---- G: warp items, node by node over the warp's assets
    if (lut) {
      const uint2* hl = hi + (upper ? hi_n : 0) + (c0 - hi0) * U;
      const uint32_t* low = tb.sob_lut + (size_t)c0 * U * 32 + lane;
      const int items = nb * U;
      // the normals of `K` items, kGenWarps apart
      auto draw = [&](int it, auto shifted, auto count) {
        constexpr int K = decltype(count)::value;
        uint32_t l[K], xa[K], xb[K];
#pragma unroll
        for (int i = 0; i < K; ++i) l[i] = __ldg(low + (it + i * kGenWarps) * 32);
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const uint2 h = hl[it + i * kGenWarps];
          xa[i] = l[i] ^ h.x;
          xb[i] = l[i] ^ h.y;
          if constexpr (!decltype(shifted)::value) {
            const int e = it + i * kGenWarps;
            const uint64_t dim = (uint64_t)__ldg(tb.node_k + c0 + e / U) * U + e % U;
            xa[i] = rg_owen(xa[i], dim, A.gen.seed);
            xb[i] = rg_owen(xb[i], dim, A.gen.seed);
          }
        }
        float2 v[K];
        rg_probit32x2(xa, xb, v);
#pragma unroll
        for (int i = 0; i < K; ++i) {
          z[(it + i * kGenWarps) * kGenPaths + lane] = v[i].x;
          z[(it + i * kGenWarps) * kGenPaths + 32 + lane] = v[i].y;
        }
      };
      using One = std::integral_constant<int, 1>;
      if (shift) {
        constexpr int kI = 5;  // items in flight
        int it = warp;
        for (; it + (kI - 1) * kGenWarps < items; it += kI * kGenWarps)
          draw(it, std::true_type{}, std::integral_constant<int, kI>{});
        for (; it < items; it += kGenWarps) draw(it, std::true_type{}, One{});
      } else {
        for (int it = warp; it < items; it += kGenWarps) draw(it, std::false_type{}, One{});
      }
    } else {
      for (int it = warp; it < nb * U; it += kGenWarps) {
        const int c = it / U, u = it - c * U;
        const uint64_t dim = (uint64_t)__ldg(tb.node_k + c0 + c) * U + u;
        for (int h = 0; h < 64; h += 32) {
          const uint64_t p = p0 + h + lane;
          z[it * kGenPaths + h + lane] = rg_qmc_normal32(A.gen, tb, A.path0 + (p < A.npaths ? p : 0), dim);
        }
      }
    }
    __syncthreads();
    // ---- C
    for (int j = warp; j < nb; j += kGenWarps) {
      float2* zj = reinterpret_cast<float2*>(z + j * U * kGenPaths) + lane;
      float2 v[UP];
#pragma unroll
      for (int b = 0; b < UP; ++b) v[b] = zj[b * 32];
#pragma unroll
      for (int u = UP - 1; u >= 0; --u) {
        float2 y = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int b = 0; b <= u; ++b) y = __ffma2_rn(Ls[u * UP + b], v[b], y);
        if (u < UP - 3 || u < U) zj[u * 32] = y;
      }
    }
    __syncthreads();
    // ---- B
    const float2 half = make_float2(0.5f, 0.5f), minus = make_float2(-1.0f, -1.0f);
    const float* zb = z + warp * kGenPaths + 2 * lane;
    for (int j = 0; j < nb; ++j, zb += U * kGenPaths) {
      const int done = s_done[j];
      const float2 c2 = make_float2(s_cf[j], s_cf[j]);
      const bool first = c0 + j == 0;
#pragma unroll
      for (int k = 0; k < KA; ++k)
        if ((k + 1) * kGenWarps <= UP || warp + k * kGenWarps < UP) {
          const float2 y = *reinterpret_cast<const float2*>(zb + k * kGenWarps * kGenPaths);
          const float2 mid = __fmul2_rn(half, __fadd2_rn(wcur[k], top[k]));
          top[k] = first ? __fmul2_rn(y, c2) : __ffma2_rn(y, c2, mid);
          if (d < slow) deep[d][k] = top[k];
          else slot(d, k) = top[k];
        }
      ++d;
      // every step whose nodes are all here takes the top of the stack
      for (; t < done; ++t, out += out_step) {
        --d;
        const int below = max(d - 1, 0);  // the entry below (none after the last step: not used then)
#pragma unroll
        for (int k = 0; k < KA; ++k) {
          // rows are padded to whole CTAs' paths, so the last CTA stores all of its own
          if (warp + k * kGenWarps < U)
            *reinterpret_cast<float2*>(out + k * out_asset) = __ffma2_rn(wcur[k], minus, top[k]);
          wcur[k] = top[k];
          if ((k + 1) * kGenWarps <= UP || warp + k * kGenWarps < UP)
            top[k] = below < slow ? deep[below][k] : slot(below, k);
        }
      }
    }
    __syncthreads();
  }
}

// `rowlen` is a multiple of 64 (at least npaths).
void launch_book_gen32(const DevTrade& gen, const DevTables& tb, const float* L32, int U, int depth, uint64_t path0,
                       uint64_t npaths, uint64_t rowlen, float* incr, cudaStream_t s) {
  // eight nodes a tile, fewer where one CTA's shared memory would not hold them
  constexpr uint32_t kMax = 227u * 1024u;
  int nodes = kGenTile;
  while (nodes > 1 && book_gen_layout(U, depth, nodes).total > kMax) nodes >>= 1;
  const uint32_t smem = book_gen_layout(U, depth, nodes).total;
  if (smem > kMax || depth > kGenFast + kGenSlow)
    raise(RG_ERR_GPU_ERROR, "book generation: the bridge stack exceeds the shared-memory limit");
  if (rowlen % kGenPaths) raise(RG_ERR_GPU_ERROR, "book generation: rows must be padded to 64 paths");
  const BookGenArgs a{gen, tb, L32, U, depth, nodes, path0, npaths, rowlen, incr};
  const unsigned blocks = (unsigned)((npaths + kGenPaths - 1) / kGenPaths);
  auto go = [&](auto kernel) {
    // process-wide attribute: always the same value, so concurrent engines never lower it
    cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMax), "book gen smem attribute");
    kernel<<<blocks, 32 * kGenWarps, smem, s>>>(a);
    cuda_check(cudaGetLastError(), "book_gen32_kernel launch");
  };
  switch ((U + 3) / 4) {
    case 1: go(book_gen32_kernel<4>); break;
    case 2: go(book_gen32_kernel<8>); break;
    case 3: go(book_gen32_kernel<12>); break;
    case 4: go(book_gen32_kernel<16>); break;
    case 5: go(book_gen32_kernel<20>); break;
    case 6: go(book_gen32_kernel<24>); break;
    case 7: go(book_gen32_kernel<28>); break;
    default: go(book_gen32_kernel<32>); break;
  }
}

// The FP32 kernels' Sobol tables (DevTables::sob_t, sob_lut), in consumption order q = node·n + factor,
// from the direction table v on the device: st[k][q] = v[row(q)][k], and lut[q][j] for the lane j whose
// point is n1 + j, n1 = a + o with a a multiple of 32.  Gray codes are linear over XOR, so for
// o + j < 32 x(n1 + j) = X(gray(a)) ^ X(gray(o + j)), and otherwise x = X(gray(a + 32)) ^
// X(gray(o + j - 32)) with X(gray(a + 32)) = X(gray(a)) ^ v[4] ^ v[ctz(a/32 + 1) + 5]; lut holds the
// lane's low-bit term X(gray((o + j) mod 32)) with the digital shift folded in, and the kernels add the 32-path group's high-bit terms.  A CTA per 32 dimensions,
// thread (k, i) on direction k, then lane k, of dimension i.  (Built on the host the tables took
// 1.1 MB of upload per 1,000 steps of 3 assets, and 1 ms for a seed not seen before.)
__global__ void __launch_bounds__(1024) sobol_lut_kernel(DevTrade tr, DevTables tb, int n, int nq, uint32_t o,
                                                         uint32_t* __restrict__ st, uint32_t* __restrict__ lut) {
  __shared__ uint32_t v[32][33];
  const int k = threadIdx.x, i = threadIdx.y, q = blockIdx.x * 32 + i;
  const uint64_t dim = q < nq ? (uint64_t)__ldg(tb.node_k + q / n) * n + q % n : 0;
  v[i][k] = __ldg(tb.sobol + 32 * (dim % (uint64_t)tr.sob_dim) + k);
  __syncthreads();
  if (q < nq) {
    const uint32_t j = (o + k) & 31u, g = j ^ (j >> 1);
    uint32_t x = tr.scrambler == RG_SCRAMBLE_DIGITAL_SHIFT ? rg_digital_shift(dim, tr.seed) : 0u;
#pragma unroll
    for (int b = 0; b < 5; ++b)
      if ((g >> b) & 1u) x ^= v[i][b];
    lut[(size_t)q * 32 + k] = x;
  }
  if (blockIdx.x * 32 + k < nq) st[(size_t)i * nq + blockIdx.x * 32 + k] = v[k][i];
}

void launch_sobol_lut(const DevTrade& tr, DevTables& tb, int n, uint64_t first_path, uint32_t* out, cudaStream_t s) {
  const int nq = (int)tr.steps * n;
  tb.sob_t = out;
  tb.sob_lut = out + (size_t)32 * nq;
  tb.sob_nq = nq;
  tb.sob_lut_o = (int32_t)((first_path + 1) & 31);
  sobol_lut_kernel<<<(nq + 31) / 32, dim3(32, 32), 0, s>>>(tr, tb, n, nq, (uint32_t)tb.sob_lut_o, out,
                                                           out + (size_t)32 * nq);
  cuda_check(cudaGetLastError(), "sobol_lut_kernel launch");
}

}  // namespace rg
