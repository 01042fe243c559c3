// Batched personalized PageRank: K teleport vectors per sweep as one SpMM.
//
// Scores are an n x K row-major FP32 matrix (K columns interleaved per
// vertex), so one column-index load feeds K gathers and each gathered
// contribution row is K*4 contiguous bytes (fully used sectors). Column c is
// personalised PageRank with a one-hot teleport at seed_c:
//   r_c' = (1 - d) e_{seed_c} + d * A^T D^{-1} r_c,   r_c(0) = e_{seed_c},
// the per-vector form of the plain update (page_rank.hpp:133) with base_i
// replaced by (1 - d) [i == seed_c]. Each column stops at its own first sweep
// whose FP64 L1 change is below the threshold; its values are then frozen
// while the other columns continue.
//
// One sweep is four kernels: the gather (merge-path tiles of W items, a group
// of K/4 lanes per tile, so a warp walks 128/K tiles side by side), the fix-up
// of rows that cross tiles, a streaming epilogue over the n x K matrix
// (update, FP64 per-column residual, next contributions) and the per-column
// convergence test. K is the batch size rounded up to 8, 16, 32, 64 or 128.
#include "common.cuh"
#include "engine.h"
#include "ppr.h"

namespace nwgpu {

// ---------------------------------------------------------------------------
// Gather. A tile is kPprTileItems merge items (entries and row ends); its
// entries are summed in order into K running sums, and a finished row stores
// its sums z into the output contribution matrix (the update, the residual and
// the next contributions are the epilogue kernel's, so nothing in this loop
// waits on a load other than the gathers). The first row of a tile that
// started in an earlier tile leaves its partial in epart[t], the last row that
// continues past the tile in cpart[t].
//
// A lane owns four columns (one 16-byte load per entry), so a tile takes
// P = K/4 lanes and a warp walks 32/P tiles at once: the instructions per
// entry fall with K, where a warp per tile would spend the same ~12 on an
// entry whatever its width. Every column is summed in the same order at every
// K: the tiles, the order within them and the crossing rows' partials do not
// depend on it.
//
// Entries come in blocks of 16, aligned to 16 in the CSR: the group's first
// lanes hold four column ids each (eight at K = 8, in 16-byte loads), and
// weights likewise, passed on by shuffles. Which entries end a row is one bit
// each (end_bits, built once per graph), so no row pointer is read per row.
// The next block's ids load while this block's rows do, and the rows of one
// sub-block of 8 entries are in flight while the sub-block before it is summed
// (64 floats per lane, two CTAs of 256 threads per SM). Blocks that lie wholly
// in their tiles, and sub-blocks in which no group's row ends, skip the
// per-entry tests (a warp vote): the walk spends ~10 instructions on an entry
// of each group instead of ~19, which made the gather 1.3x faster at K = 16.
//
// Bound by the bytes an SM takes from L2 (4 K per entry) and, below K = 32, by
// instruction issue. Measured per sweep on RMAT scale 20 (31.4M entries),
// against the warp-per-tile kernel below, which pads to 32 columns: K = 16 197
// to 417 us, K = 32 301 to 419; weighted K = 16 215 to 829, K = 32 357 to 830
// (that kernel loads every weight in every lane). Sub-blocks of 4 entries and
// three CTAs per SM: 210 us at K = 16.
// ---------------------------------------------------------------------------
constexpr int kBlock = 16, kSub = 8;  // entries per block and sub-block

// A lane holds N entries of the block: N = 16 / P for P < 4 lanes per group, else 4 (lanes sub < 4).
template <int N>
struct Block {
  uint32_t id[N];  // column ids of entries base + N sub ..
  float    w[N];   // their weights (weighted solves), 0 outside the tile
  uint32_t mask;   // bits 0..15: entry base + u is in the tile; bits 16..31: it ends its row
  bool     full;   // every group's block lies wholly in its tile (warp-uniform)
};

template <int N, bool WEIGHTED>
__device__ __forceinline__ Block<N> load_block(const PprArgs& a, uint32_t base, uint32_t k0, uint32_t k1, int sub) {
  Block<N>       b{};
  const uint32_t lo = k0 > base ? k0 - base : 0u;  // entries [lo, hi) of the block are the tile's
  const uint32_t hi = k1 > base ? min(k1 - base, (uint32_t)kBlock) : 0u;
  b.full = __all_sync(kFullMask, lo == 0u && hi == (uint32_t)kBlock);
  if (lo >= hi) return b;
  const uint32_t in = ((1u << hi) - 1u) & ~((1u << lo) - 1u);
  const uint32_t ends = __ldg(a.end_bits + (base >> 5)) >> (base & 31u);
  b.mask = in | ((ends & in) << 16);
#pragma unroll
  for (int q = 0; q < N; q += 4) {
    // the words reach at most 3 entries past the tile's last one: inside the arrays' padding
    const uint32_t first = (uint32_t)(N * sub + q);
    if (first >= hi || first + 4u <= lo) continue;
    const uint4 id = ld_stream4(reinterpret_cast<const uint4*>(a.col + base + first));
    b.id[q] = id.x;
    b.id[q + 1] = id.y;
    b.id[q + 2] = id.z;
    b.id[q + 3] = id.w;
    if (WEIGHTED) {
      const float4 w = __ldcs(reinterpret_cast<const float4*>(a.w + base + first));
      b.w[q] = (in >> first) & 1u ? w.x : 0.f;
      b.w[q + 1] = (in >> first) & 2u ? w.y : 0.f;
      b.w[q + 2] = (in >> first) & 4u ? w.z : 0.f;
      b.w[q + 3] = (in >> first) & 8u ? w.w : 0.f;
    }
  }
  return b;
}

// Rows of the block's entries kSub s .. kSub s + 7; entries outside the tile give 0.
template <int K, int N>
__device__ __forceinline__ void issue(float4 (&v)[kSub], const Block<N>& b, int s, int group,
                                      const float* __restrict__ cin4, uint64_t pol) {
  const uint32_t m = b.mask >> (kSub * s);
  const float*   row[kSub];
#pragma unroll
  for (int u = 0; u < kSub; ++u)
    row[u] = cin4 + (uint64_t)__shfl_sync(kFullMask, b.id[u % N], group * (K / 4) + (kSub * s + u) / N) * K;
  if (b.full) {
#pragma unroll
    for (int u = 0; u < kSub; ++u) v[u] = ld_gather4(reinterpret_cast<const float4*>(row[u]), pol);
  } else {
#pragma unroll
    for (int u = 0; u < kSub; ++u) {
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m & (1u << u)) v[u] = ld_gather4(reinterpret_cast<const float4*>(row[u]), pol);
    }
  }
}

template <int K, bool WEIGHTED>
__global__ void __launch_bounds__(kPprThreads, 2) ppr_gather_kernel(const PprArgs a) {
  constexpr int P = K / 4, G = 32 / P, N = P < 4 ? kBlock / P : 4;
  static_assert(kBlock == 2 * kSub, "two sub-blocks in flight");
  const int     lane = threadIdx.x & 31, sub = lane & (P - 1), group = lane / P;
  PprState*     st = a.st;
  if (a.use_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(a.cond, 0u);
  if (*(volatile unsigned int*)&st->done) return;
  const unsigned long long it = *(volatile unsigned long long*)&st->iter;
  const float* __restrict__ cin4 = ((it & 1ull) ? a.contrib1 : a.contrib0) + 4 * sub;
  float* __restrict__ cout4 = ((it & 1ull) ? a.contrib0 : a.contrib1) + 4 * sub;
  const uint64_t pol = policy_evict_last();

  const uint32_t gwarp = (blockIdx.x * kPprThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kPprThreads / 32);
  // Fewer tiles than groups: spread them over all warps, for groups beside one another share their branches and
  // their warp's issue slots (RMAT, K = 8: 40 and 48 us a sweep at scales 13 and 15, 55 at scale 14 with full warps).
  const uint32_t per = (uint32_t)min((uint64_t)G, ((uint64_t)a.num_tiles + nwarps - 1u) / nwarps);
  for (uint64_t t0 = (uint64_t)gwarp * per; t0 < a.num_tiles; t0 += (uint64_t)nwarps * per) {
    const uint64_t t = (uint32_t)group < per ? t0 + (uint32_t)group : a.num_tiles;
    uint32_t       r1 = 0u, k0 = 0u, k1 = 0u, row = 0u, pos = 0u;
    bool           carry = false;
    float*         dst = cout4;  // where the current row's sums go when it ends in this tile
    if (t < a.num_tiles) {
      row = a.tile_row[t];
      r1 = a.tile_row[t + 1];
      k0 = a.tile_nnz[t];
      k1 = a.tile_nnz[t + 1];
      const uint32_t s0 = __ldg(a.row_ptr + row), s1 = row < r1 ? __ldg(a.row_ptr + row + 1) : k1 + 1u;
      carry = k1 > __ldg(a.row_ptr + r1);  // row r1 has entries here and ends in a later tile
      bool cont = s0 < k0;                 // the first row started in an earlier tile
      if (cont && s1 == k0) {              // and all its entries are there: only its end is this tile's
        *reinterpret_cast<float4*>(a.epart + t * K + 4 * sub) = make_float4(0.f, 0.f, 0.f, 0.f);
        cont = false;
        ++row;
      }
      if (!WEIGHTED && a.full_rows) {  // rows without entries lie between the others: walk the list of those that have some
        pos = a.tile_full[t] + (row > a.tile_row[t] ? 1u : 0u);
        if (pos < a.num_full) row = a.full_rows[pos];
      }
      dst = cont ? a.epart + t * K + 4 * sub : cout4 + (uint64_t)row * K;
    }
    const uint32_t base0 = k0 & ~(uint32_t)(kBlock - 1);
    const uint32_t blocks = __reduce_max_sync(kFullMask, k1 > k0 ? (k1 - base0 + kBlock - 1u) / kBlock : 0u);
    float4         acc = make_float4(0.f, 0.f, 0.f, 0.f);
    auto           consume = [&](const float4(&v)[kSub], const Block<N>& blk, int s) {
      const uint32_t ends = (blk.mask >> (16 + kSub * s)) & ((1u << kSub) - 1u);
      float          w[kSub];
#pragma unroll
      for (int u = 0; u < kSub; ++u)
        w[u] = WEIGHTED ? __shfl_sync(kFullMask, blk.w[u % N], group * P + (kSub * s + u) / N) : 1.f;
      auto add = [&](int u) {
        acc.x = WEIGHTED ? fmaf(w[u], v[u].x, acc.x) : acc.x + v[u].x;
        acc.y = WEIGHTED ? fmaf(w[u], v[u].y, acc.y) : acc.y + v[u].y;
        acc.z = WEIGHTED ? fmaf(w[u], v[u].z, acc.z) : acc.z + v[u].z;
        acc.w = WEIGHTED ? fmaf(w[u], v[u].w, acc.w) : acc.w + v[u].w;
      };
      if (!__any_sync(kFullMask, ends != 0u)) {
#pragma unroll
        for (int u = 0; u < kSub; ++u) add(u);
        return;
      }
#pragma unroll
      for (int u = 0; u < kSub; ++u) {
        add(u);
        if (((ends >> u) & 1u) && row < r1) {
          *reinterpret_cast<float4*>(dst) = acc;
          acc = make_float4(0.f, 0.f, 0.f, 0.f);
          if (!WEIGHTED && a.full_rows) row = ++pos < a.num_full ? a.full_rows[pos] : r1;
          else ++row;
          dst = cout4 + (uint64_t)row * K;
        }
      }
    };
    float4   va[kSub], vb[kSub];
    Block<N> cur = load_block<N, WEIGHTED>(a, base0, k0, k1, sub);
    issue<K>(va, cur, 0, group, cin4, pol);
#pragma unroll 1
    for (uint32_t b = 1; b <= blocks; ++b) {
      const Block<N> nxt = load_block<N, WEIGHTED>(a, base0 + b * kBlock, k0, k1, sub);
      issue<K>(vb, cur, 1, group, cin4, pol);
      consume(va, cur, 0);
      issue<K>(va, nxt, 0, group, cin4, pol);
      consume(vb, cur, 1);
      cur = nxt;
    }
    if (carry) *reinterpret_cast<float4*>(a.cpart + t * K + 4 * sub) = acc;
  }
}

template <int K>
struct Cols {
  static constexpr int PER_LANE = K / 32;
  float v[PER_LANE];
};

template <int K>
__device__ __forceinline__ void load_row(Cols<K>& out, const float* __restrict__ base, uint32_t row, int lane,
                                         uint64_t pol) {
  const float* p = base + (uint64_t)row * K + lane * Cols<K>::PER_LANE;
  if constexpr (Cols<K>::PER_LANE == 1) {
    out.v[0] = ld_gather(p, pol);
  } else if constexpr (Cols<K>::PER_LANE == 2) {
    float2 t;
    asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0,%1}, [%2], %3;" : "=f"(t.x), "=f"(t.y) : "l"(p), "l"(pol));
    out.v[0] = t.x;
    out.v[1] = t.y;
  } else {
    const float4 t = ld_gather4(reinterpret_cast<const float4*>(p), pol);
    out.v[0] = t.x;
    out.v[1] = t.y;
    out.v[2] = t.z;
    out.v[3] = t.w;
  }
}

// ---------------------------------------------------------------------------
// Gather, a warp per tile, lanes owning K/32 columns each: unweighted solves of
// 64 and 128 columns and weighted ones of 128, where the walk above has one or
// two tiles per warp and the loads, not the instructions, bound both (per
// sweep on RMAT, against the walk above: scale 22, K = 64 2.28 to 2.33 ms; scale
// 20, K = 128 0.97 to 1.02 ms; scale 17 weighted K = 128 154 to 160 us, but
// scale 18 weighted K = 64 203 to 177); and unweighted solves of at most 32
// columns on graphs with no more tiles than the walk above has warps
// (ppr_few_tiles), where a tile's chain of loads is all of the time and a
// warp has 16 rows of it in flight, not 8 (scale 15, 16 columns: 39 to 47 us;
// scale 10: 35 to 36; scale 17, past the line: 67 to 61). A warp walks its tile's
// entries in order, U rows of the contribution matrix per group, and loads
// the next group while it sums the current one (2 * U * K * 4 bytes in flight
// per warp: 4 KB for every K). Column ids and row ends of the tile are staged
// in shared memory; the next row end sits in a register. A finished row only
// stores its K sums (z) into the output contribution matrix: the update, the
// residual and the next contributions are the epilogue kernel's, so nothing
// in this loop waits on a load other than the gathers. The first row of a
// tile that started in an earlier tile leaves its partial in epart[t], the
// last row that continues past the tile in cpart[t].
// ---------------------------------------------------------------------------
template <int K, int U>
__device__ __forceinline__ void load_group(Cols<K> (&v)[U], const float* __restrict__ cin, const uint32_t* s_col, int g,
                                           int E, int lane, uint64_t pol) {
  if ((g + 1) * U <= E) {  // a full group: no bounds checks
#pragma unroll
    for (int u = 0; u < U; ++u) load_row<K>(v[u], cin, s_col[g * U + u], lane, pol);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (g * U + u < E) load_row<K>(v[u], cin, s_col[g * U + u], lane, pol);
  }
}
// Weighted solves: the group's entry weights (the same address in every lane).
template <int U>
__device__ __forceinline__ void load_weights(float (&wv)[U], const float* __restrict__ w, uint32_t k0, int g, int E) {
#pragma unroll
  for (int u = 0; u < U; ++u) wv[u] = (g * U + u < E) ? __ldg(w + k0 + g * U + u) : 0.f;
}

template <int K, int W, int U, bool WEIGHTED>
__global__ void __launch_bounds__(256) ppr_gather_warp_kernel(const PprArgs a) {
  constexpr int P = Cols<K>::PER_LANE;
  constexpr int NWARP = 256 / 32;
  __shared__ uint32_t s_col[NWARP][W + 1];
  __shared__ uint32_t s_rp[NWARP][W + 2];
  const int           lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PprState*           st = a.st;
  if (a.use_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(a.cond, 0u);
  if (*(volatile unsigned int*)&st->done) return;
  const unsigned long long it = *(volatile unsigned long long*)&st->iter;
  const float* __restrict__ cin = (it & 1ull) ? a.contrib1 : a.contrib0;
  float* __restrict__ cout = (it & 1ull) ? a.contrib0 : a.contrib1;
  const uint64_t pol = policy_evict_last();

  const uint32_t gwarp = blockIdx.x * NWARP + warp, nwarps = gridDim.x * NWARP;
  for (uint32_t t = gwarp; t < a.num_tiles; t += nwarps) {
    const uint32_t r0 = a.tile_row[t], r1 = a.tile_row[t + 1], k0 = a.tile_nnz[t], k1 = a.tile_nnz[t + 1];
    const int      R = (int)(r1 - r0), E = (int)(k1 - k0);
    for (int j = lane; j < E; j += 32) s_col[warp][j] = __ldcs(a.col + k0 + j);
    for (int j = lane; j <= R; j += 32) s_rp[warp][j] = __ldcs(a.row_ptr + r0 + j);
    __syncwarp();
    const bool is_cont = s_rp[warp][0] < k0;
    const bool has_co = k1 > s_rp[warp][R];
    Cols<K>    acc;
#pragma unroll
    for (int q = 0; q < P; ++q) acc.v[q] = 0.f;
    int i = 0;  // next row (relative) to finish
    int next_end = (R > 0) ? (int)(s_rp[warp][1] - k0) : 0x7fffffff;
    auto flush = [&]() {
      float* dst = (i == 0 && is_cont) ? a.epart + (uint64_t)t * K : cout + (uint64_t)(r0 + i) * K;
#pragma unroll
      for (int q = 0; q < P; ++q) {
        dst[lane * P + q] = acc.v[q];
        acc.v[q] = 0.f;
      }
      ++i;
      next_end = (i < R) ? (int)(s_rp[warp][i + 1] - k0) : 0x7fffffff;
    };
    // one term: the gathered contribution (times the entry's weight when weighted)
    auto add = [&](const Cols<K>& v, float wgt) {
#pragma unroll
      for (int q = 0; q < P; ++q) acc.v[q] = WEIGHTED ? fmaf(wgt, v.v[q], acc.v[q]) : acc.v[q] + v.v[q];
    };
    auto consume = [&](const Cols<K>(&v)[U], const float(&wv)[U], int g) {
      const int e0 = g * U;
      if (next_end >= e0 + U && e0 + U <= E) {  // a full group inside the current row
#pragma unroll
        for (int u = 0; u < U; ++u) add(v[u], wv[u]);
        return;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u;
        if (e < E) {
          while (next_end <= e) flush();
          add(v[u], wv[u]);
        }
      }
    };
    Cols<K> va[U], vb[U];
    float   wa[U], wb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) wa[u] = wb[u] = 1.f;
    load_group<K, U>(va, cin, s_col[warp], 0, E, lane, pol);
    if (WEIGHTED) load_weights<U>(wa, a.w, k0, 0, E);
    for (int g = 0; g * U < E; g += 2) {
      load_group<K, U>(vb, cin, s_col[warp], g + 1, E, lane, pol);
      if (WEIGHTED) load_weights<U>(wb, a.w, k0, g + 1, E);
      consume(va, wa, g);
      if ((g + 1) * U >= E) break;
      load_group<K, U>(va, cin, s_col[warp], g + 2, E, lane, pol);
      if (WEIGHTED) load_weights<U>(wa, a.w, k0, g + 2, E);
      consume(vb, wb, g + 1);
    }
    while (next_end <= E) flush();  // rows ending at the tile's last entry, and empty rows after it
    if (has_co) {
#pragma unroll
      for (int q = 0; q < P; ++q) a.cpart[(uint64_t)t * K + lane * P + q] = acc.v[q];
    }
    __syncwarp();
  }
}

// One bit per entry: it is the last of its row. full: rows that have entries.
__global__ void ppr_row_ends_kernel(const uint32_t* __restrict__ row_ptr, uint64_t n, uint32_t* __restrict__ end_bits,
                                    unsigned int* __restrict__ full) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned int   mine = 0;
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
    const uint32_t e = row_ptr[r + 1];
    if (e == row_ptr[r]) continue;
    atomicOr(end_bits + ((e - 1u) >> 5), 1u << ((e - 1u) & 31u));
    ++mine;
  }
  mine = __reduce_add_sync(kFullMask, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(full, mine);
}

// Per tile: its first row's place in the list of rows that have entries.
__global__ void ppr_tile_full_kernel(const uint32_t* __restrict__ tile_row, uint32_t T, const uint32_t* __restrict__ rows,
                                     uint32_t num, uint32_t* __restrict__ tile_full) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
    const uint32_t want = tile_row[t];
    uint32_t       lo = 0, hi = num;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (rows[mid] < want)
        lo = mid + 1;
      else
        hi = mid;
    }
    tile_full[t] = lo;
  }
}

// Rows that cross warp tiles are fixed by the tiling: listed once per graph
// as (row, first tile, last tile). K/4 lanes per listed row sum its tile
// partials in tile order into z.
__global__ void ppr_spans_kernel(const uint32_t* __restrict__ row_ptr, const uint32_t* __restrict__ tile_row,
                                 const uint32_t* __restrict__ tile_nnz, uint32_t T, uint32_t D, uint4* __restrict__ spans,
                                 unsigned int* __restrict__ count) {
  for (uint32_t ta = blockIdx.x * blockDim.x + threadIdx.x; ta + 1 < T; ta += gridDim.x * blockDim.x) {
    const uint32_t S = tile_row[ta + 1];
    const uint32_t k1 = tile_nnz[ta + 1], rs = row_ptr[S];
    if (!(k1 > rs && ((uint64_t)S + rs) / D == ta)) continue;  // the carried-out row does not start in ta
    const uint32_t tb = (uint32_t)(((uint64_t)S + row_ptr[S + 1]) / D);
    spans[atomicAdd(count, 1u)] = make_uint4(S, ta, tb, 0u);
  }
}

template <int K>
__global__ void __launch_bounds__(256) ppr_fixup_kernel(const PprArgs a) {
  constexpr int P = K / 4;  // lanes per row, four columns each
  PprState*     st = a.st;
  if (*(volatile unsigned int*)&st->done) return;
  const unsigned long long it = *(volatile unsigned long long*)&st->iter;
  float* __restrict__ cout = (it & 1ull) ? a.contrib0 : a.contrib1;
  const uint32_t th = blockIdx.x * blockDim.x + threadIdx.x, sub = th % P, ngroups = gridDim.x * blockDim.x / P;
  for (uint32_t sp = th / P; sp < a.num_spans; sp += ngroups) {
    const uint4   span = a.spans[sp];
    const float4* part = reinterpret_cast<const float4*>(a.cpart) + sub;
    // 8 interleaved partial sums (tile u goes to sum (u - first) % 8), combined in order
    float4 z[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) z[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 e = __ldcg(reinterpret_cast<const float4*>(a.epart) + (uint64_t)span.z * P + sub);
    for (uint32_t u = span.y; u < span.z; u += 16) {  // 16 loads in flight
      float4 x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        x[j] = u + j < span.z ? __ldcg(part + (uint64_t)(u + j) * P) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        z[j % 8].x += x[j].x;
        z[j % 8].y += x[j].y;
        z[j % 8].z += x[j].z;
        z[j % 8].w += x[j].w;
      }
    }
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      t.x += z[j].x;
      t.y += z[j].y;
      t.z += z[j].z;
      t.w += z[j].w;
    }
    reinterpret_cast<float4*>(cout)[(uint64_t)span.x * P + sub] = make_float4(t.x + e.x, t.y + e.y, t.z + e.z, t.w + e.w);
  }
}

// Epilogue, streaming over the n x K matrix, four columns per thread (16-byte
// loads and stores): for each active column c, r' = (1 - d)[i == seed_c] + d z
// (or (1 - d) t_ic + d z with teleport vectors),
// FP64 |r' - r| into per-CTA column partials; converged columns keep their
// ranks. contrib = r' / deg_i for every column. The grid stride is a multiple
// of K / 4, so every thread stays on one group of four columns.
// EPI: kPprSeeds (one-hot teleports, out-degrees), kPprWeighted (base terms
// (1 - d) t, out-weight sums), kPprTeleports (base terms, out-degrees).
template <int K, int EPI>
__global__ void __launch_bounds__(256) ppr_epilogue_kernel(const PprArgs a, uint64_t n) {
  constexpr int     C4 = K / 4;
  __shared__ double s_res[256][4];
  PprState*         st = a.st;
  if (*(volatile unsigned int*)&st->done) return;
  const unsigned long long it = *(volatile unsigned long long*)&st->iter;
  float* __restrict__ cout = (it & 1ull) ? a.contrib0 : a.contrib1;
  const uint64_t total = n * C4, stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t x0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int      c0 = (int)(x0 % C4) * 4;
  bool           act[4];
  uint32_t       seed[4];
  bool           any = false;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    act[q] = a.col_done[c0 + q] == 0u;
    seed[q] = a.seeds[c0 + q];
    any = any || act[q];
  }
  const uint64_t pol = policy_evict_last();
  double         res[4] = {0.0, 0.0, 0.0, 0.0};
  if (any) {
    for (uint64_t x = x0; x < total; x += stride) {
      const uint32_t i = (uint32_t)(x / C4);
      // the gather leaves the rows without entries alone: their sum is 0
      const bool     full = a.full_rows ? __ldg(a.row_ptr + i) != __ldg(a.row_ptr + i + 1) : i < a.num_full;
      const float4   z = full ? __ldcs(reinterpret_cast<const float4*>(cout) + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4   old = __ldcs(reinterpret_cast<const float4*>(a.rank) + x);
      // weighted: divide by the out-weight sum; the base terms are (1 - d) t
      const float    dg = EPI == kPprWeighted ? __ldg(a.vaux + i) : (float)__ldg(a.deg + i);
      float4         tb = make_float4(0.f, 0.f, 0.f, 0.f);
      if (EPI != kPprSeeds) tb = __ldg(reinterpret_cast<const float4*>(a.vbase) + x);
      const float    zv[4] = {z.x, z.y, z.z, z.w}, ov[4] = {old.x, old.y, old.z, old.w};
      const float    bv[4] = {tb.x, tb.y, tb.z, tb.w};
      float          nr[4], co[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float tele = EPI != kPprSeeds ? bv[q] : ((seed[q] == i) ? a.one_minus_d : 0.f);
        nr[q] = act[q] ? fmaf(a.damping, zv[q], tele) : ov[q];
        co[q] = nr[q] / dg;
        if (act[q]) res[q] += (double)fabsf(nr[q] - ov[q]);
      }
      __stcs(reinterpret_cast<float4*>(a.rank) + x, make_float4(nr[0], nr[1], nr[2], nr[3]));
      st_keep4(reinterpret_cast<float4*>(cout) + x, make_float4(co[0], co[1], co[2], co[3]), pol);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) s_res[threadIdx.x][q] = res[q];
  __syncthreads();
  if (threadIdx.x < K) {
    const int g = threadIdx.x / 4, q = threadIdx.x % 4;
    double    b = 0.0;
    for (int j = g; j < (int)blockDim.x; j += C4) b += s_res[j][q];
    a.res_part[(uint64_t)blockIdx.x * K + threadIdx.x] = b;
  }
}

// Per-column residuals over the epilogue's CTAs and the per-column
// convergence test: one warp per column (K / 8 CTAs), lane-strided over the
// partials with a fixed tree; the last CTA to arrive updates the solve state.
template <int K>
__global__ void __launch_bounds__(256) ppr_finish_kernel(const PprArgs a) {
  __shared__ int s_last;
  PprState*      st = a.st;
  if (*(volatile unsigned int*)&st->done) return;
  const unsigned long long it = *(volatile unsigned long long*)&st->iter;
  const int      lane = threadIdx.x & 31, c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c < K && !a.col_done[c]) {  // uniform across the warp
    // lane-strided, in order, 8 loads in flight (one at a time they were 10 us of every sweep)
    double e = 0.0;
    for (uint32_t u = lane; u < a.epi_grid; u += 256u) {
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = u + 32u * j < a.epi_grid ? __ldcg(a.res_part + (uint64_t)(u + 32u * j) * K + c) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) e += v[j];
    }
    e = warp_sum_lane0(e);
    if (lane == 0) {
      a.col_err[c] = e;
      a.col_iters[c] = (uint32_t)(it + 1ull);
      if (e < st->threshold) {
        a.col_done[c] = 1u;
        a.col_conv[c] = 1u;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = (atomicAdd(&st->ticket, 1u) == gridDim.x - 1u);
  }
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  __threadfence();
  unsigned int running = 0u;
  for (int q = 0; q < K; ++q) running += *(volatile uint32_t*)&a.col_done[q] == 0u ? 1u : 0u;
  const bool               all_done = running == 0u;
  const unsigned long long done_iters = it + 1ull;
  st->iter = done_iters;
  const bool abort = a.abort_word && *a.abort_word;
  const bool end = all_done || done_iters >= st->max_iters || abort;
  // few enough columns still run to continue in a narrower layout: stop here for the host to repack
  const bool narrow = !end && st->narrow_at != 0u && running <= st->narrow_at;
  const bool done = end || narrow;
  st->aborted = (abort && !all_done) ? 1u : 0u;
  st->narrowed = narrow ? 1u : 0u;
  st->done = done ? 1u : 0u;
  st->ticket = 0u;
  __threadfence();
  if (a.use_cond && !done && done_iters < st->chunk_end) cudaGraphSetConditional(a.cond, 1u);
}

// rank(i, c) = [i == seed_c], contrib = rank / deg; four columns per thread.
template <int K>
__global__ void ppr_init_kernel(const PprArgs a, uint64_t n) {
  constexpr uint32_t C4 = K / 4;
  const uint64_t     total = n * C4;
  const uint64_t     stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const uint32_t i = (uint32_t)(x / C4);
    const int      c = (int)(x % C4) * 4;
    const float    dg = (float)__ldg(a.deg + i), none = 0.f / dg, one = 1.f / dg;
    float          r[4], z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool is_seed = __ldg(a.seeds + c + q) == i;
      r[q] = is_seed ? 1.0f : 0.0f;
      z[q] = is_seed ? one : none;
    }
    __stcs(reinterpret_cast<float4*>(a.rank) + x, make_float4(r[0], r[1], r[2], r[3]));
    reinterpret_cast<float4*>(a.contrib0)[x] = make_float4(z[0], z[1], z[2], z[3]);
  }
}

// Start from teleport vectors: per column c < k, t = t_in[inv[i] * k + c];
// vbase = (1 - d) t, rank = t, contrib = t / s_i with s the out-weight sums
// (weighted graphs: the single weighted solve's start, per column) or the
// out-degrees (vaux null); padding columns are 0.
template <int K>
__global__ void ppr_winit_kernel(const PprArgs a, const float* __restrict__ t_in, uint32_t k,
                                 const uint32_t* __restrict__ inv, uint64_t n, float* __restrict__ vbase) {
  const uint64_t total = n * K;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const uint64_t i = x / K;
    const uint32_t c = (uint32_t)(x % K);
    const uint64_t src = inv ? inv[i] : i;
    const float    t = (c < k) ? t_in[src * k + c] : 0.f;
    vbase[x] = a.one_minus_d * t;
    a.rank[x] = t;
    a.contrib0[x] = t / (a.vaux ? a.vaux[i] : (float)a.deg[i]);
  }
}

// The streaming moves below take a matrix element per thread, K = 2^lk slots
// per row: a 64-bit division by a run-time width per element held them below
// the copy rate (RMAT scale 22, 64 columns, both moves of a narrowing: output
// 1.43 to 1.16 ms, repack 0.73 to 0.43; the start, four columns per thread,
// 0.90 to 0.53).

// out[i * k + c] = rank[perm[i] * K + c] for c < k (input order, unpadded).
template <int K>
__global__ void ppr_output_kernel(const float* __restrict__ rank, const uint32_t* __restrict__ perm, uint64_t n,
                                  uint32_t k, float* __restrict__ out) {
  const uint64_t total = n * K;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const uint64_t i = x / K;
    const uint32_t c = (uint32_t)(x % K);
    if (c < k) out[i * k + c] = __ldcs(rank + (perm ? (uint64_t)__ldg(perm + i) : i) * K + c);
  }
}

// Narrowing. The gather sums every column in the same order whatever K is (the
// tiles, the rows within a tile and the crossing rows' partials do not depend
// on it), so moving the running columns into a narrower matrix changes no
// column's values.
__global__ void ppr_repack_kernel(const float* __restrict__ src, float* __restrict__ dst, uint64_t n, uint32_t K_from,
                                  int lk_to, const uint32_t* __restrict__ map, uint32_t nact) {
  const uint64_t total = n << lk_to;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const uint64_t i = x >> lk_to;
    const uint32_t j = (uint32_t)x & ((1u << lk_to) - 1u);
    dst[x] = j < nact ? src[i * K_from + __ldg(map + j)] : 0.f;
  }
}

// One CTA of 128 threads: every slot's state is read before any is written.
__global__ void ppr_repack_cols_kernel(PprArgs a, uint32_t K_to, const uint32_t* __restrict__ map, uint32_t nact) {
  __shared__ uint32_t s_seed[128], s_done[128], s_conv[128], s_iters[128];
  __shared__ double   s_err[128];
  const uint32_t      j = threadIdx.x;
  if (j < nact) {
    const uint32_t o = map[j];
    s_seed[j] = a.seeds[o];
    s_done[j] = a.col_done[o];
    s_conv[j] = a.col_conv[o];
    s_iters[j] = a.col_iters[o];
    s_err[j] = a.col_err[o];
  }
  __syncthreads();
  if (j >= K_to) return;
  const bool live = j < nact;
  const_cast<uint32_t*>(a.seeds)[j] = live ? s_seed[j] : 0xffffffffu;
  a.col_done[j] = live ? s_done[j] : 1u;
  a.col_conv[j] = live ? s_conv[j] : 0u;
  a.col_iters[j] = live ? s_iters[j] : 0u;
  a.col_err[j] = live ? s_err[j] : 0.0;
}

__global__ void ppr_output_slots_kernel(const float* __restrict__ rank, const uint32_t* __restrict__ perm, uint64_t n,
                                        int lk, const uint32_t* __restrict__ slot_orig, uint32_t k,
                                        float* __restrict__ out) {
  const uint64_t total = n << lk;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const uint64_t i = x >> lk;
    const uint32_t j = (uint32_t)x & ((1u << lk) - 1u), c = __ldg(slot_orig + j);
    if (c < k) out[i * k + c] = __ldcs(rank + ((perm ? (uint64_t)__ldg(perm + i) : i) << lk) + j);
  }
}

// Column set-up: internal seed ids, padding columns inactive from the start.
__global__ void ppr_seed_kernel(const uint32_t* __restrict__ seeds_in, uint32_t k, int K,
                                const uint32_t* __restrict__ perm, PprArgs a) {
  const int c = threadIdx.x;
  if (c >= K) return;
  if ((uint32_t)c < k) {
    const uint32_t s = seeds_in[c];
    const_cast<uint32_t*>(a.seeds)[c] = perm ? perm[s] : s;
    a.col_done[c] = 0u;
  } else {
    const_cast<uint32_t*>(a.seeds)[c] = 0xffffffffu;
    a.col_done[c] = 1u;
  }
  a.col_conv[c] = 0u;
  a.col_iters[c] = 0u;
  a.col_err[c] = 0.0;
}

cudaError_t launch_ppr_spans(const uint32_t* row_ptr, const uint32_t* tile_row, const uint32_t* tile_nnz, uint32_t T,
                             uint32_t D, uint4* spans, unsigned int* count, int sms, cudaStream_t s) {
  if (T < 2) return cudaSuccess;
  ppr_spans_kernel<<<sms * 4, 256, 0, s>>>(row_ptr, tile_row, tile_nnz, T, D, spans, count);
  return cudaGetLastError();
}

cudaError_t launch_ppr_row_ends(const uint32_t* row_ptr, uint64_t n, uint32_t* end_bits, unsigned int* full, int sms,
                                cudaStream_t s) {
  ppr_row_ends_kernel<<<sms * 8, 256, 0, s>>>(row_ptr, n, end_bits, full);
  return cudaGetLastError();
}

cudaError_t launch_ppr_tile_full(const uint32_t* tile_row, uint32_t T, const uint32_t* rows, uint32_t num,
                                 uint32_t* tile_full, int sms, cudaStream_t s) {
  ppr_tile_full_kernel<<<sms * 4, 256, 0, s>>>(tile_row, T, rows, num, tile_full);
  return cudaGetLastError();
}

cudaError_t launch_ppr_seeds(const uint32_t* seeds_in, uint32_t k, int K, const uint32_t* perm, const PprArgs& a,
                             cudaStream_t s) {
  ppr_seed_kernel<<<1, 128, 0, s>>>(seeds_in, k, K, perm, a);
  return cudaGetLastError();
}

static int log2_of(int K) {
  int l = 0;
  while ((1 << l) < K) ++l;
  return l;
}

cudaError_t launch_ppr_repack(const float* src, float* dst, uint64_t n, int K_from, int K_to, const uint32_t* map,
                              uint32_t nact, int sms, cudaStream_t s) {
  if (K_to <= 0 || K_to > K_from || nact > (uint32_t)K_to) return cudaErrorInvalidValue;
  ppr_repack_kernel<<<sms * 8, 256, 0, s>>>(src, dst, n, (uint32_t)K_from, log2_of(K_to), map, nact);
  return cudaGetLastError();
}

cudaError_t launch_ppr_repack_cols(const PprArgs& a, int K_to, const uint32_t* map, uint32_t nact, cudaStream_t s) {
  if (K_to <= 0 || K_to > 128 || nact > (uint32_t)K_to) return cudaErrorInvalidValue;
  ppr_repack_cols_kernel<<<1, 128, 0, s>>>(a, (uint32_t)K_to, map, nact);
  return cudaGetLastError();
}

cudaError_t launch_ppr_output_slots(const float* rank, const uint32_t* perm, uint64_t n, int K, const uint32_t* slot_orig,
                                    uint32_t k, float* out, int sms, cudaStream_t s) {
  ppr_output_slots_kernel<<<sms * 8, 256, 0, s>>>(rank, perm, n, log2_of(K), slot_orig, k, out);
  return cudaGetLastError();
}

__global__ void ppr_arm_kernel(PprState* st) { st->chunk_end = st->iter + kGraphChunk; }

template <int K, int EPI>
struct PprKernels {
  static constexpr bool kW = EPI == kPprWeighted;
  // Rows per group: U * K = 512 floats, 2 KB of rows per group (16 floats per lane).
  static void* gather(bool few_tiles) {
    if constexpr (K > (kW ? 64 : 32)) return (void*)ppr_gather_warp_kernel<K, kPprTileItems, 512 / K, kW>;
    if constexpr (K == 32 && !kW)
      if (few_tiles) return (void*)ppr_gather_warp_kernel<K, kPprTileItems, 512 / K, kW>;
    if constexpr (K <= (kW ? 64 : 32)) return (void*)ppr_gather_kernel<K, kW>;
    return nullptr;
  }
  static void* fn(int which, bool few_tiles) {
    return which == 0   ? gather(few_tiles)
           : which == 1 ? (void*)ppr_fixup_kernel<K>
           : which == 2 ? (void*)ppr_epilogue_kernel<K, EPI>
                        : (void*)ppr_finish_kernel<K>;
  }
};

template <int K>
static void* ppr_fn_k(int which, int mode, bool few_tiles) {
  return mode == kPprWeighted    ? PprKernels<K, kPprWeighted>::fn(which, few_tiles)
         : mode == kPprTeleports ? PprKernels<K, kPprTeleports>::fn(which, few_tiles)
                                 : PprKernels<K, kPprSeeds>::fn(which, few_tiles);
}

// kernel 0 gather, 1 fix-up, 2 epilogue, 3 finish, for the solve's mode
static void* ppr_fn(int K, int which, int mode, bool few_tiles) {
  switch (K) {
    case 8: return ppr_fn_k<8>(which, mode, few_tiles);
    case 16: return ppr_fn_k<16>(which, mode, few_tiles);
    case 32: return ppr_fn_k<32>(which, mode, few_tiles);
    case 64: return ppr_fn_k<64>(which, mode, few_tiles);
    case 128: return ppr_fn_k<128>(which, mode, few_tiles);
    default: return nullptr;
  }
}

int ppr_mode(const PprArgs& a) { return a.w ? kPprWeighted : (a.vbase ? kPprTeleports : kPprSeeds); }

// Grid of each kernel: gather persistent at its occupancy, fix-up K/4 lanes
// per row crossing tiles, epilogue epi_grid CTAs, finish one warp per column.
static int K_of(const PprArgs& a) { return (int)a.K; }
static dim3 ppr_grid(const PprArgs& a, int which, int sweep_grid) {
  if (which == 0) return dim3((unsigned)sweep_grid);
  if (which == 1) return dim3(a.num_spans ? (unsigned)(((uint64_t)a.num_spans * (a.K / 4u) + 255u) / 256u) : 1u);
  if (which == 2) return dim3(a.epi_grid);
  return dim3((unsigned)(K_of(a) / 8));
}

bool ppr_few_tiles(uint64_t tiles, int sms) { return tiles <= (uint64_t)sms * (2 * kPprThreads / 32); }

int ppr_padded_k(uint32_t k, int mode, bool few_tiles) {
  if (few_tiles && mode != kPprWeighted && k <= 32) return 32;
  return k <= 8 ? 8 : k <= 16 ? 16 : k <= 32 ? 32 : k <= 64 ? 64 : k <= 128 ? 128 : 0;
}

int ppr_sweep_grid(int K, int mode, bool few_tiles, int sms) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ppr_fn(K, 0, mode, few_tiles), kPprThreads, 0) != cudaSuccess ||
      nb < 1)
    nb = 1;
  return sms * nb;
}

cudaError_t launch_ppr_init(const PprArgs& a, int K, uint64_t n, int sms, cudaStream_t s) {
  switch (K) {
    case 8: ppr_init_kernel<8><<<sms * 8, 256, 0, s>>>(a, n); break;
    case 16: ppr_init_kernel<16><<<sms * 8, 256, 0, s>>>(a, n); break;
    case 32: ppr_init_kernel<32><<<sms * 8, 256, 0, s>>>(a, n); break;
    case 64: ppr_init_kernel<64><<<sms * 8, 256, 0, s>>>(a, n); break;
    case 128: ppr_init_kernel<128><<<sms * 8, 256, 0, s>>>(a, n); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_ppr_winit(const PprArgs& a, int K, const float* t_in, uint32_t k, const uint32_t* inv, uint64_t n,
                             float* vbase, int sms, cudaStream_t s) {
  switch (K) {
    case 8: ppr_winit_kernel<8><<<sms * 8, 256, 0, s>>>(a, t_in, k, inv, n, vbase); break;
    case 16: ppr_winit_kernel<16><<<sms * 8, 256, 0, s>>>(a, t_in, k, inv, n, vbase); break;
    case 32: ppr_winit_kernel<32><<<sms * 8, 256, 0, s>>>(a, t_in, k, inv, n, vbase); break;
    case 64: ppr_winit_kernel<64><<<sms * 8, 256, 0, s>>>(a, t_in, k, inv, n, vbase); break;
    case 128: ppr_winit_kernel<128><<<sms * 8, 256, 0, s>>>(a, t_in, k, inv, n, vbase); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_ppr_output(const float* rank, const uint32_t* perm, uint64_t n, int K, uint32_t k, float* out,
                              int sms, cudaStream_t s) {
  switch (K) {
    case 8: ppr_output_kernel<8><<<sms * 8, 256, 0, s>>>(rank, perm, n, k, out); break;
    case 16: ppr_output_kernel<16><<<sms * 8, 256, 0, s>>>(rank, perm, n, k, out); break;
    case 32: ppr_output_kernel<32><<<sms * 8, 256, 0, s>>>(rank, perm, n, k, out); break;
    case 64: ppr_output_kernel<64><<<sms * 8, 256, 0, s>>>(rank, perm, n, k, out); break;
    case 128: ppr_output_kernel<128><<<sms * 8, 256, 0, s>>>(rank, perm, n, k, out); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_ppr_sweep(const PprArgs& a, int K, int sweep_grid, cudaStream_t s) {
  void* args[] = {(void*)&a};
  for (int w = 0; w < 4; ++w) {
    uint64_t    n = a.n;
    void*       eargs[] = {(void*)&a, (void*)&n};
    cudaError_t e = cudaLaunchKernel(ppr_fn(K, w, ppr_mode(a), a.few_tiles != 0), ppr_grid(a, w, sweep_grid), dim3(256),
                                     w == 2 ? eargs : args, 0, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t build_ppr_graph(cudaGraph_t g, const PprArgs& proto, int K, int sweep_grid, PprState* st,
                            cudaGraphExec_t* exec) {
  cudaGraphNode_t      arm;
  cudaKernelNodeParams kp = {};
  void*                sargs[] = {(void*)&st};
  kp.func = (void*)ppr_arm_kernel;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(1);
  kp.kernelParams = sargs;
  cudaError_t e = cudaGraphAddKernelNode(&arm, g, nullptr, 0, &kp);
  if (e != cudaSuccess) return e;
  cudaGraphConditionalHandle cond;
  if ((e = cudaGraphConditionalHandleCreate(&cond, g, 1u, cudaGraphCondAssignDefault)) != cudaSuccess) return e;
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = cond;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t wnode;
  if ((e = cudaGraphAddNode(&wnode, g, &arm, 1, &cp)) != cudaSuccess) return e;
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  PprArgs     a = proto;
  a.cond = cond;
  a.use_cond = 1;
  uint64_t             n = a.n;
  void*                args[] = {(void*)&a};
  void*                eargs[] = {(void*)&a, (void*)&n};
  cudaGraphNode_t      prev = nullptr;
  for (int i = 0; i < 4 * kPprLoopSweeps; ++i) {
    const int            w = i % 4;
    cudaKernelNodeParams kp2 = {};
    kp2.func = ppr_fn(K, w, ppr_mode(a), a.few_tiles != 0);
    kp2.gridDim = ppr_grid(a, w, sweep_grid);
    kp2.blockDim = dim3(256);
    kp2.kernelParams = w == 2 ? eargs : args;
    cudaGraphNode_t node;
    if ((e = cudaGraphAddKernelNode(&node, body, prev ? &prev : nullptr, prev ? 1 : 0, &kp2)) != cudaSuccess) return e;
    prev = node;
  }
  return cudaGraphInstantiate(exec, g, 0);
}

}  // namespace nwgpu
