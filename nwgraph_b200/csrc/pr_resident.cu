// Resident PageRank solve of small graphs: one cooperative launch runs every
// sweep, with each CTA's rows in its SM's shared memory.
//
// A sweep of the binned kernel takes a small graph as long as its chains of
// dependent loads (a row of 2048 entries is 16 steps of one half-warp, each
// waiting for its ids; every bin refills row_ptr -> id -> contribution), plus
// a finishing kernel and the gaps of the while loop. Here a CTA owns a
// contiguous range of rows and a sweep is
//   stage   the hubs' contributions into shared memory,
//   gather  the range's entries in CSR order, every thread on its own, all
//           loads independent, values to shared memory,
//   sum     the rows from there, in the binned sweep's order (chunks of long
//           rows, half-warps, groups of G lanes), update, next contributions,
//   barrier over the grid; every CTA then adds up all CTAs' residuals itself
//           and comes to the same stopping decision, while the next sweep's
//           hubs are loading.
// A row's entries, ranks, degrees and offsets stay in shared memory and the
// first eight column ids of a thread in registers, so a sweep reads only the
// contributions (and the ids past those eight). Row sums take the binned
// sweep's order exactly: ranks are bitwise equal to its.
//
// Bound on the smallest graphs by the latencies of a sweep's phases (1024
// entries on one CTA or 20,000 on twelve: about 2500 cycles until the residual
// is known, 1400 to gather, 3000 to sum, 750 to reduce, 1600 in the barrier),
// on the largest by the gathers past the hubs (one L2 request per SM and
// clock). Per sweep, against the binned sweep, its finishing kernel and the
// loop: RMAT scale 10 5.1 to 21 us, scale 13 5.8 to 27, scale 16 10.9 to 43,
// scale 17 16.8 to 38; 1M-vertex grid 13.7 to 24. A whole solve adds 10 to 20 us
// of start and end (the loop's launches, copies and host waits took 50).
// Barrier words that carry the residuals (each CTA polls all CTAs' 16-byte
// packets) took 6000 cycles and more with 148 CTAs, the counter 1800.
#include "common.cuh"
#include "resident.h"

namespace nwgpu {

constexpr int      kResidentThreads = 1024;
constexpr uint32_t kWarps = kResidentThreads / 32;
constexpr int      kIdRegs = 8;               // column ids a thread keeps
constexpr uint32_t kRowCost = 3;              // a row's update, in entries
constexpr uint32_t kItemsPerCta = 2048;       // at least this much work per CTA

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Place of the CTA's entry e in s_val: one spare word per 32, so that lanes
// reading every fourth entry hit 32 banks.
__device__ __forceinline__ uint32_t skew(uint32_t e) { return e + (e >> 5); }

// Sum of the entries [start, end) over LANES lanes in windows of 8 LANES
// entries: a lane adds 4 consecutive entries of each half of a window
// (window_entry of the binned sweep), window after window.
template <uint32_t LANES>
__device__ __forceinline__ float lane_sum(const float* s_val, uint32_t start, uint32_t end, uint32_t lanei) {
  constexpr uint32_t L = 8u * LANES;
  float              acc = 0.f;
  uint32_t           base = start + 4u * lanei;
#pragma unroll 2
  for (uint32_t left = end - start; left >= L; left -= L, base += L) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = s_val[skew(base + (L / 2u) * (uint32_t)(q >> 2) + (uint32_t)(q & 3))];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc += v[q];
  }
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t e = base + (L / 2u) * (uint32_t)(q >> 2) + (uint32_t)(q & 3);
    v[q] = e < end ? s_val[skew(e)] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) acc += v[q];
  return acc;
}

struct ResidentRows {
  const uint32_t* s_row;  // local entry offsets of the CTA's rows
  float*          s_rank;
  const uint32_t* s_deg;
  const float*    s_val;
  float* __restrict__ cout;
  uint32_t first;         // the CTA's first row
  uint32_t seed;          // internal id of the teleport vertex
};

__device__ __forceinline__ double resident_update(const ResidentArgs& a, const ResidentRows& x, uint32_t r, float z) {
  const uint32_t i = r - x.first;
  const float    base = (a.teleport == kTeleportSeed && r != x.seed) ? 0.f : a.base;
  const float    old = x.s_rank[i], nr = fmaf(a.damping, z, base);
  x.s_rank[i] = nr;
  x.cout[r] = nr / (float)x.s_deg[i];
  return (double)fabsf(nr - old);
}

// Rows [lo, hi) of a G-bin: G = 2^lg lanes per row, at most 4 entries per lane. One
// body for every G: the sums' code, run once per sweep, should stay short.
__device__ __forceinline__ double group_rows(const ResidentArgs& a, const ResidentRows& x, uint32_t lo, uint32_t hi, uint32_t lg,
                                             uint32_t w, uint32_t lane) {
  const uint32_t G = 1u << lg, per = 32u >> lg, sub = lane & (G - 1u);
  double         res = 0.0;
  for (uint32_t r0 = lo + w * per; r0 < hi; r0 += per * kWarps) {
    const uint32_t r = r0 + (lane >> lg);
    float          acc = 0.f;
    if (r < hi) {
      const uint32_t s0 = x.s_row[r - x.first], len = x.s_row[r - x.first + 1] - s0;
      float          v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t o = sub + ((uint32_t)q << lg);
        v[q] = (o < len) ? x.s_val[skew(s0 + o)] : 0.f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) acc += v[q];
    }
    for (uint32_t off = G / 2u; off > 0u; off >>= 1) acc += __shfl_xor_sync(kFullMask, acc, off);
    if (r < hi && sub == 0u) res += resident_update(a, x, r, acc);
  }
  return res;
}

// MISSING: CTAs that the grid barriers wait for beside those there are (0; 1 in
// the self-test, with its poll limit). A limit and a count at run time changed
// the code of every phase: a sweep 10.8 to 11.7 us at RMAT scale 16, 13.1 to
// 15.1 on the 1M-vertex grid.
template <unsigned MISSING>
__global__ void __launch_bounds__(kResidentThreads, 1) pr_resident_kernel(const ResidentArgs a) {
  extern __shared__ float4 smem4[];
  __shared__ double        s_red[kResidentThreads / 32];
  __shared__ uint32_t      s_seed, s_bins;
  __shared__ uint32_t      s_bin[kNumBins][3];  // the bins the CTA has rows of: bin, first row, end
  __shared__ int           s_done, s_fault;
  __shared__ unsigned long long s_start;
  const int                tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t           cta = blockIdx.x, ctas = gridDim.x;
  const uint32_t           ra = a.bounds[cta], rb = a.bounds[cta + 1], R = rb - ra;
  const uint32_t           ea = a.row_ptr[ra], E = a.row_ptr[rb] - ea;
  // hub | val | row offsets | ranks | degrees | chunk partials (resident_words)
  float*    s_hub = reinterpret_cast<float*>(smem4);
  float*    s_val = s_hub + a.hub_ids;
  uint32_t* s_row = reinterpret_cast<uint32_t*>(s_val + skew(E) + 1u);
  float*    s_rank = reinterpret_cast<float*>(s_row + R + 1u);
  uint32_t* s_deg = reinterpret_cast<uint32_t*>(s_rank + R);
  float*    s_part = reinterpret_cast<float*>(s_deg + R);

  if (tid == 0) {
    s_seed = 0xffffffffu;
    s_done = a.iter0 >= a.max_iters;
    s_fault = 0;
    uint32_t k = 0;
    for (int b = 0; b < kNumBins; ++b) {
      const uint32_t lo = max(ra, a.bin_row_begin[b]), hi = min(rb, a.bin_row_end[b]);
      if (lo >= hi) continue;
      s_bin[k][0] = (uint32_t)b;
      s_bin[k][1] = lo;
      s_bin[k][2] = hi;
      ++k;
    }
    s_bins = k;
  }
  __syncthreads();
  for (uint32_t i = tid; i <= R; i += kResidentThreads) s_row[i] = a.row_ptr[ra + i] - ea;
  for (uint32_t i = tid; i < R; i += kResidentThreads) {
    const uint32_t in = a.inv[ra + i], dg = a.deg[in];
    const bool     is_seed = a.teleport == kTeleportSeed && in == a.seed;
    if (is_seed) s_seed = ra + i;
    s_deg[i] = dg;
    const float r = a.iter0 ? a.rank[ra + i] : a.teleport == kTeleportSeed ? (is_seed ? 1.0f : 0.0f) : a.init;
    s_rank[i] = r;
    if (a.iter0 == 0) a.contrib0[ra + i] = r / (float)dg;
  }
  uint32_t id[kIdRegs];
#pragma unroll
  for (int j = 0; j < kIdRegs; ++j) {
    const uint32_t e = (uint32_t)tid + (uint32_t)j * kResidentThreads;
    id[j] = e < E ? __ldg(a.col + ea + e) : 0u;
  }
  if (cta == 0 && tid == 0) a.sync[a.turn ^ 1u] = 0u;  // for the next launch
  unsigned int target = 0;
  // All CTAs' writes before it are seen by all CTAs after it. False once a wait gave up.
  auto barrier = [&]() {
    __syncthreads();
    target += ctas + MISSING;
    if (tid == 0 && ctas + MISSING > 1u) {
      __threadfence();
      atomicAdd(a.sync + a.turn, 1u);
      unsigned polls = 0;
      while (ld_acquire(a.sync + a.turn) < target)
        if (++polls == (MISSING ? a.polls : kBarrierPolls)) {
          s_fault = 1;
          break;
        }
    }
    __syncthreads();
    return s_fault == 0;
  };
  bool ok = barrier();
  if (cta == 0 && tid == 0) s_start = clock_ns();

  unsigned long long it = a.iter0;
  while (ok) {
    const float* cin = (it & 1ull) ? a.contrib1 : a.contrib0;
    // the hubs load while the last sweep's residual is added up (not needed if that ends the solve)
    for (uint32_t i = tid; i < a.hub_ids / 4u; i += kResidentThreads)
      reinterpret_cast<float4*>(s_hub)[i] = __ldcg(reinterpret_cast<const float4*>(cin) + i);
    if (it != a.iter0 && warp == 0) {
      const double* part = a.part + ((it - 1ull) & 1ull) * (ctas + 1u);
      double        e = 0.0;
      for (uint32_t u = lane; u < ctas; u += 32u) e += __ldcg(part + u);
      const bool abort_seen = __ldcg(part + ctas) != 0.0;
      e = warp_sum_lane0(e);
      if (lane == 0) {
        const bool conv = e < a.threshold;
        s_done = conv || it >= a.max_iters || abort_seen;
        if (cta == 0) {
          if (a.err_hist && it - 1ull < a.err_cap) a.err_hist[it - 1ull] = e;
          if (s_done || it == a.chunk_end) {
            a.state->iter = it;
            a.state->last_error = e;
            a.state->converged = conv ? 1u : 0u;
            a.state->aborted = (abort_seen && !conv) ? 1u : 0u;
            a.state->done = s_done ? 1u : 0u;
            *a.sweeps_ns = clock_ns() - s_start;
          }
        }
      }
    }
    __syncthreads();
    if (s_done || it == a.chunk_end) break;

    // gather: independent loads, CSR order. Plain cached loads are coherent here: the barrier's acquire drops the
    // SM's L1 lines; between barriers a mesh's rows find their neighbours' values in L1 (13.7 us a sweep of the
    // 1M-vertex grid, 14.3 through L2).
    unsigned int abort_word = 0u;
    if (cta == 0 && tid == kResidentThreads - 1) abort_word = *a.abort_word;
    auto gather = [&](uint32_t e0, const uint32_t(&from)[kIdRegs]) {
      float v[kIdRegs];
#pragma unroll
      for (int j = 0; j < kIdRegs; ++j) {
        v[j] = 0.f;
        if (e0 + (uint32_t)j * kResidentThreads < E) v[j] = from[j] < a.hub_ids ? s_hub[from[j]] : __ldca(cin + from[j]);
      }
#pragma unroll
      for (int j = 0; j < kIdRegs; ++j)
        if (e0 + (uint32_t)j * kResidentThreads < E) s_val[skew(e0 + (uint32_t)j * kResidentThreads)] = v[j];
    };
    gather((uint32_t)tid, id);
#pragma unroll 1
    for (uint32_t e0 = (uint32_t)tid + kIdRegs * kResidentThreads; e0 < E; e0 += kIdRegs * kResidentThreads) {
      uint32_t more[kIdRegs];
#pragma unroll
      for (int j = 0; j < kIdRegs; ++j) {
        const uint32_t e = e0 + (uint32_t)j * kResidentThreads;
        more[j] = e < E ? __ldg(a.col + ea + e) : 0u;
      }
      gather(e0, more);
    }
    __syncthreads();

    // sums and updates
    const ResidentRows x{s_row, s_rank, s_deg, s_val, (it & 1ull) ? a.contrib0 : a.contrib1, ra, s_seed};
    double             res = 0.0;
    const uint32_t     long_end = min(rb, a.num_long_rows);
    uint32_t           unit = 0;  // warp units handed out so far: bins of few rows go to different warps
    if (ra < long_end) {
      // chunks of the long rows, a warp each, then the rows
      for (uint32_t r = ra; r < long_end; ++r) {
        const uint32_t s0 = s_row[r - ra], s1 = s_row[r - ra + 1];
        for (uint32_t k = s0; k < s1; k += a.chunk, ++unit) {
          if (unit % kWarps != (uint32_t)warp) continue;
          const float z = warp_sum_lane0(lane_sum<32>(s_val, k, min(s1, k + a.chunk), (uint32_t)lane));
          if (lane == 0) s_part[unit] = z;
        }
      }
      __syncthreads();
      unit = 0;
      for (uint32_t r = ra; r < long_end; ++r) {
        const uint32_t len = s_row[r - ra + 1] - s_row[r - ra], chunks = (len + a.chunk - 1u) / a.chunk;
        if ((r - ra) % kWarps == (uint32_t)warp) {
          float p = 0.f;
          if (len > 32u * a.chunk) {
            for (uint32_t c = lane; c < chunks; c += 32u) p += s_part[unit + c];
            p = warp_sum_lane0(p);
          } else {
            for (uint32_t c = 0; c < chunks; ++c) p += s_part[unit + c];
          }
          if (lane == 0) res += resident_update(a, x, r, p);
        }
        unit += chunks;
      }
      unit = long_end - ra;
    }
    for (uint32_t k = 0; k < s_bins; ++k) {
      const uint32_t b = s_bin[k][0], lo = s_bin[k][1], hi = s_bin[k][2];
      const uint32_t w = ((uint32_t)warp + kWarps - unit % kWarps) % kWarps;
      if (b == 0u) {
        if (a.bin0_rows == 1u) {
          for (uint32_t r = lo + w; r < hi; r += kWarps) {
            const float z = warp_sum_lane0(lane_sum<32>(s_val, s_row[r - ra], s_row[r - ra + 1], (uint32_t)lane));
            if (lane == 0) res += resident_update(a, x, r, z);
          }
        } else {
          const unsigned half = (lane & 16) ? 0xffff0000u : 0x0000ffffu;
          for (uint32_t r = lo + 2u * w + ((uint32_t)lane >> 4); r < hi; r += 2u * kWarps) {
            float z = lane_sum<16>(s_val, s_row[r - ra], s_row[r - ra + 1], (uint32_t)lane & 15u);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) z += __shfl_xor_sync(half, z, off);
            if ((lane & 15) == 0) res += resident_update(a, x, r, z);
          }
        }
        __syncwarp();
      } else if (b == kNumBins - 1) {
        for (uint32_t r = lo + 32u * w + (uint32_t)lane; r < hi; r += kResidentThreads) res += resident_update(a, x, r, 0.f);
        __syncwarp();
      } else {
        res += group_rows(a, x, lo, hi, 6u - b, w, (uint32_t)lane);
      }
      unit += b == 0u ? (hi - lo + 1u) / 2u : b == kNumBins - 1 ? (hi - lo + 31u) / 32u : ((hi - lo - 1u) >> (b - 1u)) + 1u;
    }
    res = warp_sum_lane0(res);
    if (lane == 0) s_red[warp] = res;
    double* part = a.part + (it & 1ull) * (ctas + 1u);
    if (cta == 0 && tid == kResidentThreads - 1) part[ctas] = abort_word ? 1.0 : 0.0;
    __syncthreads();
    if (warp == 0) {
      const double s = warp_sum_lane0(s_red[lane]);
      if (lane == 0) part[cta] = s;
    }
    ok = barrier();
    ++it;
  }
  if (!ok) {
    if (tid == 0) {
      a.state->fault = kFaultResidentWait;
      a.state->done = 1u;
    }
    return;
  }
  float* const keep = s_done ? a.out : a.rank;
  for (uint32_t i = tid; i < R; i += kResidentThreads) keep[s_done ? a.inv[ra + i] : ra + i] = s_rank[i];
  if (it == a.iter0 && cta == 0 && tid == 0) {  // no sweep was asked for
    a.state->iter = it;
    a.state->done = 1u;
  }
}

__global__ void resident_bounds_kernel(const uint32_t* __restrict__ row_ptr, uint32_t n, uint32_t nnz, uint32_t ctas,
                                       uint32_t* __restrict__ bounds, uint32_t* __restrict__ out) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c <= ctas) {
    const uint64_t want = ((uint64_t)nnz + (uint64_t)kRowCost * n) * c / ctas;
    uint32_t       lo = 0, hi = n;
    while (lo < hi) {  // first row that starts at or after the work before this range
      const uint32_t mid = (lo + hi) >> 1;
      if ((uint64_t)row_ptr[mid] + (uint64_t)kRowCost * mid < want)
        lo = mid + 1;
      else
        hi = mid;
    }
    bounds[c] = lo;
    out[c] = lo;
    out[ctas + 1u + c] = row_ptr[lo];
  } else if (c <= ctas + kNumResidentHubs) {
    const uint32_t i = c - ctas - 1u;
    out[2u * (ctas + 1u) + i] = row_ptr[min(n, kResidentHubStep * (i + 1u))];
  }
}

// A thread per entry; the sectors' numbers go into a hash set (at most 1024 of them in 4096 places, so every probe ends).
__global__ void __launch_bounds__(1024) resident_gathers_kernel(const uint32_t* __restrict__ col, uint32_t entries,
                                                                uint32_t hub_ids, uint32_t* __restrict__ counts) {
  constexpr uint32_t  kPlaces = 4096, kNone = 0xffffffffu;
  __shared__ uint32_t s_set[kPlaces];
  for (uint32_t i = threadIdx.x; i < kPlaces; i += 1024u) s_set[i] = kNone;
  __syncthreads();
  const uint32_t e = blockIdx.x * 1024u + threadIdx.x, id = e < entries ? col[e] : 0u;
  const bool     past = e < entries && id >= hub_ids;
  bool           is_new = false;
  if (past) {
    const uint32_t sector = id >> 3;
    for (uint32_t at = (sector * 2654435761u) >> 20;; at = (at + 1u) % kPlaces) {
      const uint32_t was = atomicCAS(s_set + at, kNone, sector);
      is_new = was == kNone;
      if (is_new || was == sector) break;
    }
  }
  const int gathers = __syncthreads_count(past), sectors = __syncthreads_count(is_new);
  if (threadIdx.x == 0) {
    atomicAdd(counts, (uint32_t)gathers);
    atomicAdd(counts + 1, (uint32_t)sectors);
  }
}

cudaError_t launch_resident_gathers(const uint32_t* col, uint32_t entries, uint32_t hub_ids, uint32_t* counts, cudaStream_t s) {
  resident_gathers_kernel<<<(entries + 1023u) / 1024u, 1024, 0, s>>>(col, entries, hub_ids, counts);
  return cudaGetLastError();
}

cudaError_t launch_resident_bounds(const uint32_t* row_ptr, uint64_t n, uint64_t nnz, int ctas, uint32_t* bounds,
                                   uint32_t* out, cudaStream_t s) {
  const unsigned threads = (unsigned)ctas + 1u + kNumResidentHubs;
  resident_bounds_kernel<<<(threads + 127u) / 128u, 128, 0, s>>>(row_ptr, (uint32_t)n, (uint32_t)nnz, (uint32_t)ctas, bounds, out);
  return cudaGetLastError();
}

int resident_ctas(uint64_t n, uint64_t nnz, int sms) {
  const uint64_t want = (nnz + kRowCost * n + kItemsPerCta - 1) / kItemsPerCta;
  return want < 1 ? 1 : want < (uint64_t)sms ? (int)want : sms;
}

// Words of shared memory of a CTA with E entries and R rows beside its hubs.
// Chunk partials: a long row of len entries has at most len / 256 + 1 chunks,
// and a CTA at most E / 256 long rows.
uint64_t resident_words(uint64_t E, uint64_t R) { return E + E / 32u + 1u + 3u * R + 1u + E / 128u + 4u; }

uint32_t resident_smem_limit() { return binned_hot_capacity() * 4u; }

cudaError_t configure_resident_kernel() {
  for (void* fn : {(void*)pr_resident_kernel<0>, (void*)pr_resident_kernel<1>}) {
    const cudaError_t e =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)resident_smem_limit());
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_resident(const ResidentArgs& a, int ctas, uint32_t smem_bytes, cudaStream_t s) {
  void* args[] = {(void*)&a};
  void* fn = a.polls ? (void*)pr_resident_kernel<1> : (void*)pr_resident_kernel<0>;
  return cudaLaunchCooperativeKernel(fn, dim3((unsigned)ctas), dim3(kResidentThreads), args, smem_bytes, s);
}

}  // namespace nwgpu
