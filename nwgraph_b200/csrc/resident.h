// Internal interface of the resident solve (pr_resident.cu).
#pragma once

#include "binned.h"

namespace nwgpu {

// Launch plan of the resident solve of one graph: its rows cut into one
// contiguous range per CTA, everything a CTA needs of them in shared memory.
struct ResidentPlan {
  bool      tried = false;       // looked at (the first solve does)
  bool      ok = false;          // the graph is small enough
  int       ctas = 0;
  uint32_t  hub_ids = 0;         // contrib[0, hub_ids) is staged in shared memory every sweep
  uint32_t  smem_bytes = 0;
  uint32_t* bounds = nullptr;    // ctas + 1 row bounds
  unsigned int* sync = nullptr;  // two arrival counters, used by turns
  unsigned int  turn = 0;
  double*   part = nullptr;      // 2 x (ctas + 1): residual partials and the abort word, by sweep parity
  void      release(cudaStream_t s);
};

struct ResidentArgs {
  const uint32_t* row_ptr;
  const uint32_t* col;
  const uint32_t* inv;       // internal id -> input id
  const uint32_t* deg;       // out-degrees, input order
  float*          out;       // ranks, input order
  float*          rank;      // internal order: ranks of a solve that goes on in another launch
  float*          contrib0;  // ping-pong by sweep parity
  float*          contrib1;
  const uint32_t* bounds;
  unsigned int*   sync;
  unsigned int    turn;
  unsigned int    polls;     // the self-test's, whose barriers wait for one CTA too many and give up after so many; else 0
  double*         part;
  PrState*        state;     // host-mapped: written once, at the end
  unsigned long long* sweeps_ns;  // beside it: from the first sweep's start to the last one's residual
  double*         err_hist;
  uint32_t        err_cap;
  const volatile unsigned int* abort_word;
  unsigned long long iter0;  // sweeps done by earlier launches (0: start from init)
  unsigned long long max_iters;
  unsigned long long chunk_end;
  double          threshold;
  float           damping;
  float           base;
  float           init;
  int             teleport;  // TeleportMode
  uint32_t        seed;      // input id of the one-hot teleport vertex
  uint32_t        long_row, chunk, bin0_rows, num_long_rows;
  uint32_t        bin_row_begin[kNumBins];
  uint32_t        bin_row_end[kNumBins];
  uint32_t        hub_ids;
};

constexpr unsigned int kBarrierPolls = 1u << 22;  // about 3 s: then the solve ends with an error
constexpr unsigned int kFaultResidentWait = 0x52455349u;  // PrState::fault: a grid barrier gave up

// Largest entry count the resident solve is considered for.
constexpr uint64_t kResidentMaxEntries = 8ull << 20;
// What the fullest CTA may gather past the hubs per sweep (plan_resident has the measurements): of any graph, in
// sectors; of one with long rows and no CTA above kResidentUneven times the average, in gathers.
constexpr uint32_t kResidentSectors = 17000;
constexpr uint32_t kResidentSkewedGathers = 33000;
constexpr double   kResidentUneven = 2.5;

cudaError_t configure_resident_kernel();
// Row bounds of `ctas` ranges of about equal work into bounds[0..ctas]; what the host sizes the plan by into
// out: the bounds, row_ptr at them, then row_ptr[min(n, kResidentHubStep (i + 1))].
constexpr uint32_t kNumResidentHubs = 8, kResidentHubStep = 6144;
cudaError_t launch_resident_bounds(const uint32_t* row_ptr, uint64_t n, uint64_t nnz, int ctas, uint32_t* bounds,
                                   uint32_t* out, cudaStream_t s);
// counts[0], counts[1] (zeroed) += among the `entries` entries at col, the gathers past the first hub_ids
// contributions and, per 1024 consecutive entries, the distinct 32-byte sectors they fall in.
cudaError_t launch_resident_gathers(const uint32_t* col, uint32_t entries, uint32_t hub_ids, uint32_t* counts, cudaStream_t s);
int      resident_ctas(uint64_t n, uint64_t nnz, int sms);
uint64_t resident_words(uint64_t E, uint64_t R);
uint32_t resident_smem_limit();
cudaError_t launch_resident(const ResidentArgs& a, int ctas, uint32_t smem_bytes, cudaStream_t s);

}  // namespace nwgpu
