// pps_tensor.cuh -- the tensor walk: plan, arguments and launcher shared by the
// one-job and batched host code.  The kernel is in pps_tensor.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pps_internal.h"

namespace pps {

constexpr uint32_t TW_ROWS = 128;    // MMA rows: giant steps of one unit
constexpr uint32_t TW_MAX_NB = 512;  // columns (baby steps) of one unit, at most

// How one job runs on the tensor walk (tensor_plan).
struct TensorPlan {
  uint32_t s;       // n per test
  uint32_t nb;      // columns: tests per row, a multiple of 16
  uint32_t units;   // units of 128 x nb tests per prime
  uint32_t digits;  // bits per digit: 4 (p < 2^47) or 5 (p < 2^62)
  uint32_t pitch;   // words of a prime's expansion in shared memory (odd)
  uint32_t off;     // offset of the tested fraction, and the test's bound, in 2^-16
  uint32_t thr;
  double cost;      // estimated SM clocks per prime
};

// Whether the tensor walk can run the job at all, and how.
bool tensor_plan(const pps_job_params* jp, TensorPlan* out);

// Where the candidates go, and the idx of prime i's: idx_base + i idx_step
// (a twin candidate of the +1 side: and bit 31).
struct TensorHits {
  pps_hit* hits;
  uint32_t* hit_count;
  uint32_t hit_cap;
  uint32_t idx_base, idx_step;
};

struct TensorArgs {
  const uint64_t* P;
  const uint64_t* Pinv;  // or null: computed
  uint64_t np;
  const uint64_t* list;  // a caller's list, whose primes may lie outside [pmin, pmax)
  uint64_t listed;       // its length (0: the primes are known to lie inside)
  uint64_t pmin, pmax, kmin, kmax;
  uint32_t nmin, nmax;
  uint32_t side;         // 1: K = -2^-n (Proth), 0: K = 2^-n (Riesel), 2: both (twin)
  TensorPlan plan;
  uint32_t batch;        // units a CTA takes at a time (1..32)
  uint32_t* work;        // zeroed before a call's first launch
                         // [0] batches taken (the re-check zeroes it again)
                         // [1] set when a prime outside [pmin, pmax) was met: nothing more is walked
                         // [2] set when a launch failed: TW_TIMED_OUT, TW_BAD_TMEM
  long long wait_limit;  // clocks that a wait may take
  uint32_t stall_at;     // batch of each CTA before which the seeds stop (pps_debug_tensor_stall; ~0: none)
  uint4* masks;          // which rows pass: of each unit, tile and 32 rows a bit per row for columns 0-31,
                         // 32-63, 64-95 and 96-111 of the tile
  uint32_t mask_cap;     // masks that there is room for: more primes are walked in parts
  TensorHits to;
};

constexpr uint32_t TW_TIMED_OUT = 1u;  // a bounded wait ran out
constexpr uint32_t TW_BAD_TMEM = 2u;   // tensor memory did not start at 0
constexpr long long TW_WAIT_LIMIT = 8000000000ll;  // clocks: about 4 s
constexpr uint64_t TW_SCAN = 16384;    // of a list: 16 primes a thread of each block
constexpr double TW_LEAST_COST = 635.0;      // of one unit (TensorPlan::cost)
constexpr uint32_t TW_MAX_MASKS = 1u << 24;  // 268 MB; their numbers have 25 bits in k_tensor_check

// Masks for np primes, or for one part of them.
size_t tensor_masks(const TensorPlan& plan, uint64_t np);
// Once for a device, before its first walk: lets the kernels have all the shared
// memory that a plan may ask for.  (The setting is the device's and not a
// launch's: set to each job's size, one thread's smaller job would make another's
// launches fail.)
cudaError_t tensor_setup();
// The walk and the re-check of np primes, in parts of mask_cap masks.  *launches += the kernels launched.
cudaError_t launch_tensor_walk(TensorArgs a, int num_sms, cudaStream_t st, uint64_t* launches);

}  // namespace pps

// (pps_engine.cu) Whether the engine takes it for np primes of the job (0: as many as fill the GPU); *saved:
// SM clocks per prime by the estimates.
bool tensor_choice(const pps_engine* e, const pps_job_params* jp, double np, pps::TensorPlan* plan,
                   double* saved = nullptr);
// Room for its masks (for a part of np primes at least), or an error.
int ensure_masks(pps_engine* e, const pps::TensorPlan& plan, uint64_t np);
int run_tensor_walk(pps_engine* e, const pps_job_params* jp, const pps::TensorPlan& plan, const uint64_t* dP,
                    const uint64_t* dPinv, uint64_t np, const pps::TensorHits& to, bool caller_list = false);
// The status words in the pinned copy of the counters: an error if a wait ran
// out, *outside if a prime was outside the job's range.
int tensor_status(const pps_engine* e, bool* outside);
