// Device-side description of one case of an ensemble stepped in lockstep.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "kernels.h"

namespace imx {

struct BatchCase {
  DevGrid g;
  CoefR<float> c;
  const uint8_t* mask;
  const double* inlet;
  void* fb[2];          // population buffers of the case
  const void* fill;     // its boundary fill list (DevFill32 if fill_narrow)
  int64_t n_fill;
  int fill_narrow;
  int parity0;          // buffer holding the post-BC state when the call starts
  int nsteps;           // iterations this case takes in the call
  int pad;
};

// One case as the lockstep step kernel takes it, by value with the launch (the
// constant bank), so that a block goes from its index to its cells without a
// load from memory.
struct BatchNode {
  void* fb[2];
  const uint8_t* mask;
  const double* inlet;
  const uint32_t* bnd;   // DevState's fused boundary plan (null: the fill
  const uint32_t* bnd_at;  // kernel keeps the case's boundary slots)
  const DevFill32* push;
  int64_t N, dy, dz, pshift;
  uint32_t id_lo, id_hi;
  CoefR<float> k;
  int case_id;
};
// Cases of one launch: up to kBatchPart, whose BatchNodes are 28 of the 32 KB that a
// launch's parameters may take. A part of no more than kBatchFew has them in 4 KB:
// a launch is as fast either way (24 cylinder cases of 256 to 1024 nodes along x 12.55
// and 12.46 ms per 300 iterations), but a captured run keeps a copy for each of them
// (100 such cases: 113 and 27 MB on the device, 16.3 and 9.2 ms for a first 40 iterations).
constexpr int kBatchFew = 16, kBatchPart = 128;
template <int CAP>
struct BatchArgs {
  int n;
  uint32_t first[CAP + 1];  // first block of each case; the total
  BatchNode c[CAP];
};

// The parts of a batch, by chain: plan[chain][part] lists its cases. A part
// holds at most `cap` cases and at most `room` bytes of populations (a larger
// case is a part of its own).
typedef std::vector<std::vector<std::vector<int>>> BatchPlan;
constexpr int kBatchChains = 2;
BatchPlan plan_batch(const std::vector<int64_t>& bytes, int64_t room, int cap, int chains);

// What one block of the boundary refresh works on: 256 entries of a case's
// fill list.
struct BatchBlock {
  uint32_t item, case_id;
};

// Step-kernel launch shapes the autotuner chooses from: threads per block and
// lattice nodes per thread.
struct BatchShape {
  int block, cpt;
};
constexpr int kNumBatchShapes = 6;
extern const BatchShape kBatchShapes[kNumBatchShapes];

// Iteration *counter + k of the cases of `a` whose budget it is below
// (cases: all cases of the batch, by case_id), and the boundary refresh of
// `fills`.
template <int CAP>
cudaError_t launch_batch_iteration(int dim, int store, int shape, const BatchArgs<CAP>& a,
                                   const BatchCase* cases, const BatchBlock* fills, int64_t nfills,
                                   const int* counter, int k, cudaStream_t s);
// Load the step kernel of a shape now (a kernel is otherwise loaded at its
// first launch, which a timed launch would include).
template <int CAP>
cudaError_t load_batch_kernel(int dim, int store, int shape);
// *counter += n.
cudaError_t launch_batch_tick(int* counter, int n, cudaStream_t s);

// ---- Persistent stepping (batch_persist.cu): one cooperative launch per
// call; work items are step tiles and fill chunks of each case's iterations.
constexpr int kPersistCPT = 4;                   // cells per thread of a step tile
constexpr int kPersistTile = 256 * kPersistCPT;  // cells per step tile
constexpr int kPersistFillChunk = 1024;          // fill entries per chunk
constexpr int kPersistTimeout = 1;               // status: a wait ran out of budget

struct PersistSched {
  const BatchCase* cases;
  const int* order;             // cases by descending iteration budget
  const long long* tile_pre;    // [ncases + 1] prefix sums of step tiles in `order`
  const long long* fill_pre;    // [ncases + 1] prefix sums of fill chunks in `order`
  const long long* iter_start;  // [niters + 1] first item of each iteration
  const int* active;            // [niters] cases still running at each iteration
  long long nitems;
  int ncases;
  unsigned long long* next;     // work counter (zero at launch)
  unsigned* done_step;          // per case: step tiles finished in this call
  unsigned* done_fill;          // per case: fill chunks finished in this call
  int* status;                  // 0, or kPersistTimeout
  int* info;                    // case, iteration, kind (0 step, 1 fill) of the wait that gave up
  unsigned long long budget_ns; // bound of every wait (device global timer)
  int stall_case;               // testing: this case's step tiles after its first iteration
                                // wait for a count nothing reaches (-1: none)
};

// Resident blocks of the persistent kernel for this device (SMs x blocks per
// SM) for a batch of ncases cases, and its dynamic shared memory.
cudaError_t persistent_grid(int dim, int store, int ncases, int* blocks);
size_t persistent_smem(int ncases);
cudaError_t launch_batch_persistent(int dim, int store, int blocks, const PersistSched& s,
                                    cudaStream_t st);

}  // namespace imx
