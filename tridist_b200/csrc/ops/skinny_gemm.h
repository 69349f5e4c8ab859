// C = A @ B^T for at most 256 rows of A on one rank: how the work is laid out, and its launch.
#pragma once
#include <cuda.h>

#include <array>
#include <cstdint>
#include <string>
#include <vector>

#include "../common/status.h"

namespace tdb {

constexpr int kSkinnyMaxStages = 16;
constexpr int kSkinnyMaxCluster = 4;
constexpr int kSkinnySmem = 225 * 1024;

// n runs of a total, the first `more` of them one longer than `len`. (No division where a run is looked up.)
struct EvenRuns {
  int32_t len, more;
#ifdef __CUDACC__
  __host__ __device__
#endif
  int start(int v) const { return v * len + (v < more ? v : more); }
};

struct SkinnyParams {
  CUtensorMap tma_a;       // A [M, K], box ar rows x 64 columns
  CUtensorMap tma_b;       // B [rows, K], box wr rows x 64 columns
  int32_t M, N;            // output (SwiGLU: B holds 2N rows)
  int32_t k_blocks;
  int32_t bf16;
  int32_t swiglu, up_row0;
  int32_t cluster_log2;    // CTAs of a worker, each with a range of K: 1, 2 or 4
  int32_t groups;          // N / 8
  int32_t shares;          // runs of groups, dealt round-robin to the workers
  EvenRuns share, range;   // groups of the shares, k-blocks of the ranges
  int32_t workers;
  int32_t mb;              // 128-row blocks of A
  int32_t ar;              // rows of A in shared memory
  int32_t wr, nb, boxes;   // rows of B per box, rows of shared memory per box, boxes per k-block (SwiGLU: gate, up)
  int32_t kw;              // k-blocks per stage
  int32_t stages, stage_bytes;
  int32_t pad;             // bytes behind the ring: the MMA reads whole blocks of A, whatever the number of rows
  int32_t mma_n;           // columns of the MMA
  int32_t accs_log2, acc_cols;   // accumulators a CTA's K sum is spread over, tensor memory columns of each
  int32_t tmem_cols;
  int32_t own;             // most groups of a share that one CTA of the cluster sums up
  int32_t warps;           // 32-row quarters of the blocks that have rows
  int32_t parts_in_ring;   // the CTAs of a cluster exchange parts in the ring, when it has been read
  int32_t smem_bytes;
  double us;               // expected time
  void* c;
  int64_t ldc;
  WaitEnv env;
};

// Fills everything but the tensor maps, c, ldc and env. `sms`: CTAs that can run at once; `odd_rows`: rows of an operand start
// on odd multiples of 16 bytes (of the expected time only).
SkinnyParams skinny_plan(int M, int N, int K, bool swiglu, bool bf16, int sms, bool odd_rows = false);
// First and end group of every share.
std::vector<std::array<int, 2>> skinny_shares(const SkinnyParams& p);
// What a layout would read or write outside the memory that it is given, one sentence each (for the checked mode).
std::vector<std::string> skinny_check(const SkinnyParams& p);
void skinny_launch(const SkinnyParams& p, bool early_start, void* stream);

}  // namespace tdb
