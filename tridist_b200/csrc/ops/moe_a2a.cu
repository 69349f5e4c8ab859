#include "moe_a2a.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <stdexcept>
#include <string>

#include "../common/ptx.cuh"
#include "../common/sync.cuh"
#include "fused_gemm.h"

namespace tdb {

static void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("tridist_b200: ") + what + ": " + cudaGetErrorString(e));
}

// With nv > 1 one launch carries several emulated ranks: consecutive CTAs
// belong to consecutive ranks so that the first CTA of every rank is in the
// first wave (those CTAs raise the flags all others wait on).
#define TDB_MOE_PROLOGUE                                              \
  const int vr = (nv > 1) ? static_cast<int>(blockIdx.x % nv) : 0;    \
  const int cta = (nv > 1) ? static_cast<int>(blockIdx.x / nv) : static_cast<int>(blockIdx.x); \
  const int ncta = (nv > 1) ? static_cast<int>(gridDim.x / nv) : static_cast<int>(gridDim.x);  \
  const MoeDesc& d = (nv > 1) ? dv[vr] : d0;                          \
  (void)cta; (void)ncta;

// ----------------------------------------------------------------------------
// Metadata: histogram of topk_idx -> splits, with a slot for every pair; exchange with every
// rank by direct peer stores + ticket; prefix sums -> segment tables. No host sync (the
// reference needs two: moe_a2a.py:463-492).
//
// CTA c owns pairs [c * meta_chunk, (c + 1) * meta_chunk): it counts them in shared memory, keeps
// the running count of each pair's expert as that pair's slot, and reserves its share of every
// expert's rows with one global add per expert (cta_base). The last CTA in does the exchange and
// the three prefix sums. One CTA alone took 36 us over 160 000 pairs (one SM's worth of load
// latency) and 6.6 us over 512 (a system-scope exchange with itself, a serial prefix sum): now 6.3
// and 3.6.
// ----------------------------------------------------------------------------
constexpr int kMetaThreads = 1024;      // one expert per thread in the prefix sums (E <= 1024)

// Exclusive prefix sums of three values per thread over the whole CTA.
__device__ __forceinline__ void scan3(int32_t (&v)[3], int32_t* part /* [3][32] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t inc[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    int32_t x = v[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    inc[q] = x;
    if (lane == 31) part[q * 32 + warp] = x;
  }
  __syncthreads();
  if (warp < 3) {
    int32_t x = part[warp * 32 + lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    part[warp * 32 + lane] = x;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = inc[q] - v[q] + (warp > 0 ? part[q * 32 + warp - 1] : 0);
}

__global__ void __launch_bounds__(kMetaThreads)
moe_meta_kernel(const __grid_constant__ MoeDesc d0, const MoeDesc* __restrict__ dv, int nv) {
  TDB_MOE_PROLOGUE
  extern __shared__ int32_t sm[];
  int32_t* hist = sm;                 // [E]
  int32_t* pre_own = hist + d.E;      // [E + 1] prefix sums of this rank's counts
  int32_t* pre_low = pre_own + d.E + 1;   // [E + 1] prefix sums of the lower ranks' counts
  int32_t* meta = pre_low + d.E + 1;  // [R * E]
  __shared__ int32_t part[3 * 32];
  __shared__ int s_ok, s_last;
  const int tid = threadIdx.x;
  const int E = d.E, R = d.R;

  for (int e = tid; e < E; e += kMetaThreads) hist[e] = 0;
  if (tid == 0) s_ok = 1;
  __syncthreads();
  griddep_wait();
  if (d.R == 1) griddep_launch();
  const int pairs = d.T * d.topk;
  const int lo = cta * d.meta_chunk, hi = min(pairs, lo + d.meta_chunk);
  for (int i = lo + tid; i < hi; i += 2 * kMetaThreads) {
    const int i2 = i + kMetaThreads;
    const int e = d.topk_idx[i];
    const int e2 = i2 < hi ? d.topk_idx[i2] : -1;
    if (e >= 0 && e < E) d.slots[i] = atomicAdd(&hist[e], 1);
    if (e2 >= 0 && e2 < E) d.slots[i2] = atomicAdd(&hist[e2], 1);
  }
  __syncthreads();
  if (ncta > 1) {
    for (int e = tid; e < E; e += kMetaThreads) {
      const int n = hist[e];
      d.cta_base[cta * E + e] = n > 0 ? atomicAdd(&d.counters[e], n) : 0;
    }
    __syncthreads();
    // the barrier ordered the CTA's adds before this arrival; the last arrival sees all of them
    if (tid == 0) s_last = atom_add_acq_rel_gpu(d.meta_counter, 1u) + 1u == static_cast<uint32_t>(ncta);
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) *d.meta_counter = 0u;
    for (int e = tid; e < E; e += kMetaThreads) {
      hist[e] = *reinterpret_cast<const volatile int32_t*>(d.counters + e);
      d.counters[e] = 0;              // ready for the next round
    }
    __syncthreads();
  } else {
    for (int e = tid; e < E; e += kMetaThreads) d.cta_base[e] = 0;
  }
  for (int e = tid; e < E; e += kMetaThreads) d.splits[e] = hist[e];
  if (R > 1) {
    for (int i = tid; i < R * E; i += kMetaThreads) {
      const int dst = i / E, e = i - dst * E;
      d.peer_meta[dst][d.rank * E + e] = hist[e];
    }
    // the barrier orders every thread's stores before the releases below (cumulative)
    __syncthreads();
    if (tid < R) {
      st_release_sys(d.peer_meta_flags[tid] + d.rank, d.round);
      if (!wait_flag_ge(d.peer_meta_flags[d.rank] + tid, d.round, d.env, SITE_MOE_META, tid)) s_ok = 0;
    }
    __syncthreads();
    if (s_ok == 0) return;
    for (int i = tid; i < R * E; i += kMetaThreads)
      meta[i] = *reinterpret_cast<const volatile int32_t*>(d.peer_meta[d.rank] + i);
  } else {
    for (int e = tid; e < E; e += kMetaThreads) meta[e] = hist[e];   // nobody to exchange with
  }
  __syncthreads();

  // thread i, as a destination: segment i = (source, local expert) in order; as a source: expert i
  int32_t cnt = 0, own_cnt = 0, low_cnt = 0;
  if (tid < E) {
    cnt = meta[(tid / d.epr) * E + d.rank * d.epr + tid % d.epr];
    own_cnt = meta[d.rank * E + tid];
    for (int s = 0; s < d.rank; ++s) low_cnt += meta[s * E + tid];
  }
  int32_t v[3] = {cnt, own_cnt, low_cnt};
  scan3(v, part);
  if (tid < E) {
    d.recv_seg[tid] = v[0];
    d.recv_counts[tid] = cnt;
    pre_own[tid] = v[1];
    pre_low[tid] = v[2];
  }
  if (tid == E - 1) {
    pre_own[E] = v[1] + own_cnt;
    pre_low[E] = v[2] + low_cnt;
    const int run = v[0] + cnt;
    *d.recv_total = run;
    if (run > d.max_recv_rows)
      report_failure(d.env, ST_OVERFLOW, SITE_MOE_META, d.max_recv_rows, run, 0);
  }
  __syncthreads();
  // where my rows for expert e start inside the owner's buffer: after all rows of the lower ranks
  // for that owner, and after my own rows for its earlier experts
  if (tid < E) {
    const int first = tid / d.epr * d.epr;
    d.dst_row_base[tid] = pre_low[first + d.epr] - pre_low[first] + v[1] - pre_own[first];
  }
}

// ----------------------------------------------------------------------------
// Dispatch: one warp per (token, run of 32 * V 16-byte pieces). The pieces are read once and
// stored to all topk destination rows, straight into the owner ranks' receive buffers; lane j
// works out the row of the token's j-th expert, so one round of look-ups serves the whole warp.
// Bound by the writes. (One warp per (token, expert) read the token 8 times through L2 and waited
// for a chain of look-up, atomic slot and load per row: 20 011 tokens of 8 KB, topk 8, skewed
// routing, took 369 us against 251 now, 5.9 TB/s.)
// The last CTA to finish tells every rank "my rows are in place" and waits until
// every rank said the same, so the kernel's completion means recv is complete.
// ----------------------------------------------------------------------------
constexpr int kMaxTopk = 32;            // one lane per expert of a token
constexpr int kRowThreads = 128;

// Metadata and dispatch of one rank's small batch in one kernel: every CTA counts ALL the pairs, and those in
// front of its own tokens, in shared memory, so that no CTA waits for another and a pair's slot is its place among
// the pairs of its expert. Bound by latency: the pairs' load, the counts, the prefix sum and the rows' stores follow
// one another once, where two kernels did so twice (64 tokens of 8 KB, topk 8: 7.2 us a round against 10.0). CTA (c, s)
// then stores slice s of the rows of tokens [c * per, (c + 1) * per). It is the first kernel of a round, launched while
// the GEMM or combine in front of it still writes the tokens: they are not read past the coherent path, which wants data
// that nobody writes while the kernel lives. (moe_dispatch_kernel stands behind the metadata kernel and may.)
constexpr int kRouteThreads = 256;

__global__ void __launch_bounds__(kRouteThreads)
moe_route_dispatch_kernel(const __grid_constant__ MoeDesc d, int per, int slices) {
  extern __shared__ int32_t sm[];
  const int E = d.E, topk = d.topk, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int32_t* const hist = sm;              // [E] pairs of an expert; their exclusive prefix sum in the end
  int32_t* const before = hist + E;      // [E] those in front of this CTA's first token
  __shared__ int32_t part[kRouteThreads / 32], own_e[kRouteThreads], own_row[kRouteThreads];
  const int c = static_cast<int>(blockIdx.x) / slices, slice = static_cast<int>(blockIdx.x) - c * slices;
  const int t0 = c * per, t1 = min(d.T, t0 + per);
  const int lo = t0 * topk, hi = t1 * topk, pairs = d.T * topk;
  for (int e = tid; e < 2 * E; e += kRouteThreads) sm[e] = 0;
  __syncthreads();
  griddep_wait();
  griddep_launch();
  const int64_t row_bytes = static_cast<int64_t>(d.H) * 2;
  const int n16 = static_cast<int>(row_bytes >> 4);
  const int i0 = slice * kRouteThreads + tid;      // this thread's first 16-byte piece of a row
  const uint8_t* const tokens = reinterpret_cast<const uint8_t*>(d.tokens) + (static_cast<int64_t>(i0) << 4);
  uint4 first = make_uint4(0u, 0u, 0u, 0u);        // (on its way while the pairs are counted)
  if (t0 < t1 && i0 < n16) first = ld_global_cg_v4(tokens + t0 * row_bytes);
  constexpr int kU = 8;                            // pairs of a thread whose loads are in flight together
  for (int b = tid; b < pairs; b += kU * kRouteThreads) {
    int e[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int i = b + u * kRouteThreads;
      e[u] = i < pairs ? d.topk_idx[i] : -1;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int i = b + u * kRouteThreads;
      if (i >= lo && i < hi) own_e[i - lo] = e[u];
      if (e[u] < 0 || e[u] >= E) continue;
      atomicAdd(&hist[e[u]], 1);
      if (i < lo) atomicAdd(&before[e[u]], 1);
    }
  }
  __syncthreads();
  // exclusive prefix sum of hist: each thread a run of experts
  const int each = (E + kRouteThreads - 1) / kRouteThreads;
  int32_t sum = 0;
  for (int k = 0; k < each; ++k) {
    const int e = tid * each + k;
    if (e < E) sum += hist[e];
  }
  int32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) part[warp] = inc;
  __syncthreads();
  int32_t run = inc - sum;
  for (int w = 0; w < warp; ++w) run += part[w];
  const bool writes = blockIdx.x == 0;
  for (int k = 0; k < each; ++k) {
    const int e = tid * each + k;
    if (e >= E) break;
    const int32_t n = hist[e];
    hist[e] = run;
    if (writes) {
      d.splits[e] = n;
      d.recv_counts[e] = n;
      d.recv_seg[e] = run;
      d.dst_row_base[e] = run;
      if (e == E - 1) {
        *d.recv_total = run + n;
        if (run + n > d.max_recv_rows)
          report_failure(d.env, ST_OVERFLOW, SITE_MOE_META, d.max_recv_rows, run + n, 0);
      }
    }
    run += n;
  }
  __syncthreads();
  if (tid < hi - lo) {
    const int e = own_e[tid];
    int row = -1;
    if (e >= 0 && e < E) {
      row = hist[e] + before[e];
      for (int j = 0; j < tid; ++j) row += own_e[j] == e ? 1 : 0;
      if (row >= d.max_recv_rows) {
        if (slice == 0) report_failure(d.env, ST_OVERFLOW, SITE_MOE_DISPATCH_DONE, d.max_recv_rows, row, e);
        row = -1;
      }
    }
    own_row[tid] = row;
    if (slice == 0) d.scatter_idx[lo + tid] = row;
  }
  __syncthreads();
  uint8_t* const recv = reinterpret_cast<uint8_t*>(d.peer_recv[0]) + (static_cast<int64_t>(i0) << 4);
  const int64_t step = static_cast<int64_t>(slices) * kRouteThreads * 16;
  for (int t = t0; t < t1; ++t) {
    const int32_t* const rows = own_row + (t - t0) * topk;
    int64_t off = 0;
    for (int i = i0; i < n16; i += slices * kRouteThreads, off += step) {
      const uint4 v = (t == t0 && off == 0) ? first : ld_global_cg_v4(tokens + t * row_bytes + off);
#pragma unroll 4
      for (int j = 0; j < topk; ++j) {
        const int r = rows[j];
        if (r >= 0) st_global_v4(recv + r * row_bytes + off, v);
      }
    }
  }
}

template <int V>
__global__ void __launch_bounds__(kRowThreads)
moe_dispatch_kernel(const __grid_constant__ MoeDesc d0, const MoeDesc* __restrict__ dv, int nv) {
  TDB_MOE_PROLOGUE
  __shared__ int s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row_bytes = static_cast<int64_t>(d.H) * 2;
  const int n16 = static_cast<int>(row_bytes >> 4);
  const int runs = (n16 + 32 * V - 1) / (32 * V);
  const int64_t units = static_cast<int64_t>(d.T) * runs;
  const int topk = d.topk;
  griddep_wait();
  if (d.R == 1) griddep_launch();
  for (int64_t unit = static_cast<int64_t>(cta) * (kRowThreads / 32) + warp; unit < units;
       unit += static_cast<int64_t>(ncta) * (kRowThreads / 32)) {
    const int t = static_cast<int>(unit / runs);
    const int run = static_cast<int>(unit - static_cast<int64_t>(t) * runs);
    const int i0 = run * 32 * V + lane;
    const uint8_t* src = reinterpret_cast<const uint8_t*>(d.tokens) + t * row_bytes;
    uint4 v[V];
#pragma unroll
    for (int u = 0; u < V; ++u)
      if (i0 + 32 * u < n16) v[u] = ld_global_nc_v4(src + (static_cast<int64_t>(i0 + 32 * u) << 4));
    int row = -1, dest = 0;
    if (lane < topk) {
      const int pair = t * topk + lane;
      const int e = d.topk_idx[pair];
      if (e >= 0 && e < d.E) {
        row = d.dst_row_base[e] + d.cta_base[(pair / d.meta_chunk) * d.E + e] + d.slots[pair];
        dest = e / d.epr;
        if (row < 0) {
          // the base comes from counts other ranks wrote: a negative row is recorded, never used
          if (run == 0)
            report_failure(d.env, ST_BAD_INDEX, SITE_INDEX_CHECK, 0u, static_cast<uint32_t>(row), e);
          row = -1;
        } else if (row >= d.max_recv_rows) {
          if (run == 0)
            report_failure(d.env, ST_OVERFLOW, SITE_MOE_DISPATCH_DONE, d.max_recv_rows, row, e);
          row = -1;
        }
      }
      if (run == 0) d.scatter_idx[pair] = row;
    }
    for (int j = 0; j < topk; ++j) {
      const int r = __shfl_sync(0xFFFFFFFFu, row, j);
      const int o = __shfl_sync(0xFFFFFFFFu, dest, j);
      if (r < 0) continue;
      uint8_t* dst = reinterpret_cast<uint8_t*>(d.peer_recv[o]) + r * row_bytes;
#pragma unroll
      for (int u = 0; u < V; ++u)
        if (i0 + 32 * u < n16) st_global_v4(dst + (static_cast<int64_t>(i0 + 32 * u) << 4), v[u]);
    }
  }
  if (d.R == 1) return;      // nobody else reads or writes recv: the end of the kernel says it all
  // one system fence per CTA, by the thread that counts the CTA in, after the barrier that
  // orders all of the CTA's row stores before it (a fence in every thread costs microseconds)
  __syncthreads();
  if (tid == 0) {
    __threadfence_system();
    const uint32_t old = atomicAdd(d.done_counter, 1u);
    s_last = (old + 1u == static_cast<uint32_t>(ncta)) ? 1 : 0;
  }
  __syncthreads();
  if (s_last) {
    if (tid == 0) {
      atomicExch(d.done_counter, 0u);
      __threadfence_system();
    }
    __syncthreads();
    if (tid < d.R) {
      st_release_sys(d.peer_done_flags[tid] + d.rank, d.round);
      wait_flag_ge(d.peer_done_flags[d.rank] + tid, d.round, d.env, SITE_MOE_DISPATCH_DONE, tid);
    }
  }
}

// ----------------------------------------------------------------------------
// Combine: pull model, bound by the reads of topk expert rows per token. fp32 sums in the order of a
// token's experts, in two forms with the same bits.
//
// By registers (moe_combine_rows_kernel): one warp per (token, run of 32 * V 16-byte pieces), lane j
// looking the token's j-th row up one unit ahead, eight loads per lane on their way at a time. As many
// bytes in flight for one expert per token or a narrow row as for many and a wide one.
//
// By a ring (moe_combine_kernel): a CTA works through its (token, 8 KB run) units with three stages of
// eight rows in shared memory. Lane j of the producer warp looks the token's j-th row up (one item ahead)
// and copies its run into the stage with one bulk copy; warp w sums its 16-byte columns of the stage.
// A whole 8 KB row is one request and a full stage keeps 64 KB in flight whatever the look-ups take,
// where scattered reads of 2 KB are what DRAM serves slowly: 20 011 tokens of 8 KB rows, topk 8, 237 us,
// 6.2 TB/s. A row is read once, so its lines are the first to leave L2 again and what dispatch or the experts
// left there stays until it is read: 4096 tokens of 8 KB, topk 8, a round 115 us without, 108.5 with. (The same on the
// register form's loads: 8192 tokens of 8 KB, topk 4, 128 and 125 us, but 9000 of 16 KB, topk 2, 166 and 170, 20000 of 8 KB,
// topk 4, 299 and 304.) A stage that is not full is wasted: 24 KB in flight at topk 1 (see launch_combine).
// ----------------------------------------------------------------------------
template <bool kBf16>
__device__ __forceinline__ void fma8(float (&acc)[8], const uint4& v, float w) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 f;
    if constexpr (kBf16) f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j]));
    else f = __half22float2(*reinterpret_cast<const __half2*>(&u[j]));
    acc[2 * j] = fmaf(w, f.x, acc[2 * j]);
    acc[2 * j + 1] = fmaf(w, f.y, acc[2 * j + 1]);
  }
}

template <bool kBf16>
__device__ __forceinline__ uint4 pack8(const float (&a)[8]) {
  uint4 o;
  uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (kBf16) {
      __nv_bfloat162 v = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
      w[j] = *reinterpret_cast<uint32_t*>(&v);
    } else {
      __half2 v = __floats2half2_rn(a[2 * j], a[2 * j + 1]);
      w[j] = *reinterpret_cast<uint32_t*>(&v);
    }
  }
  return o;
}

// "My expert outputs are complete" to every rank, and the same from every rank. False = gave up (all
// threads of the CTA agree).
__device__ __forceinline__ bool combine_ready(const MoeDesc& d, int cta, int tid) {
  if (cta == 0 && tid < d.R) {
    __threadfence_system();
    st_release_sys(d.peer_ready_flags[tid] + d.rank, d.round);
  }
  int ok = 1;
  if (tid < d.R)
    ok = wait_flag_ge(d.peer_ready_flags[d.rank] + tid, d.round, d.env, SITE_MOE_COMBINE_READY, tid) ? 1 : 0;
  return __syncthreads_and(ok) != 0;
}

// First byte of the expert row of a pair, or nullptr where it has none (an expert that does not exist, a
// pair dropped at dispatch, a row out of range, which is recorded when `report` is set).
__device__ __forceinline__ const uint8_t* expert_row(const MoeDesc& d, int e, int row, int64_t row_bytes, bool report) {
  if (e < 0 || e >= d.E) return nullptr;
  if (row >= 0 && row < d.max_recv_rows) return reinterpret_cast<const uint8_t*>(d.peer_out[e / d.epr]) + row * row_bytes;
  if (row != -1 && report)
    report_failure(d.env, ST_BAD_INDEX, SITE_INDEX_CHECK, static_cast<uint32_t>(d.max_recv_rows),
                   static_cast<uint32_t>(row), e);
  return nullptr;
}

template <bool kBf16, int V>
__global__ void __launch_bounds__(kRowThreads)
moe_combine_rows_kernel(const __grid_constant__ MoeDesc d0, const MoeDesc* __restrict__ dv, int nv) {
  TDB_MOE_PROLOGUE
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  griddep_wait();
  if (d.R == 1) griddep_launch();
  if (d.R > 1 && !combine_ready(d, cta, tid)) return;
  constexpr int kRows = 8 / V;            // expert rows whose pieces are loaded together
  const int64_t row_bytes = static_cast<int64_t>(d.H) * 2;
  const int n16 = static_cast<int>(row_bytes >> 4);
  const int runs = (n16 + 32 * V - 1) / (32 * V);
  const int topk = d.topk;
  const int64_t units = static_cast<int64_t>(d.T) * runs;
  const int64_t step = static_cast<int64_t>(ncta) * (kRowThreads / 32);
  int64_t unit = static_cast<int64_t>(cta) * (kRowThreads / 32) + warp;
  int e = -1, row = -1;
  float w = 0.f;
  auto look_up = [&](int64_t n) {
    if (n < units && lane < topk) {
      const int64_t pair = n / runs * topk + lane;
      e = d.topk_idx[pair];
      row = d.scatter_idx[pair];
      w = d.has_weights ? d.topk_weights[pair] : 1.0f;
    }
  };
  look_up(unit);
  for (; unit < units; unit += step) {
    const int64_t t = unit / runs;
    const int run = static_cast<int>(unit - t * runs);
    const int i0 = run * 32 * V + lane;
    const uint8_t* src = lane < topk ? expert_row(d, e, row, row_bytes, run == 0) : nullptr;
    const float my_w = w;
    look_up(unit + step);
    float acc[V][8];
#pragma unroll
    for (int u = 0; u < V; ++u)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
#pragma unroll 1
    for (int j0 = 0; j0 < topk; j0 += kRows) {
      uint4 v[kRows][V];
#pragma unroll
      for (int b = 0; b < kRows; ++b) {
        const uint8_t* from = reinterpret_cast<const uint8_t*>(
            __shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(src), (j0 + b) & 31));
        const bool have = j0 + b < topk && from != nullptr;
#pragma unroll
        for (int u = 0; u < V; ++u)
          v[b][u] = (have && i0 + 32 * u < n16) ? ld_global_cg_v4(from + (static_cast<int64_t>(i0 + 32 * u) << 4))
                                                : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int b = 0; b < kRows; ++b) {
        const float wj = __shfl_sync(0xFFFFFFFFu, my_w, (j0 + b) & 31);
        if (j0 + b < topk) {
#pragma unroll
          for (int u = 0; u < V; ++u) fma8<kBf16>(acc[u], v[b][u], wj);
        }
      }
    }
    uint8_t* dst = reinterpret_cast<uint8_t*>(d.output) + t * row_bytes;
#pragma unroll
    for (int u = 0; u < V; ++u)
      if (i0 + 32 * u < n16) st_global_v4(dst + (static_cast<int64_t>(i0 + 32 * u) << 4), pack8<kBf16>(acc[u]));
  }
}

constexpr int kCombineWarps = 8;        // and one more that produces
constexpr int kCombineRows = 8;         // expert rows per stage
constexpr int kRunBytes = 8192;         // of a row, per stage
constexpr int kStageBytes = kCombineRows * kRunBytes;
constexpr int kDepth = 3;               // stages (192 KB)

template <bool kBf16>
__global__ void __launch_bounds__((kCombineWarps + 1) * 32)
moe_combine_kernel(const __grid_constant__ MoeDesc d0, const MoeDesc* __restrict__ dv, int nv) {
  TDB_MOE_PROLOGUE
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ __align__(8) uint64_t s_full[kDepth], s_empty[kDepth];
  __shared__ float s_w[kDepth][kCombineRows];
  __shared__ uint32_t s_have[kDepth];     // rows of the stage that were copied
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < kDepth) {
    mbar_init(&s_full[tid], 1);
    mbar_init(&s_empty[tid], kCombineWarps);
  }
  mbar_fence_init();
  __syncthreads();
  griddep_wait();
  if (d.R == 1) griddep_launch();
  if (d.R > 1) {
    if (!combine_ready(d, cta, tid)) return;
    fence_proxy_async_all();        // what the peers' kernels stored, before the bulk copies read it
  }

  const int64_t row_bytes = static_cast<int64_t>(d.H) * 2;
  const int runs = static_cast<int>(row_bytes / kRunBytes);      // (the launch asks for whole runs)
  const int topk = d.topk;
  const int groups = (topk + kCombineRows - 1) / kCombineRows;
  const int64_t units = static_cast<int64_t>(d.T) * runs;
  // work item k of this CTA: rows [8 * (k % groups), ...) of unit cta + (k / groups) * ncta
  const int64_t items = cta < units ? ((units - cta + ncta - 1) / ncta) * groups : 0;
  int slot = 0;
  uint32_t phase = 0;
  const uint64_t once = l2_evict_first();

  if (warp == kCombineWarps) {
    int64_t unit = cta;
    int group = 0, run = 0, e = -1, row = -1;
    float w = 0.f;
    auto look_up = [&]() {
      const int t = static_cast<int>(unit / runs);
      run = static_cast<int>(unit - static_cast<int64_t>(t) * runs);
      const int j = group * kCombineRows + lane;
      e = -1;
      w = 0.f;
      if (lane < kCombineRows && j < topk) {
        const int pair = t * topk + j;
        e = d.topk_idx[pair];
        row = d.scatter_idx[pair];
        w = d.has_weights ? d.topk_weights[pair] : 1.0f;
      }
    };
    if (items > 0) look_up();
    int64_t k = 0;
    for (; k < items; ++k) {
      bool ok = true;
      if (lane == 0) ok = wait_mbar(&s_empty[slot], phase ^ 1u, d.env, SITE_PIPE_EMPTY, slot);
      ok = __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      const uint8_t* src = expert_row(d, e, row, row_bytes, run == 0);
      const int64_t off = static_cast<int64_t>(run) * kRunBytes;
      const uint32_t have = __ballot_sync(0xFFFFFFFFu, src != nullptr);
      if (lane < kCombineRows) s_w[slot][lane] = w;
      if (lane == 0) s_have[slot] = have;
      __syncwarp();                     // the weights before the arrival that publishes the stage
      if (lane == 0) mbar_arrive_expect_tx(&s_full[slot], kRunBytes * __popc(have));
      __syncwarp();
      if (src != nullptr)
        bulk_load_1d_hint(ring + slot * kStageBytes + lane * kRunBytes, src + off, kRunBytes, &s_full[slot], once);
      if (++slot == kDepth) { slot = 0; phase ^= 1u; }
      if (++group == groups) { group = 0; unit += ncta; }
      if (k + 1 < items) look_up();
    }
    // the copies in flight land before the shared memory goes, whoever has given up (each wait bounded)
    WaitEnv quiet{};
    quiet.rank = d.env.rank;
    quiet.timeout_ns = 2000000ull;
    for (int s = 0; lane == 0 && s < kDepth && s < k; ++s)
      wait_mbar(&s_full[s], s < slot ? phase : phase ^ 1u, quiet, SITE_PIPE_FULL, s);
    return;
  }

  constexpr int V = kRunBytes / (kCombineWarps * 512);      // 16-byte columns per lane
  constexpr int kColStep = kCombineWarps * 512;
  const int col = (warp * 32 + lane) * 16;                  // the first of them
  float acc[V][8];
  int64_t unit = cta;
  int group = 0;
  for (int64_t k = 0; k < items; ++k) {
    if (group == 0) {
#pragma unroll
      for (int u = 0; u < V; ++u)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
    }
    bool ok = true;
    if (lane == 0) ok = wait_mbar(&s_full[slot], phase, d.env, SITE_PIPE_FULL, slot);
    ok = __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
    if (!ok) return;
    const uint32_t have = s_have[slot];
    const int rows = min(kCombineRows, topk - group * kCombineRows);
    const uint8_t* stage = ring + slot * kStageBytes + col;
#pragma unroll
    for (int j = 0; j < kCombineRows; ++j) {
      if (j >= rows) break;
      const float w = s_w[slot][j];
#pragma unroll
      for (int u = 0; u < V; ++u) {
        const uint4 v = (have >> j & 1u) ? *reinterpret_cast<const uint4*>(stage + j * kRunBytes + u * kColStep)
                                         : make_uint4(0u, 0u, 0u, 0u);
        fma8<kBf16>(acc[u], v, w);
      }
    }
    __syncwarp();                       // every lane has read the stage
    if (lane == 0) mbar_arrive(&s_empty[slot]);
    if (++slot == kDepth) { slot = 0; phase ^= 1u; }
    if (++group == groups) {
      const int t = static_cast<int>(unit / runs);
      const int64_t off = (unit - static_cast<int64_t>(t) * runs) * kRunBytes + col;
#pragma unroll
      for (int u = 0; u < V; ++u)
        st_global_v4(reinterpret_cast<uint8_t*>(d.output) + t * row_bytes + off + u * kColStep, pack8<kBf16>(acc[u]));
      group = 0;
      unit += ncta;
    }
  }
}

// ----------------------------------------------------------------------------
// Launchers
// ----------------------------------------------------------------------------
static void validate(const MoeDesc& d) {
  if (d.R < 1 || d.R > 8) throw std::runtime_error("tridist_b200: MoE needs 1..8 ranks");
  if (d.E < 1 || d.E > 1024 || d.E % d.R != 0)
    throw std::runtime_error("tridist_b200: MoE needs num_experts <= 1024 and divisible by ranks");
  if (d.topk < 1 || d.topk > kMaxTopk) throw std::runtime_error("tridist_b200: MoE needs topk <= 32");
  if ((static_cast<int64_t>(d.H) * 2) % 16 != 0)
    throw std::runtime_error("tridist_b200: MoE needs hidden % 8 == 0");
}

// CTAs of the metadata kernel: 2048 pairs (two per thread) each, at most kMoeMetaCtas.
static int meta_ctas(const MoeDesc& d) {
  const int64_t pairs = static_cast<int64_t>(d.T) * d.topk;
  int64_t g = (pairs + 2047) / 2048;
  if (g > kMoeMetaCtas) g = kMoeMetaCtas;
  return g < 1 ? 1 : static_cast<int>(g);
}

static size_t meta_smem(const MoeDesc& d) {
  return sizeof(int32_t) * (d.E + 2 * (d.E + 1) + static_cast<size_t>(d.R) * d.E);
}

// Pairs per metadata CTA: the same in the metadata and the dispatch launch of a round.
static MoeDesc with_chunk(const MoeDesc& d, int ctas) {
  MoeDesc m = d;
  const int64_t pairs = static_cast<int64_t>(d.T) * d.topk;
  m.meta_chunk = static_cast<int32_t>((pairs + ctas - 1) / ctas);
  if (m.meta_chunk < 1) m.meta_chunk = 1;
  return m;
}

// 16-byte pieces per lane (V) of the row kernels: as many as the row is wide, fewer while that
// leaves SMs without a few warps each.
static int row_pieces(const MoeDesc& d, int most) {
  const int n16 = d.H / 8;
  int v = most;
  while (v > 1 && (n16 < 32 * v || static_cast<int64_t>(d.T) * ((n16 + 32 * v - 1) / (32 * v)) < 148 * 16)) v /= 2;
  return v;
}

static int row_ctas(const MoeDesc& d, int v, int per_sm) {
  const int n16 = d.H / 8;
  const int64_t units = static_cast<int64_t>(d.T) * ((n16 + 32 * v - 1) / (32 * v));
  int64_t g = (units + kRowThreads / 32 - 1) / (kRowThreads / 32);
  if (g > 148 * per_sm) g = 148 * per_sm;
  return g < 1 ? 1 : static_cast<int>(g);
}

// One launch; a single rank's kernels overlap their start with the end of the one before (see
// griddep_wait), kernels that wait for peers keep plain stream order.
static void launch(void (*kernel)(const MoeDesc, const MoeDesc*, int), int grid, int threads, size_t smem,
                   const MoeDesc& d, const MoeDesc* dev, int nv, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (d.R == 1 && nv == 1) ? 1 : 0;
  check(cudaLaunchKernelEx(&cfg, kernel, d, dev, nv), "MoE kernel launch");
}

static void launch_dispatch(const MoeDesc& d, const MoeDesc* dev, int nv, cudaStream_t s) {
  const int v = row_pieces(d, 8);
  const int g = row_ctas(d, v, 16) * nv;
  if (v == 8) launch(moe_dispatch_kernel<8>, g, kRowThreads, 0, d, dev, nv, s);
  else if (v == 4) launch(moe_dispatch_kernel<4>, g, kRowThreads, 0, d, dev, nv, s);
  else if (v == 2) launch(moe_dispatch_kernel<2>, g, kRowThreads, 0, d, dev, nv, s);
  else launch(moe_dispatch_kernel<1>, g, kRowThreads, 0, d, dev, nv, s);
}

template <bool kBf16>
static void launch_combine_ring(const MoeDesc& d, const MoeDesc* dev, int nv, cudaStream_t s) {
  auto* kernel = moe_combine_kernel<kBf16>;
  static std::atomic<uint64_t> ready{0};      // devices on which the ring's size has been allowed
  int dev_id = 0;
  check(cudaGetDevice(&dev_id), "cudaGetDevice");
  if (!(ready.load() >> (dev_id & 63) & 1u)) {
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDepth * kStageBytes),
          "cudaFuncSetAttribute(combine ring)");
    ready.fetch_or(1ull << (dev_id & 63));
  }
  launch(kernel, 148 * nv, (kCombineWarps + 1) * 32, kDepth * kStageBytes, d, dev, nv, s);
}

template <bool kBf16, int V>
static void launch_combine_rows(const MoeDesc& d, const MoeDesc* dev, int nv, cudaStream_t s) {
  launch(moe_combine_rows_kernel<kBf16, V>, row_ctas(d, V, 16) * nv, kRowThreads, 0, d, dev, nv, s);
}

template <bool kBf16>
static void launch_combine(const MoeDesc& d, const MoeDesc* dev, int nv, cudaStream_t s) {
  // The ring where its stages fill: whole 8 KB runs, six of the eight rows, a few tokens for every SM.
  // 32768 tokens, us by ring and by registers: 8 KB rows, topk 8 395 and 434, topk 6 336 and 346, topk 4
  // 295 and 254, topk 1 238 and 123; 2 KB rows, topk 8 320 and 125; 4096 tokens of 10 KB rows, topk 8 96 and
  // 86, of 8 KB rows, topk 16 109 and 117; 512 tokens of 8 KB rows, topk 8 20 and 18.
  const int groups = (d.topk + kCombineRows - 1) / kCombineRows;
  if ((d.H * 2) % kRunBytes == 0 && 4 * d.topk >= 3 * kCombineRows * groups && d.T >= 148 * 4) {
    launch_combine_ring<kBf16>(d, dev, nv, s);
    return;
  }
  const int v = row_pieces(d, 4);
  if (v == 4) launch_combine_rows<kBf16, 4>(d, dev, nv, s);
  else if (v == 2) launch_combine_rows<kBf16, 2>(d, dev, nv, s);
  else launch_combine_rows<kBf16, 1>(d, dev, nv, s);
}

void moe_meta_launch(const MoeDesc& d, void* stream_) {
  validate(d);
  const int g = meta_ctas(d);
  launch(moe_meta_kernel, g, kMetaThreads, meta_smem(d), with_chunk(d, g), nullptr, 1,
         reinterpret_cast<cudaStream_t>(stream_));
  launch_count_add(1);
}

void moe_dispatch_launch(const MoeDesc& d, void* stream_) {
  validate(d);
  launch_dispatch(with_chunk(d, meta_ctas(d)), nullptr, 1, reinterpret_cast<cudaStream_t>(stream_));
  launch_count_add(1);
}

void moe_route_and_dispatch_launch(const MoeDesc& d, void* stream_) {
  // Up to 4096 pairs, which every CTA counts in two batches of loads, and 2048 tokens, which leave each CTA a few.
  // us a round in one kernel and in two, 8 KB rows, topk 8: 1 token 5.7 and 8.9, 64 7.2 and 10.0, 128 10.7 and 10.9, 256
  // 12.6 and 14.4, 512 17.9 and 20.2, 1024 31.9 and 31.8; 4000 tokens of 2 KB, topk 1, 14.7 and 14.1; 1024 tokens of
  // 2 KB, topk 8, 17.6 and 16.2.
  const int64_t pairs = static_cast<int64_t>(d.T) * d.topk;
  if (d.R != 1 || pairs > 4096 || d.T > 2048) {
    moe_meta_launch(d, stream_);
    moe_dispatch_launch(d, stream_);
    return;
  }
  validate(d);
  const int n16 = d.H / 8;
  int slices = 1;
  while (d.T * slices < 148 * 4 && 2 * slices * kRouteThreads <= n16) slices *= 2;
  const int per = std::max(1, (d.T * slices + 148 * 8 - 1) / (148 * 8));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::max(1, (d.T + per - 1) / per) * slices, 1, 1);
  cfg.blockDim = dim3(kRouteThreads, 1, 1);
  cfg.dynamicSmemBytes = 2 * sizeof(int32_t) * d.E;
  cfg.stream = reinterpret_cast<cudaStream_t>(stream_);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  check(cudaLaunchKernelEx(&cfg, moe_route_dispatch_kernel, d, per, slices), "MoE route and dispatch launch");
  launch_count_add(1);
}

void moe_combine_launch(const MoeDesc& d, void* stream_) {
  validate(d);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (d.bf16) launch_combine<true>(d, nullptr, 1, s);
  else launch_combine<false>(d, nullptr, 1, s);
  launch_count_add(1);
}

void moe_emulated_launch(const std::vector<MoeDesc>& ds, int phase, void* stream_) {
  const int nv = static_cast<int>(ds.size());
  if (nv < 1 || nv > 8) throw std::runtime_error("tridist_b200: bad emulated rank count");
  for (auto& d : ds) validate(d);
  // the metadata CTAs of a rank wait for those of the others: all of them in one wave
  const int g = std::min(meta_ctas(ds[0]), 148 / nv);
  std::vector<MoeDesc> host;
  for (auto& d : ds) host.push_back(with_chunk(d, g));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  static MoeDesc* dev = nullptr;
  if (!dev) check(cudaMalloc(&dev, sizeof(MoeDesc) * 8), "cudaMalloc(moe descs)");
  check(cudaMemcpyAsync(dev, host.data(), sizeof(MoeDesc) * nv, cudaMemcpyHostToDevice, s), "copy descs");
  check(cudaStreamSynchronize(s), "sync descs");
  const MoeDesc& d = host[0];
  if (phase == 0) {
    MoeDesc dummy = d;
    const MoeDesc* dp = dev;
    int nvv = nv;
    void* args[3] = {&dummy, &dp, &nvv};
    check(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(moe_meta_kernel), dim3(nv * g), dim3(kMetaThreads),
                                      args, meta_smem(d), s),
          "moe_meta cooperative launch");
  } else if (phase == 1) {
    launch_dispatch(d, dev, nv, s);
  } else {
    if (d.bf16) launch_combine<true>(d, dev, nv, s);
    else launch_combine<false>(d, dev, nv, s);
  }
  check(cudaGetLastError(), "moe emulated launch");
  launch_count_add(1);
}

}  // namespace tdb
