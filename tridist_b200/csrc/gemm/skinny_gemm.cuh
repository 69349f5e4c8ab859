// C = A @ B^T for few rows of A (at most 256, a decode batch): the time is that of reading B once.
//
// A worker is a cluster of 1, 2 or 4 CTAs. It takes a share of B's rows, an even run of 8-row groups, whole, and
// its CTAs a range of K each. Rows of A are re-read through L2 by every worker; what a CTA reads in all bounds
// the cluster's size from below and its width from above (see skinny_plan). The CTAs hand one another the parts of their
// sums in shared memory, each adds up a run of the share's groups in the order of the K ranges and stores it:
// nothing passes through global memory and no two workers meet.
//
// Tiles of 128 or 256 columns cut along K, whose fp32 partials met in L2, spent 12 us of a launch on the meeting and
// 0.4 us on a k-block whatever its width. us a launch then and now, back to back over weights from DRAM: 64 x 4096 x
// 1376 14.7 and 7.6, 128 x 8192 x 3584 23 and 15.5, 128 x 2 x 3584 x 8192 with SwiGLU 35.6 and 29.
//
// Roles (224 threads): warp 0 loads B, warp 6 A, warp 1 multiplies and owns the tensor memory, warps 2-5 store,
// one TMEM lane quarter (32 rows) each of every 128-row block of A. A long range of K is summed in up to four
// accumulators, one run of it each, that the epilogue adds in order. Loads and MMAs are issued by an elected lane of a warp whose control flow is
// uniform, with a stage of kW k-blocks unrolled: a k-block is 32 to 128 cycles of the tensor pipe for so few
// rows, and a loop that issues it from one diverged lane takes 400 or more.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../common/ptx.cuh"
#include "../common/sync.cuh"
#include "../ops/skinny_gemm.h"

namespace tdb {

constexpr int kSkinnyThreads = 224;

__device__ __forceinline__ float skinny_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

template <int kW>
__global__ void __launch_bounds__(kSkinnyThreads, 1) skinny_gemm_kernel(const __grid_constant__ SkinnyParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* const ring = smem;
  // parts from the other CTAs of the cluster
  uint8_t* const xbuf = p.parts_in_ring ? ring : smem + p.stages * p.stage_bytes + p.pad;
  __shared__ __align__(8) uint64_t full_bar[kSkinnyMaxStages], empty_bar[kSkinnyMaxStages], acc_full[2], acc_empty[2],
      x_full, x_ready, drain_bar;
  __shared__ uint32_t tmem_slot;

  const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int cl2 = p.cluster_log2, cluster = 1 << cl2;
  const int sub = cluster > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int worker = static_cast<int>(blockIdx.x) >> cl2;
  const WaitEnv& env = p.env;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    mbar_init(&x_full, max(1, (cluster - 1) * min(4, p.warps)));
    mbar_init(&x_ready, max(1, cluster - 1));
    mbar_init(&drain_bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (cluster > 1) cluster_arrive();              // (the other half stands where a peer's barrier is first touched)

  const int kb0 = p.range.start(sub), kb1 = p.range.start(sub + 1);
  const int steps = (kb1 - kb0 + kW - 1) / kW, stages = p.stages, shares = p.shares, workers = p.workers;
  if (warp == 0 || warp == 6) {
    const bool lead = elect_one();
    const int a_step = p.ar * 128, b_step = p.nb * 128;      // bytes of a k-block of A and of one box of B
    const bool two_boxes = p.boxes == 2;
    const int b_blk = two_boxes ? 2 * b_step : b_step;
    const int b_off = kW * a_step;                // a stage: kW k-blocks of A, then kW of B
    const uint32_t block_tx = static_cast<uint32_t>((p.ar + p.boxes * p.wr) * 128);
    const int up_row0 = p.up_row0, stage_bytes = p.stage_bytes;
    const EvenRuns share = p.share;
    const CUtensorMap* const amap = &p.tma_a;
    const CUtensorMap* const bmap = &p.tma_b;
    if (lead && warp == 6) tma_prefetch_desc(amap);
    if (lead && warp == 0) {
      // What the first stages will load of B is asked of L2 while the kernel in front still runs: a
      // request brings no data here, so it does not matter whether that kernel writes B.
      tma_prefetch_desc(bmap);
      const int row = share.start(worker) * 8;
      for (int kb = kb0; kb < min(kb1, kb0 + stages * kW); ++kb) {
        tma_prefetch_l2_2d(bmap, kb * 64, row);
        if (two_boxes) tma_prefetch_l2_2d(bmap, kb * 64, row + up_row0);
      }
    }
    __syncwarp();
    griddep_wait();
    griddep_launch();
    int stage = 0;
    uint32_t phase = 0, armed = 0;                // armed: stages that a load was asked for
    bool ok = true;
    for (int v = worker; ok && v < shares; v += workers) {
      const int b_row = share.start(v) * 8;
      for (int i = 0; i < steps; ++i) {
        ok = wait_mbar(&empty_bar[stage], phase ^ 1u, env, SITE_PIPE_EMPTY, stage);
        ok = __all_sync(0xFFFFFFFFu, ok) != 0;
        if (!ok) break;
        if (lead) {
          uint64_t* const bar = &full_bar[stage];
          uint8_t* const sa = ring + stage * stage_bytes;
          const int kb = kb0 + i * kW;
          const int n = min(kW, kb1 - kb);
          if (warp == 0) {
            uint8_t* const sb = sa + b_off;
            mbar_arrive_expect_tx(bar, block_tx * n);
#pragma unroll
            for (int j = 0; j < kW; ++j) {
              if (j >= n) break;
              tma_load_2d(sb + j * b_blk, bmap, bar, (kb + j) * 64, b_row);
              if (two_boxes) tma_load_2d(sb + j * b_blk + b_step, bmap, bar, (kb + j) * 64, b_row + up_row0);
            }
          } else {
#pragma unroll
            for (int j = 0; j < kW; ++j) {
              if (j >= n) break;
              tma_load_2d(sa + j * a_step, amap, bar, (kb + j) * 64, 0);
            }
          }
        }
        __syncwarp();
        armed |= 1u << stage;
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
    if (lane == 0) {
      // The loads in flight land before the shared memory goes, whoever else has given up: a loader that is through has
      // up to a ring of them on their way, which nobody but the MMA warp would wait for.
      if (!ok) {
        // (no barrier counts these alone: the other loader may have left its half of a stage out; they take microseconds)
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      } else if (warp == 0) {
        WaitEnv quiet{};                          // no status, no abort word: this wait only drains
        quiet.rank = env.rank;
        quiet.timeout_ns = 2000000ull;
        for (int s = 0; s < stages; ++s)
          if ((armed >> s & 1u) != 0u && !wait_mbar(&full_bar[s], s < stage ? phase : phase ^ 1u, quiet, SITE_PIPE_FULL, s)) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    tmem_alloc(&tmem_slot, p.tmem_cols);
    tmem_relinquish();
    // (the loads need no tensor memory and do not wait for it)
    tc_fence_before_sync();
    named_bar_sync(2, 160);
    tc_fence_after_sync();
    const bool lead = elect_one();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    const uint64_t a_step = static_cast<uint64_t>(p.ar * 8), b_step = static_cast<uint64_t>(p.nb * p.boxes * 8);   // of a k-block, 16-byte units
    const uint64_t da0 = umma_desc_k_sw128(smem_u32(ring));
    const uint64_t db0 = umma_desc_k_sw128(smem_u32(ring) + kW * p.ar * 128);
    const uint64_t stage_step = static_cast<uint64_t>(p.stage_bytes >> 4);
    const uint32_t idesc = umma_idesc_f16(p.bf16 != 0, 128, p.mma_n);
    const int al2 = p.accs_log2, acc_cols = p.acc_cols;
    const bool two_blocks = p.mb == 2;
    const uint32_t d_block = static_cast<uint32_t>(acc_cols << al2);      // from block 0's accumulators to block 1's
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int it = 0;
    for (int v = worker; ok && v < shares; v += workers, ++it) {
      const int buf = it & 1;
      ok = wait_mbar(&acc_empty[buf], static_cast<uint32_t>(it >> 1 & 1) ^ 1u, env, SITE_TMEM_EMPTY, buf);
      ok = __all_sync(0xFFFFFFFFu, ok) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t d = tmem + static_cast<uint32_t>(buf * p.mb) * d_block;
      int acc = 0, acc_end = steps >> al2;
      uint32_t keep = 0u;                           // 0: the next MMA overwrites its accumulator
      for (int i = 0; i < steps; ++i) {
        if (i == acc_end) {                         // the next run of K has an accumulator of its own
          ++acc;
          acc_end = ((acc + 1) * steps) >> al2;
          d += static_cast<uint32_t>(acc_cols);
          keep = 0u;
        }
        ok = wait_mbar(&full_bar[stage], phase, env, SITE_PIPE_FULL, stage);
        ok = __all_sync(0xFFFFFFFFu, ok) != 0;
        if (!ok) break;
        tc_fence_after_sync();
        if (lead) {
          const uint64_t da = da0 + static_cast<uint64_t>(stage) * stage_step;
          const uint64_t db = db0 + static_cast<uint64_t>(stage) * stage_step;
          const int n = min(kW, kb1 - kb0 - i * kW);
#pragma unroll
          for (int j = 0; j < kW; ++j) {
            if (j >= n) break;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_ss(d, da + j * a_step + k * 2, db + j * b_step + k * 2, idesc, (j | k) ? 1u : keep);
            if (two_blocks) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_f16_ss(d + d_block, da + j * a_step + 1024 + k * 2, db + j * b_step + k * 2, idesc, (j | k) ? 1u : keep);
            }
          }
          umma_commit(&empty_bar[stage]);
        }
        __syncwarp();
        keep = 1u;
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
      if (!ok) break;
      if (lead) umma_commit(&acc_full[buf]);
      __syncwarp();
    }
    if (lead) {
      // The MMAs issued retire before tensor and shared memory go, also where the warps that wait for their sums
      // have given up.
      umma_commit(&drain_bar);
      WaitEnv quiet{};
      quiet.rank = env.rank;
      quiet.timeout_ns = env.timeout_ns;
      wait_mbar(&drain_bar, 0u, quiet, SITE_TMEM_FULL, 0);
    }
    __syncwarp();
  } else {
    named_bar_sync(2, 160);
    tc_fence_after_sync();
    griddep_wait();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    const int q = warp & 3;                         // TMEM lane quarter
    const bool warp_on = q < p.warps;
    const int accs = 1 << p.accs_log2, acc_cols = p.acc_cols, swiglu = p.swiglu;
    const EvenRuns share = p.share;
    const bool bf16 = p.bf16 != 0;
    const int up_col = p.nb;                        // the up columns stand behind the gate columns
    // xbuf: [source, the owner left out][gate, up][group of the owner's run][two 16-byte halves][row]
    const int rows = p.warps * 32;
    const int x_half = rows * 16, x_group = 2 * x_half, x_part = p.own * x_group, x_src = (swiglu ? 2 : 1) * x_part;
    // sum of the accumulators, columns [col, col + 8 G)
    auto take = [&](uint32_t t, int col, auto& x) {
      constexpr int kCols = sizeof(x) / 4;
#pragma unroll 1
      for (int a = 0; a < accs; ++a) {
        uint32_t r[kCols];
        const uint32_t at = t + static_cast<uint32_t>(a * acc_cols + col);
        if constexpr (kCols == 16) tmem_ld_32x32b_x16(at, r);
        else tmem_ld_32x32b_x8(at, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kCols; ++j) x[j] = a == 0 ? __uint_as_float(r[j]) : x[j] + __uint_as_float(r[j]);
      }
    };
    if (cluster > 1) cluster_wait();                // the peers' barriers are initialised
    int it = 0;
    bool ok = true;
    for (int v = worker; ok && v < shares; v += workers, ++it) {
      const int buf = it & 1;
      if (lane == 0) ok = wait_mbar(&acc_full[buf], static_cast<uint32_t>(it >> 1 & 1), env, SITE_TMEM_FULL, buf);
      ok = __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t t0 = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * p.mb * accs * acc_cols);
      const int g_lo = share.start(v);
      const int n = share.start(v + 1) - g_lo;      // groups of the share
      auto owned = [&](int r) { return (n * r) >> cl2; };      // first of them that CTA r of the cluster adds up
      if (warp_on) {
        if (cluster > 1) {
          // (a cluster has one share: the parts' buffer is written once)
          if (p.parts_in_ring) {
            // this CTA's loads and MMAs are through with its ring; the others' must be before it writes there
            if (q == 0 && lane == 0)
              for (int o = 1; o < cluster; ++o) mbar_arrive_cluster(&x_ready, static_cast<uint32_t>((sub + o) & (cluster - 1)));
            __syncwarp();
            if (lane == 0) ok = wait_mbar(&x_ready, 0u, env, SITE_SPLITK, sub);
            ok = __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
          }
          for (int o = 1; o < cluster; ++o) {
            const int dst = (sub + o) & (cluster - 1);
            const int lo = owned(dst), hi = owned(dst + 1);
            for (int m = 0; m < p.mb && m * 4 + q < p.warps; ++m) {
              const uint32_t t = t0 + static_cast<uint32_t>(m * accs * acc_cols);
              const uint32_t base =
                  cluster_smem_addr(xbuf + (sub < dst ? sub : sub - 1) * x_src + (m * 128 + q * 32 + lane) * 16, static_cast<uint32_t>(dst));
              for (int h = 0; h < (swiglu ? 2 : 1); ++h) {
                auto send = [&](int g, auto& x) {
                  take(t, h * up_col + g * 8, x);
#pragma unroll
                  for (int k = 0; k < static_cast<int>(sizeof(x) / 32); ++k) {
                    const uint32_t to = base + static_cast<uint32_t>(h * x_part + (g + k - lo) * x_group);
                    st_cluster_v4(to, x[8 * k], x[8 * k + 1], x[8 * k + 2], x[8 * k + 3]);
                    st_cluster_v4(to + static_cast<uint32_t>(x_half), x[8 * k + 4], x[8 * k + 5], x[8 * k + 6], x[8 * k + 7]);
                  }
                };
                int g = lo;
                for (float x[16]; g + 2 <= hi; g += 2) send(g, x);
                if (g < hi) {
                  float x[8];
                  send(g, x);
                }
              }
            }
            __syncwarp();                           // the warp's stores before the arrival that publishes them
            if (lane == 0) mbar_arrive_cluster(&x_full, static_cast<uint32_t>(dst));
          }
          if (lane == 0) ok = wait_mbar(&x_full, 0u, env, SITE_SPLITK, sub);
          ok = __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
          if (!ok) break;
          fence_acq_rel_cluster();
        }
        const int lo = owned(sub), hi = owned(sub + 1);
        for (int m = 0; m < p.mb && m * 4 + q < p.warps; ++m) {
          const uint32_t t = t0 + static_cast<uint32_t>(m * accs * acc_cols);
          const int token = m * 128 + q * 32 + lane;
          const bool row_ok = token < p.M;
          uint8_t* const c_row = reinterpret_cast<uint8_t*>(p.c) + static_cast<int64_t>(token) * p.ldc * 2;
          // the sum over the K ranges, in their order, of the gate (h = 0) or up columns of the groups from g on
          auto sum = [&](int h, int g, auto& x) {
            constexpr int kGroups = sizeof(x) / 32;
            if (cluster == 1) {
              take(t, h * up_col + g * 8, x);
              return;
            }
            float mine[8 * kGroups];
            take(t, h * up_col + g * 8, mine);
#pragma unroll
            for (int j = 0; j < 8 * kGroups; ++j) x[j] = 0.f;
            const uint8_t* from = xbuf + h * x_part + (g - lo) * x_group + token * 16;
#pragma unroll 1
            for (int s = 0; s < cluster; ++s) {
#pragma unroll
              for (int k = 0; k < 2 * kGroups; ++k) {
                const float4 y = s == sub ? make_float4(mine[4 * k], mine[4 * k + 1], mine[4 * k + 2], mine[4 * k + 3])
                                          : *reinterpret_cast<const float4*>(from + k * x_half);
                x[4 * k] += y.x;
                x[4 * k + 1] += y.y;
                x[4 * k + 2] += y.z;
                x[4 * k + 3] += y.w;
              }
              if (s != sub) from += x_src;
            }
          };
          auto finish = [&](int g, auto& x, auto& u) {
            constexpr int kCols = sizeof(x) / 4;
            sum(0, g, x);
            if (swiglu) {
              sum(1, g, u);
#pragma unroll
              for (int j = 0; j < kCols; ++j) x[j] = skinny_silu(x[j]) * u[j];
            }
            uint32_t w[kCols / 2];
            if (bf16) {
#pragma unroll
              for (int j = 0; j < kCols / 2; ++j) {
                __nv_bfloat162 y = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
                w[j] = *reinterpret_cast<uint32_t*>(&y);
              }
            } else {
#pragma unroll
              for (int j = 0; j < kCols / 2; ++j) {
                __half2 y = __floats2half2_rn(x[2 * j], x[2 * j + 1]);
                w[j] = *reinterpret_cast<uint32_t*>(&y);
              }
            }
            if (row_ok) {
              uint8_t* const dst = c_row + static_cast<int64_t>(g_lo + g) * 16;
#pragma unroll
              for (int k = 0; k < kCols / 8; ++k) st_global_v4(dst + k * 16, make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]));
            }
          };
          int g = lo;
          for (float x[16], u[16]; g + 2 <= hi; g += 2) finish(g, x, u);
          if (g < hi) {
            float x[8], u[8];
            finish(g, x, u);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  if (cluster > 1) {
    // a cluster leaves together: nobody's shared memory goes while another can still write to it
    if (warp <= 1 || warp == 6) cluster_wait();
    cluster_sync_all();
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(&tmem_slot), p.tmem_cols);
  }
}

}  // namespace tdb
