#include "skinny_gemm.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <stdexcept>
#include <string>

#include "../gemm/skinny_gemm.cuh"

namespace tdb {

static void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("tridist_b200: ") + what + ": " + cudaGetErrorString(e));
}

static int ceil_div(int a, int b) { return (a + b - 1) / b; }
static int up_to(int a, int m) { return ceil_div(a, m) * m; }

static EvenRuns even_runs(int total, int n) { return {total / n, total % n}; }

// Everything that follows from a cluster size and the most rows of B in a share.
static SkinnyParams lay_out(int M, int N, int K, bool swiglu, bool bf16, int sms, int cluster_log2, int most) {
  SkinnyParams p;
  std::memset(&p, 0, sizeof(p));
  const int cluster = 1 << cluster_log2;
  p.M = M;
  p.N = N;
  p.k_blocks = ceil_div(K, 64);
  p.bf16 = bf16 ? 1 : 0;
  p.swiglu = swiglu ? 1 : 0;
  p.up_row0 = N;
  p.cluster_log2 = cluster_log2;
  p.range = even_runs(p.k_blocks, cluster);
  p.groups = N / 8;
  p.boxes = swiglu ? 2 : 1;
  const int can_run = std::max(1, cluster <= 2 ? sms / cluster : sms * 7 / 8 / cluster);   // (larger clusters leave SMs out)
  const int rounds = ceil_div(ceil_div(p.groups, can_run), most / 8 / p.boxes);
  p.shares = std::min(rounds * can_run, ceil_div(p.groups, 2));
  p.share = even_runs(p.groups, p.shares);
  p.workers = std::min(p.shares, can_run);
  p.mb = ceil_div(M, 128);
  p.ar = up_to(M, 8);
  p.wr = 8 * (p.share.len + (p.share.more > 0 ? 1 : 0));
  p.nb = up_to(p.wr, 16);
  p.mma_n = p.boxes * p.nb;
  p.own = ceil_div(p.wr / 8, cluster);
  p.warps = ceil_div(M, 32);
  const int parts = (cluster - 1) * p.boxes * p.own * p.warps * 1024;
  // (two blocks' parts would take two stages of the ring from it)
  p.parts_in_ring = (cluster > 1 && p.mb == 2) ? 1 : 0;
  const int xbuf = p.parts_in_ring ? 0 : parts;
  const int block = (p.ar + p.nb * p.boxes) * 128;
  p.pad = (128 * p.mb - p.ar) * 128;
  const int room = kSkinnySmem - p.pad - xbuf;
  const int range = p.range.len + (p.range.more > 0 ? 1 : 0);
  p.kw = 8;
  while (p.kw > 1 && ((p.kw == 8 ? 2 : 3) * p.kw * block > room || p.kw >= 2 * range)) p.kw /= 2;
  p.stage_bytes = p.kw * block;
  p.stages = std::min(kSkinnyMaxStages, room / p.stage_bytes);
  p.stages = std::max(1, std::min(p.stages, ceil_div(range, p.kw) * ceil_div(p.shares, p.workers)));
  p.smem_bytes = std::max(p.stages * p.stage_bytes + p.pad + xbuf, parts);
  p.acc_cols = up_to(p.mma_n, 32);
  const int bufs = p.shares > p.workers ? 2 : 1;
  // runs of 16 k-blocks or more, four of them over the whole of K
  while (2 << p.accs_log2 <= 4 / cluster && (p.mb * bufs * p.acc_cols << (p.accs_log2 + 1)) <= 512 &&
         (32 << p.accs_log2) <= p.range.len) ++p.accs_log2;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.mb * bufs * p.acc_cols << p.accs_log2) p.tmem_cols *= 2;
  return p;
}

SkinnyParams skinny_plan(int M, int N, int K, bool swiglu, bool bf16, int sms, bool odd_rows) {
  // The expected time: B from DRAM; what a CTA loads in all, at about 120 GB/s through its L2 port, or its k-blocks,
  // 130 ns each however small; the two overlap, not wholly. A cluster starts later and exchanges parts, 2.5 us for
  // two CTAs and 5 for four. us measured with clusters of 1, 2 and 4 (rows x N x K), back to back over one set of operands, the
  // 126 MB of L2 clean (over changing inputs the first takes 87, behind 256 MB of writes 99): 128 x 8192 x 28672 89.5, 81.7 and 104;
  // 128 x 8192 x 3584 15.2, 16.6 and 23.7; 64 x 4096 x 1376 7.6, 8.4 and 9.3; 64 x 2048 x 16384 36.7, 25.7 and 21.3;
  // 128 x 512 x 8192 23.7, 15.9 and 15.5. 128 x 28672 x 8192 by shares of 104 and of 200 rows 92.7 and 76.8.
  auto cta_us = [](const SkinnyParams& p, double port) {
    const double mma = p.mb * 4 * std::max(p.mma_n, 48) / 2 / 1.7e3;        // us a k-block
    const double rounds = ceil_div(p.shares, p.workers);
    return rounds * (p.range.len + 1) * std::max({(p.ar + p.wr * p.boxes) * 128 / 0.12e6 * port, mma, 0.13});
  };
  const double dram = static_cast<double>(N) * (swiglu ? 2 : 1) * K * 2 / 6.3e6;
  SkinnyParams best;
  double best_us = -1;
  for (int cl2 = 0; 1 << cl2 <= kSkinnyMaxCluster; ++cl2)
    for (int most = 128; most <= 256; most *= 2) {
      SkinnyParams p = lay_out(M, N, K, swiglu, bf16, sms, cl2, most);
      if (best_us >= 0 && (p.tmem_cols > 512 || p.smem_bytes > kSkinnySmem)) continue;
      if (cl2 > 0 && (p.range.len < 2 || p.shares > p.workers)) continue;     // (a cluster meets once)
      if (best_us >= 0 && p.stages * p.stage_bytes < 120 * 1024) continue;    // (too little in flight)
      const double meet = cl2 == 0 ? 0.0 : cl2 == 1 ? 2.5 : p.mb == 1 ? 5.0 : 9.0;
      const double cta = cta_us(p, 1.0);
      const double us = std::max(dram, cta) + 0.3 * std::min(dram, cta) + meet;
      if (best_us < 0 || us < 0.98 * best_us) {
        best = p;
        best_us = us;
        const double odd = odd_rows ? cta_us(p, 1.6) : cta;
        best.us = std::max(dram, odd) + 0.3 * std::min(dram, odd) + meet;
      }
    }
  // With start and epilogue. Two blocks of A leave the ring three to five short stages: 12 % more. The tiles of the general
  // kernel are faster where they fill the device with a long K to cut. us here and there: 192 x 896 x 608 8.9 and 14.3,
  // 256 x 11008 x 4096 45 and 67, 192 x 29568 x 8192 109 and 132; 192 x 8192 x 28672 120 and 111.
  // Rows on odd multiples of 16 bytes (`odd_rows`): a 128-byte piece of each lies in five sectors and two lines, and the
  // port takes 1.6 times as long (median of 100 shapes of 40 to 256 rows); the layout stays.
  best.us = (best.us + 4.0) * (best.mb == 2 ? 1.12 : 1.0);
  return best;
}

std::vector<std::array<int, 2>> skinny_shares(const SkinnyParams& p) {
  std::vector<std::array<int, 2>> out;
  for (int v = 0; v < p.shares; ++v) out.push_back({p.share.start(v), p.share.start(v + 1)});
  return out;
}

std::vector<std::string> skinny_check(const SkinnyParams& p) {
  std::vector<std::string> bad;
  auto need = [&](bool ok, const char* what) {
    if (!ok) bad.push_back(std::string("few-rows layout: ") + what);
  };
  const int cluster = 1 << p.cluster_log2;
  need(cluster <= kSkinnyMaxCluster && p.workers >= 1 && p.workers <= p.shares && (cluster == 1 || p.workers == p.shares),
       "workers and shares");
  need(p.share.start(p.shares) == p.groups && p.groups * 8 == p.N, "the shares do not cover the columns");
  need(p.range.start(cluster) == p.k_blocks && p.range.len >= 1, "the ranges do not cover K");
  const int most = p.share.len + (p.share.more > 0 ? 1 : 0);
  need(p.share.len >= 1 && most * 8 <= p.wr && p.wr <= p.nb && p.wr <= 256, "a share is larger than its box");
  need(p.M <= p.ar && p.ar <= 256 && p.M <= 32 * p.warps && p.M <= 128 * p.mb, "rows outside the boxes of A");
  need(ceil_div(most, cluster) <= p.own, "a CTA adds up more groups than its parts have room for");
  const int block = (p.ar + p.nb * p.boxes) * 128;
  const int parts = (cluster - 1) * p.boxes * p.own * p.warps * 1024;
  const int ring = p.stages * p.stage_bytes + p.pad;
  need(p.stages >= 1 && p.stages <= kSkinnyMaxStages && p.stage_bytes >= p.kw * block, "stages of the ring");
  need((p.parts_in_ring ? std::max(ring, parts) : ring + parts) <= p.smem_bytes && p.smem_bytes <= kSkinnySmem, "shared memory");
  // (the MMA reads whole 128-row blocks of A: the last k-block's end in the columns of B and the pad)
  need((p.kw - 1) * p.ar * 128 + p.mb * 128 * 128 <= p.stage_bytes + p.pad, "the MMA reads behind the ring");
  const int bufs = p.shares > p.workers ? 2 : 1;
  need(p.mma_n <= p.acc_cols && p.mma_n <= 256 && (p.mb * bufs * p.acc_cols << p.accs_log2) <= p.tmem_cols && p.tmem_cols <= 512,
       "tensor memory");
  return bad;
}

template <int kW>
static void launch(const SkinnyParams& p, bool early_start, cudaStream_t stream) {
  auto* kernel = skinny_gemm_kernel<kW>;
  static std::atomic<uint64_t> ready{0};      // devices on which the ring's size has been allowed
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  if (!(ready.load() >> (dev & 63) & 1u)) {
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSkinnySmem),
          "cudaFuncSetAttribute(few-rows GEMM)");
    ready.fetch_or(1ull << (dev & 63));
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.workers << p.cluster_log2, 1, 1);
  cfg.blockDim = dim3(kSkinnyThreads, 1, 1);
  cfg.dynamicSmemBytes = p.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1 << p.cluster_log2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early_start ? 2 : 1;
  check(cudaLaunchKernelEx(&cfg, kernel, p), "few-rows GEMM launch");
}

void skinny_launch(const SkinnyParams& p, bool early_start, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  switch (p.kw) {
    case 1: launch<1>(p, early_start, stream); break;
    case 2: launch<2>(p, early_start, stream); break;
    case 4: launch<4>(p, early_start, stream); break;
    case 8: launch<8>(p, early_start, stream); break;
    default: throw std::runtime_error("tridist_b200: bad stage depth");
  }
}

}  // namespace tdb
