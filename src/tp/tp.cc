// Host side of the fused tensor-parallel GEMMs: contexts, TMA descriptors, launches.
// See include/nccl_tp.h for the API and src/tp/gemm_sm100.cu for the kernels.
#include "tp.h"

#include <cuda.h>

#include <map>

#include "../comm/device_plane.h"
#include "nccl_tp.h"

using namespace b200;

namespace b200 {
B200_PARAM(TpCommCtas, "B200_TP_COMM_CTAS", 0, "CTAs that gather remote rows in all-gather -> GEMM (0: 4 for two ranks, 8 up to four, 16 beyond)")
B200_PARAM(TpSplit, "B200_TP_SPLIT", 8, "Largest cluster of CTAs that shares the K dimension of a tile in plain bf16 GEMMs with few tiles (1: never, at most 8)")
B200_PARAM(TpWidth, "B200_TP_WIDTH", 0, "Tile width of plain bf16 GEMMs whose tiles are not split: 128, 160, 192, 224 or 256 (0: by shape)")
B200_PARAM(TpFp8Width, "B200_TP_FP8_WIDTH", 0, "Tile width of plain block-scaled fp8 GEMMs: 128 or 256 (0: by shape)")
B200_PARAM(TpFp8Split, "B200_TP_FP8_SPLIT", 0, "CTAs that share the K blocks of a tile in plain block-scaled fp8 GEMMs: 1 to 8 (0: by shape)")
B200_PARAM(TpPair, "B200_TP_PAIR", 1, "bf16 GEMM on CTA pairs (256 x 256 tiles, tcgen05 cta_group::2) when the row count allows")
}

struct ncclTpContext {
  ncclComm* comm = nullptr;
  int smCount = 0;
  int pairClusters = 0;   // clusters of the CTA-pair GEMM kernel that can be resident at once (0: unavailable)
  int splitClusters[kTpMaxSplit + 1] = {};   // clusters of each size of the split kernel that can be resident at once
  int fp8Clusters[kTpMaxSplit + 1] = {};     // the same for the fp8 kernel
  void* accum = nullptr;           // symmetric staging window: bf16 [n sources][maxRows / n][maxCols]
  size_t accumBytes = 0;
  SymWindow* accumWin = nullptr;
  uint32_t* blockFlags = nullptr;  // one word per 128-row block (all-gather -> GEMM)
  size_t maxBlocks = 0;
  uint32_t epoch = 0;
  std::map<void*, SymWindow*> gathered;
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encodeFn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess) fn = (EncodeTiledFn)p;
    else (void)cudaGetLastError();
  }
  return fn;
}

// Row-major [rows, K] tensor of bf16 (elemBytes 2) or fp8 (1), tiles of boxRows x 128 bytes with 128-byte swizzle.
// Comm CTAs of all-gather -> GEMM: each moves about 33 GB/s (128 KiB of loads in flight over NVLink, measured at two
// ranks); the remote share of the rows and how early the first remote chunk is needed both grow with the number of ranks.
static int tpCommCtas(const ncclTpContext* tp, int nRanks);

static ncclResult_t makeMap(CUtensorMap* map, const void* base, int rows, int K, int boxRows, int elemBytes = 2) {
  EncodeTiledFn enc = encodeFn();
  if (!enc) { WARN("cuTensorMapEncodeTiled is not available"); return ncclUnhandledCudaError; }
  if ((uintptr_t)base & 15) { WARN("tensor-parallel GEMM operands must be 16-byte aligned"); return ncclInvalidArgument; }
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * elemBytes};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elemBytes), (cuuint32_t)boxRows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, elemBytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { WARN("cuTensorMapEncodeTiled failed (%d)", (int)r); return ncclUnhandledCudaError; }
  return ncclSuccess;
}

static void clusterAttribute(cudaLaunchAttribute* attr, int ctas) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
}

// Launches with programmatic stream serialisation when `pdl`: the kernel's set-up overlaps the end of the kernel before it. Plain
// calls only: the fused kernels meet their partners on other GPUs before they would wait.
static ncclResult_t launchTp(ncclTpContext* tp, const void* fn, dim3 grid, int threads, size_t smem, void** args, bool pdl, int cluster, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attrs[2];
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attrs;
  if (cluster > 1) clusterAttribute(&attrs[cfg.numAttrs++], cluster);
  if (pdl && devPlanePdl()) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  if (e != cudaSuccess) { WARN("tensor-parallel kernel launch failed: %s", cudaGetErrorString(e)); (void)cudaGetLastError(); return ncclUnhandledCudaError; }
  if (tp->comm->devPlane) tp->comm->devPlane->launches++;
  return ncclSuccess;
}

static int tpCommCtas(const ncclTpContext* tp, int nRanks) {
  int64_t want = paramTpCommCtas();
  if (want <= 0) want = nRanks <= 2 ? 4 : nRanks <= 4 ? 8 : 16;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, tp->smCount / 4));
}

static ncclResult_t checkShape(int M, int N, int K, int n) {
  if (M <= 0 || N <= 0 || K <= 0 || M % (128 * n) || N % 256 || K % 64) {
    WARN("tensor-parallel GEMM: M=%d must be a multiple of %d, N=%d of 256, K=%d of 64", M, 128 * n, N, K);
    return ncclInvalidArgument;
  }
  return ncclSuccess;
}

static void fillSyncTp(ncclComm* comm, SyncArgs* s) {
  memset(s, 0, sizeof(*s));
  DevicePlane* dp = comm->devPlane;
  if (comm->nRanks > 1 && dp && dp->resWin) {
    for (int p = 0; p < comm->nRanks; ++p) s->inbox[p] = (uint32_t*)dp->resWin->host.peerPtr[p];
    s->epoch[comm->rank] = dp->epochs;
  }
  s->status[comm->rank] = comm->devStatusDev;
  s->abortFlag = comm->abortFlagDev;
  s->timeoutNs = dp ? dp->timeoutNs : 5000000000ull;
}

// Parts of K that a plain bf16 GEMM sums by themselves, 1 for none, and the CTAs that share a tile of 256 columns: as many as leave every cluster resident at once,
// when the 128 x 256 tiles alone would leave half of the SMs idle, and each CTA keeps kSplitMinBlocks K blocks. Where short loops save
// no more than the exchange of the partial sums costs, a CTA keeps its tile. Kernel times against the kernel that the call would
// take instead, weights from memory and from L2, 4 to 72 tiles. One CTA to a tile: K = 1024 1.01-1.10, 1280 0.94-1.05, 1536
// 0.87-1.00, 1792 0.84-0.96, 2560 0.71-0.88. CTA pairs: K = 1024 0.95-1.03, 1280 0.92-1.00, 2560 0.80-0.90.
constexpr int kSplitMinBlocks = 8, kSplitFromOne = 1536 / 64;   // clusters on tiles of 256 columns
static int splitOf(const ncclTpContext* tp, const TpGemmArgs* a, bool insteadOfPairs) {
  const int tiles = (a->M / 128) * (a->N / 256), blocks = a->K / 64;
  if (!insteadOfPairs && blocks < kSplitFromOne) return 1;
  int s = std::min(std::min(std::min((int)paramTpSplit(), kTpMaxSplit), tp->smCount / tiles), blocks / kSplitMinBlocks);
  while (s > 1 && tiles > tp->splitClusters[s]) --s;
  return std::max(s, 1);
}

static ncclResult_t launchGemmSplit(ncclTpContext* tp, const void* A, const void* W, TpGemmArgs* a, int width, cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  tpGemmSplitPlan(a, width);
  NCCLCHECK(makeMap(&tmA, A, a->M, a->K, 128));
  NCCLCHECK(makeMap(&tmB, W, a->N, a->K, width));
  void* args[3] = {&tmA, &tmB, a};
  return launchTp(tp, tpGemmSplitKernelFn(width), dim3((a->M / 128) * (a->N / width) * a->splitK), tpGemmSplitThreads(), tpGemmSplitSmemBytes(), args, true, a->splitK, stream);
}

// How a plain bf16 GEMM runs: one-CTA tiles of 128 x width, CTA pairs (256 x width), or (shares > 1) clusters of `split` CTAs that share the K
// steps of a tile of 128 x width.
struct GemmPlan {
  bool pair = false;
  int width = 256, split = 1, shares = 1;
};

// Tiles of 256 columns, by what the widths below do not change: clusters for few tiles, else pairs where they pay.
static GemmPlan basePlan(const ncclTpContext* tp, const TpGemmArgs* a, bool pairs) {
  GemmPlan p;
  p.split = p.shares = splitOf(tp, a, pairs && a->M % 256 == 0);
  if (p.split > 1) return p;
  p.pair = pairs;
  if (p.pair && a->M % 256) {
    // Pairs leave half of the last row tile empty. A K step of a pair tile takes 0.92 to 0.97 of the time of one of two
    // 128 x 256 tiles (32 KiB of operands from L2 per SM against 48), but a launch of pairs takes about 1.5 us longer, so they pay
    // when they need no more waves and have enough steps. Kernel times of pairs over one-CTA tiles, weights from memory and from
    // L2: two waves 0.97-1.02 at K = 1024, 0.96-1.01 at 1536, 0.91-1.01 at 4096; three and more 0.91-0.98 from 1024 on, about 1.0 at
    // 512; four waves where one-CTA tiles need three 1.1. One wave 1.2 at 512, 1.08 at 1536; at 4096 to 7168 0.90-0.98 when
    // the operands are more than 60 MiB or come from memory, 1.00-1.06 when they are fewer and in L2.
    const int tilesN = a->N / 256, one = a->M / 128 * tilesN, two = (a->M / 128 + 1) / 2 * tilesN;
    const int wavesOne = (one + tp->smCount - 1) / tp->smCount, wavesTwo = (two + tp->pairClusters - 1) / tp->pairClusters;
    const bool enough = wavesOne > 2 ? a->K >= 1024 : wavesOne > 1 ? a->K >= 1536 : a->K >= 4096 && ((size_t)a->M + a->N) * a->K * 2 > (size_t)60 << 20;
    p.pair = wavesTwo <= wavesOne && enough;
  }
  return p;
}

static int wavesOf(const ncclTpContext* tp, const TpGemmArgs* a, const GemmPlan& p) {
  const int tilesN = (a->N + p.width - 1) / p.width;
  return p.pair ? ((a->M + 255) / 256 * tilesN + tp->pairClusters - 1) / tp->pairClusters : (a->M / 128 * tilesN + tp->smCount - 1) / tp->smCount;
}

// Expected time in us, operands in L2: start and last store, K steps of 64 with every SM at work, what a wave of tiles adds, and the
// exchange of a cluster. Fitted to 31 shapes of 4 to 2048 tiles and 8 to 128 K steps, the shared forms to 32; up to four waves it is
// within about 10 %.
static float expectedUs(const ncclTpContext* tp, const TpGemmArgs* a, const GemmPlan& p) {
  const int steps = a->K / 64, own = (p.shares + p.split - 1) / p.split, waves = p.shares > 1 ? 1 : wavesOf(tp, a, p);
  const int share = p.shares > 1 ? (steps * own + p.shares - 1) / p.shares : steps;   // K steps of a CTA
  float step;
  switch (p.width) {
    case 128: step = 0.21f; break;
    case 160: step = 0.255f; break;
    case 192: step = p.pair ? 0.26f : 0.31f; break;
    case 224: step = p.pair ? 0.315f : 0.38f; break;
    default: step = p.pair ? 0.35f : 0.385f; break;
  }
  float exchange = 0.0f;
  if (p.shares > 1 && p.split == 1) {   // nothing to exchange: the sums are in the CTA's own tensor memory
    exchange = 0.6f;
    step = 0.235f;
  } else if (p.shares > 1) {
    exchange = p.width == 256 ? (p.split == 2 ? 2.2f : p.split == 3 ? 4.0f : 5.5f) : 2.0f + 0.4f * p.split + (p.split == 3 ? 0.6f : 0.0f);   // three: one has two chunks
  }
  return (p.pair ? 4.1f : 3.3f) + waves * share * step + (waves - 1) * 0.8f + exchange;
}

// Narrower tiles, alone or shared by a cluster, where 256 columns leave the last wave (or all but a few SMs) empty: a step of 160 columns
// takes 0.65 of the time of one of 256, so what counts is how the tiles fill the chip. Up to four waves of pair tiles: beyond, the
// last wave matters less and the widest tiles have the best rate (8192 x 8192 x 3584: pairs of 256 303 us, 224 312, 192 349).
// Kernel times with 256 columns / the choice, us: 1152 x 2304 x 7168 40.6 / 31.8 (160 columns), 2048 x 2560 x 4096 46.1 / 35.4 (160),
// 1280 x 4096 x 3584 38.4 / 31.9 (pairs of 192), 2560 x 3072 x 2048 25.6 / 23.7 (pairs of 224).
// The other side of the line: 1920 x 4096 x 7168 82.3 with pairs of 256, 91.7 of 192; 3328 x 4096 x 1536 29.5 / 31.7. Pairs of 160 were never
// faster than both pairs of 192 and one CTA with 160 columns (16 shapes, 0.99 to 1.12 of the better one).
// The width never changes the sums: where K is summed in shares it stays so, with an accumulator per share. Weights from memory: 128 x
// 1024 x 2048 10.2 / 7.5 (128 columns, four CTAs), 128 x 4096 x 4096 17.5 / 14.3 (six shares on four CTAs), 128 x 8192 x 8192 29.7 / 29.3 (four on
// two), 512 x 4096 x 1024 10.2 / 8.2 (two on one); 896 x 1536 x 3264 stays, 14.7 / 17.2 (three on one). Fewer shares would be faster by what their sums
// cost to exchange (12.5, 28.3 and 7.5 us for the second to fourth shape), but twice as many results would not be the rounded product
// (0.25 % for 0.12 % of the third).
static GemmPlan planGemm(const ncclTpContext* tp, const TpGemmArgs* a, bool pairs) {
  GemmPlan best = basePlan(tp, a, pairs);
  for (int w : kTpWidths)
    if (w == paramTpWidth()) {
      if (best.shares == 1) {
        best.width = w;
        best.pair = best.pair && w >= kTpPairWidth;
      }
      return best;
    }
  if (((a->M + 255) / 256 * (a->N / 256) + tp->smCount / 2 - 1) / (tp->smCount / 2) > 4) return best;
  float us = (best.shares > 1 ? 0.97f : 0.95f) * expectedUs(tp, a, best);   // what is simpler stays where the others are hardly faster
  auto consider = [&](const GemmPlan& p) {
    const float t = expectedUs(tp, a, p);
    if (t < us) { us = t; best = p; }
  };
  auto earlySums = [](int split, int shares) {
    TpGemmArgs form = {};
    form.splitK = split;
    form.shares = shares;
    return tpGemmSplitPlan(&form, 128);
  };
  const int shares = best.shares, tiles = a->M / 128 * (a->N / 128);
  if (shares > 1) {
    for (int s = (shares + kTpMaxOwnShares - 1) / kTpMaxOwnShares; s <= shares && tiles <= (s > 1 ? tp->splitClusters[s] : tp->smCount); ++s)
      if (earlySums(s, shares) <= kTpMaxEarly) consider({false, 128, s, shares});
    return best;
  }
  for (int w : kTpWidths)
    for (bool pair : {false, true})
      if (!pair || (pairs && w >= kTpPairWidth)) consider({pair, w});
  return best;
}

// Launches the bf16 GEMM kernel in the mode of `a`. Grid: one CTA per SM (fewer when there are fewer
// tiles); in all-gather mode the last CTAs are the comm CTAs. The CTA-pair kernel runs when enabled, when its clusters
// fit and, in the fused modes, when every rank's rows split into 256-row tiles.
static ncclResult_t launchGemm(ncclTpContext* tp, const void* A, const void* W, TpGemmArgs* a, cudaStream_t stream) {
  const int n = a->nRanks;
  const bool fused = n > 1 && a->mode != TP_MODE_STORE;
  const bool gather = fused && a->mode == TP_MODE_GATHER;
  const bool pairs = paramTpPair() != 0 && tp->pairClusters > 0;
  GemmPlan plan;
  if (fused) plan.pair = pairs && a->M % (256 * n) == 0;
  else plan = planGemm(tp, a, pairs);
  a->splitK = plan.split;
  a->shares = plan.shares;
  if (plan.shares > 1) return launchGemmSplit(tp, A, W, a, plan.width, stream);
  const bool pair = plan.pair;
  const int width = plan.width;
  int commCtas = gather ? tpCommCtas(tp, n) : 0;
  int grid;
  const int tilesN = (a->N + width - 1) / width;
  if (pair) {
    commCtas = (commCtas + 1) & ~1;   // both CTAs of a cluster have the same role
    const int tiles = (a->M + 255) / 256 * tilesN;
    const int pairs = std::max(1, std::min(tp->pairClusters - commCtas / 2, tiles));
    a->gemmCtas = 2 * pairs;
    grid = 2 * pairs + commCtas;
  } else {
    const int tiles = (a->M / 128) * tilesN;
    grid = gather ? tp->smCount : std::min(tp->smCount, tiles);
    a->gemmCtas = grid - commCtas;
  }
  CUtensorMap tmA, tmB;
  NCCLCHECK(makeMap(&tmA, A, a->M, a->K, 128));
  NCCLCHECK(makeMap(&tmB, W, a->N, a->K, pair ? width / 2 : width));
  void* args[3] = {&tmA, &tmB, a};
  return launchTp(tp, pair ? tpGemmPairKernelFn(width) : tpGemmKernelFn(width), dim3(grid), pair ? tpGemmPairThreads() : tpGemmThreads(),
                  pair ? tpGemmPairSmemBytes() : tpGemmSmemBytes(), args, !fused, 1, stream);
}

static ncclResult_t launchGemmFp8(ncclTpContext* tp, const void* A, const void* W, TpGemmArgs* a, int grid, cudaStream_t stream, int width = 256) {
  CUtensorMap tmA, tmB;
  NCCLCHECK(makeMap(&tmA, A, a->M, a->K, 128, 1));
  NCCLCHECK(makeMap(&tmB, W, a->N, a->K, width, 1));
  void* args[3] = {&tmA, &tmB, a};
  const bool fused = a->nRanks > 1 && a->mode != TP_MODE_STORE;
  return launchTp(tp, tpGemmFp8KernelFn(fused, width, a->splitK > 1), dim3(grid), tpGemmFp8Threads(), tpGemmFp8SmemBytes(), args, !fused, std::max(a->splitK, 1), stream);
}

// Tile width, CTAs that share the K blocks of a tile (1: none), and grid of a plain fp8 GEMM: the least expected time. A K block takes
// 0.46 us in a tile of 256 columns, 0.54 at the clock of a long run (0.50 below; no choice changes between 0.46 and 0.56), about 0.53 where CTAs share
// it and 0.38 us in one of 128 (the round trip of the accumulator bounds them), a wave of tiles about 3.0 and 2.4 us besides (start, first
// operands, store), the exchange of a cluster 3.7 us (7 us for three CTAs and more on 256 columns, which are not used). Kernel times with
// operands in L2, whole 128 x 256 tiles / the choice: 128 x 1024 x 7168 28.1 / 11.5 us (128 columns, four CTAs), 128 x 4096 x 4096 17.9 / 10.5
// (the same), 512 x 2048 x 7168 28.6 / 17.4 (two CTAs), 1024 x 2048 x 7168 29.2 / 22.4 (256 columns, two CTAs), 512 x 4096 x 1024 8.1 / 6.9 (128
// columns, whole), 896 x 2560 x 3584 17.1 / 15.0 (the same). The other side of the line: 2560 x 3072 x 2048 in 128 columns 32.0 / 22.2, 256 x 4096 x
// 1536 with two CTAs to tiles of 256 columns 10.9 / 8.2. Six and eight CTAs to a tile gained nothing over four; widths of 160 to 224, whose warps meet
// two scales of W, lost 5 to 50 %.
static void planFp8(const ncclTpContext* tp, TpGemmArgs* a, int* width, int* grid) {
  const int blocks = a->K / 128;
  const int only = paramTpFp8Width() == 128 || paramTpFp8Width() == 256 ? (int)paramTpFp8Width() : 0;
  float best = 0.0f;
  *width = 0;
  for (int w : {256, 128}) {
    const int tiles = a->M / 128 * (a->N / w);
    const int forced = (int)std::max<int64_t>(0, std::min<int64_t>(paramTpFp8Split(), kTpMaxSplit)), most = forced ? forced : w == 256 ? 2 : 4;
    if (only && only != w) continue;
    for (int s = forced ? std::max(1, std::min(most, blocks)) : 1; s <= std::min(most, blocks); ++s) {
      if (s > 1 && !forced && tiles > tp->fp8Clusters[s]) break;
      const int waves = (tiles + tp->smCount - 1) / tp->smCount, share = (blocks + s - 1) / s;
      const float us = waves * (w == 256 ? 3.0f + (s > 1 ? 0.53f : 0.50f) * share : 2.4f + 0.38f * share) + (s > 1 ? 3.7f : 0.0f);
      if (*width && us > 0.97f * best) continue;   // what is simpler stays where the others are hardly faster
      best = us;
      *width = w;
      a->splitK = s;
      *grid = s > 1 ? tiles * s : std::min(tp->smCount, tiles);
    }
  }
}

static ncclResult_t checkShapeFp8(int M, int N, int K, int n) {
  if (M <= 0 || N <= 0 || K <= 0 || M % (128 * n) || N % 256 || K % 128) {
    WARN("fp8 tensor-parallel GEMM: M=%d must be a multiple of %d, N=%d of 256, K=%d of 128", M, 128 * n, N, K);
    return ncclInvalidArgument;
  }
  return ncclSuccess;
}

extern "C" {

ncclResult_t ncclTpQuantizeFp8(ncclTp_t tp, const void* x, void* q, float* scales, int rows, int K, int blockRows, cudaStream_t stream) {
  if (!tp || !x || !q || !scales || rows <= 0 || K <= 0 || K % 128 || (blockRows != 1 && blockRows != 128)) return ncclInvalidArgument;
  if (blockRows == 128 && rows % 128) return ncclInvalidArgument;
  if (((uintptr_t)x & 7) || ((uintptr_t)q & 3)) return ncclInvalidArgument;
  void* args[5] = {(void*)&x, &q, &scales, &rows, &K};
  int gx = 0, gy = 0;
  tpQuantRowsWideGrid(rows, K, &gx, &gy);
  // A CTA of the wide kernel covers 16 K blocks: with fewer than four most of its threads idle. Kernel times of the wide kernel
  // over the other: 8192 rows K = 128 4.5 / 2.8 us, 256 4.7 / 4.0, 384 4.8 / 5.2, 512 5.0 / 6.1; 32768 rows 13.5 / 6.1, 14.1 / 10.4,
  // 14.6 / 14.3, 15.0 / 17.9.
  if (blockRows == 1 && K >= 512 && !(((uintptr_t)x | (uintptr_t)q) & 15) && gy <= 65535) {
    return launchTp(tp, tpQuantRowsWideKernelFn(), dim3(gx, gy), 256, 0, args, true, 1, stream);
  } else if (blockRows == 1) {
    size_t warps = (size_t)rows * (K / 128);
    int ctas = (int)std::min<size_t>((warps + 7) / 8, (size_t)tp->smCount * 16);
    return launchTp(tp, tpQuantRowsKernelFn(), dim3(std::max(ctas, 1)), 256, 0, args, true, 1, stream);
  } else {
    int blocks = (rows / 128) * (K / 128);
    return launchTp(tp, tpQuantBlocksKernelFn(), dim3(std::min(blocks, tp->smCount * 8)), 256, 0, args, true, 1, stream);
  }
}

ncclResult_t ncclTpGemmFp8(ncclTp_t tp, const void* A, const float* scaleA, const void* W, const float* scaleW, void* C, int M, int N, int K, cudaStream_t stream) {
  if (!tp || !A || !W || !C || !scaleA || !scaleW) return ncclInvalidArgument;
  NCCLCHECK(checkShapeFp8(M, N, K, 1));
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.C = C; a.ldc = N; a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_STORE;
  a.rank = tp->comm->rank; a.nRanks = tp->comm->nRanks;
  a.scaleA = scaleA; a.scaleW = scaleW;
  fillSyncTp(tp->comm, &a.sync);
  int width, grid;
  planFp8(tp, &a, &width, &grid);
  return launchGemmFp8(tp, A, W, &a, grid, stream, width);
}

ncclResult_t ncclTpGemmReduceScatterFp8(ncclTp_t tp, const void* A, const float* scaleA, const void* W, const float* scaleW, void* out, int M, int N, int K,
                                        cudaStream_t stream) {
  if (!tp || !A || !W || !out || !scaleA || !scaleW) return ncclInvalidArgument;
  ncclComm* comm = tp->comm;
  const int n = comm->nRanks;
  NCCLCHECK(checkShapeFp8(M, N, K, n));
  NCCLCHECK(devPlaneCheckStatus(comm));
  if (n > 1) NCCLCHECK(devPlaneOrderStreams(comm, stream));   // the fused kernels use the communicator's barrier slots: one kernel of a communicator at a time
  if (n == 1) return ncclTpGemmFp8(tp, A, scaleA, W, scaleW, out, M, N, K, stream);
  const size_t need = (size_t)M * N * 2;
  if (need > tp->accumBytes) { WARN("ncclTpGemmReduceScatterFp8: %d x %d exceeds the context's staging window", M, N); return ncclInvalidArgument; }
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_REDUCE;
  a.rank = comm->rank; a.nRanks = n;
  a.scaleA = scaleA; a.scaleW = scaleW;
  for (int p = 0; p < n; ++p) a.partial[p] = tp->accumWin->host.peerPtr[p];
  fillSyncTp(comm, &a.sync);
  int tiles = (M / 128) * (N / 256);
  NCCLCHECK(launchGemmFp8(tp, A, W, &a, std::min(tp->smCount, tiles), stream));
  size_t count = (size_t)(M / n) * N;
  int ctas = (int)std::min<size_t>((count / 8 + 255) / 256, (size_t)tp->smCount * 8);
  const void* staged = tp->accum;
  int nSources = n;
  void* args[4] = {(void*)&staged, &out, &count, &nSources};
  CUDACHECK(cudaLaunchKernel(tpReduceKernelFn(), dim3(ctas), dim3(256), args, 0, stream));
  if (comm->devPlane) comm->devPlane->launches++;
  return ncclSuccess;
}

ncclResult_t ncclTpAllocGatheredFp8(ncclTp_t tp, size_t rows, size_t cols, void** q, float** scales) {
  if (!tp || !q || !scales || cols % 128) return ncclInvalidArgument;
  // one window: rows x cols bytes of e4m3, then cols/128 x rows fp32 scales
  const size_t qBytes = (rows * cols + 255) / 256 * 256;
  const size_t bytes = qBytes + (cols / 128) * rows * sizeof(float);
  void* p = nullptr;
  NCCLCHECK(memAlloc(&p, bytes, tp->comm->cudaDev));
  SymWindow* w = nullptr;
  if (tp->comm->nRanks > 1) {
    NCCLCHECK(symWindowRegister(tp->comm, p, bytes, &w, NCCL_WIN_COLL_SYMMETRIC));
    if (!w->symmetric) { WARN("ncclTpAllocGatheredFp8: window could not be mapped by the peers"); return ncclInternalError; }
  }
  tp->gathered[p] = w;
  // activations belong to the caller: a suspend saves them to host memory and a resume brings them back
  memTrack(tp->comm, p, bytes, MEM_OFFLOAD, "gathered activations (fp8)", tp->comm->nRanks > 1 ? &tp->gathered[p] : nullptr, NCCL_WIN_COLL_SYMMETRIC);
  *q = p;
  *scales = (float*)((char*)p + qBytes);
  return ncclSuccess;
}

ncclResult_t ncclTpAllGatherGemmFp8(ncclTp_t tp, void* gatheredA, const void* W, const float* scaleW, void* C, int M, int N, int K, cudaStream_t stream) {
  if (!tp || !gatheredA || !W || !scaleW || !C) return ncclInvalidArgument;
  ncclComm* comm = tp->comm;
  const int n = comm->nRanks;
  NCCLCHECK(checkShapeFp8(M, N, K, n));
  NCCLCHECK(devPlaneCheckStatus(comm));
  const size_t scaleOffset = ((size_t)M * K + 255) / 256 * 256;
  if (n == 1) return ncclTpGemmFp8(tp, gatheredA, (const float*)((char*)gatheredA + scaleOffset), W, scaleW, C, M, N, K, stream);
  auto it = tp->gathered.find(gatheredA);
  if (it == tp->gathered.end() || !it->second) { WARN("ncclTpAllGatherGemmFp8: the activation buffer must come from ncclTpAllocGatheredFp8"); return ncclInvalidArgument; }
  if ((size_t)(M / 128) > tp->maxBlocks) { WARN("ncclTpAllGatherGemmFp8: M=%d exceeds the context's row limit", M); return ncclInvalidArgument; }
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.C = C; a.ldc = N; a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_GATHER;
  a.rank = comm->rank; a.nRanks = n;
  for (int p = 0; p < n; ++p) a.peerA[p] = it->second->host.peerPtr[p];
  a.scaleOffset = scaleOffset;
  a.scaleW = scaleW;
  a.blockFlags = tp->blockFlags;
  a.flagEpoch = ++tp->epoch;
  int commCtas = tpCommCtas(tp, n);
  a.gemmCtas = tp->smCount - commCtas;
  fillSyncTp(comm, &a.sync);
  return launchGemmFp8(tp, gatheredA, W, &a, tp->smCount, stream);
}

ncclResult_t ncclTpCreate(ncclComm_t comm, size_t maxRows, size_t maxCols, ncclTp_t* out) {
  if (!out) return ncclInvalidArgument;
  *out = nullptr;
  if (!commValid(comm) || comm->hostOnly) { WARN("ncclTpCreate needs a GPU communicator"); return ncclInvalidArgument; }
  NCCLCHECK(commEnsureReady(comm));
  if (comm->nRanks > 1 && !comm->lsaAll) { WARN("ncclTpCreate: ranks must be able to map each other's memory"); return ncclInvalidUsage; }
  if (comm->compCap < 100) { WARN("ncclTpCreate: the fused GEMM kernels need compute capability 10.0 (found %d)", comm->compCap); return ncclInvalidUsage; }
  ncclTpContext* tp = new ncclTpContext;
  tp->comm = comm;
  int cur = -1;
  CUDACHECK(cudaGetDevice(&cur));
  if (cur != comm->cudaDev) CUDACHECK(cudaSetDevice(comm->cudaDev));
  CUDACHECK(cudaDeviceGetAttribute(&tp->smCount, cudaDevAttrMultiProcessorCount, comm->cudaDev));
  // function attributes are per device: set them here, with this context's device current, not once per process
  for (int width : kTpWidths) CUDACHECK(cudaFuncSetAttribute(tpGemmKernelFn(width), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tpGemmSmemBytes()));
  for (int width : {128, 256}) CUDACHECK(cudaFuncSetAttribute(tpGemmSplitKernelFn(width), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tpGemmSplitSmemBytes()));
  CUDACHECK(cudaFuncSetAttribute(tpGemmFp8KernelFn(true, 256, false), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tpGemmFp8SmemBytes()));
  for (int width : {128, 256})
    for (bool split : {false, true})
      CUDACHECK(cudaFuncSetAttribute(tpGemmFp8KernelFn(false, width, split), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tpGemmFp8SmemBytes()));
  {
    // how many clusters of two CTAs of the pair kernel the device can hold at once: the grid never exceeds it,
    // because its CTAs wait for one another (comm CTAs, cross-GPU barriers)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tp->smCount & ~1);
    cfg.blockDim = dim3(tpGemmPairThreads());
    cfg.dynamicSmemBytes = tpGemmPairSmemBytes();
    int clusters = 0;
    bool pairsFit = true;
    for (int width : kTpWidths)
      if (width >= kTpPairWidth) pairsFit = pairsFit && cudaFuncSetAttribute(tpGemmPairKernelFn(width), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tpGemmPairSmemBytes()) == cudaSuccess;
    if (pairsFit && cudaOccupancyMaxActiveClusters(&clusters, tpGemmPairKernelFn(256), &cfg) == cudaSuccess)
      tp->pairClusters = std::min(clusters, tp->smCount / 2);
    else
      (void)cudaGetLastError();
    cudaLaunchAttribute cluster;
    cfg.attrs = &cluster;
    cfg.numAttrs = 1;
    for (int size = 2; size <= kTpMaxSplit; ++size) {
      clusterAttribute(&cluster, size);
      cfg.gridDim = dim3(tp->smCount / size * size);
      cfg.blockDim = dim3(tpGemmSplitThreads());
      cfg.dynamicSmemBytes = tpGemmSplitSmemBytes();
      if (cudaOccupancyMaxActiveClusters(&clusters, tpGemmSplitKernelFn(256), &cfg) == cudaSuccess) tp->splitClusters[size] = clusters;
      else (void)cudaGetLastError();
      // both widths have the same threads, registers and shared memory
      cfg.blockDim = dim3(tpGemmFp8Threads());
      cfg.dynamicSmemBytes = tpGemmFp8SmemBytes();
      if (cudaOccupancyMaxActiveClusters(&clusters, tpGemmFp8KernelFn(false, 256, true), &cfg) == cudaSuccess) tp->fp8Clusters[size] = clusters;
      else (void)cudaGetLastError();
    }
    INFO(SUB_INIT, "tensor-parallel GEMM: %d SMs, %d resident CTA pairs", tp->smCount, tp->pairClusters);
  }
  const int n = comm->nRanks;
  tp->accumBytes = n > 1 ? maxRows * maxCols * 2 : 0;   // bf16 staging: one [maxRows / n, maxCols] slot per source rank
  if (tp->accumBytes) {
    NCCLCHECK(memAlloc((void**)&tp->accum, tp->accumBytes, comm->cudaDev));
    if (n > 1) {
      NCCLCHECK(symWindowRegister(comm, tp->accum, tp->accumBytes, &tp->accumWin, NCCL_WIN_COLL_SYMMETRIC));
      if (!tp->accumWin->symmetric) { WARN("ncclTpCreate: accumulation window could not be mapped by the peers"); return ncclInternalError; }
    }
    memTrack(comm, tp->accum, tp->accumBytes, MEM_SCRATCH, "tensor-parallel partial sums", n > 1 ? &tp->accumWin : nullptr, NCCL_WIN_COLL_SYMMETRIC);
  }
  tp->maxBlocks = maxRows / 128 + 1;
  CUDACHECK(cudaMalloc(&tp->blockFlags, tp->maxBlocks * sizeof(uint32_t)));
  CUDACHECK(cudaMemset(tp->blockFlags, 0, tp->maxBlocks * sizeof(uint32_t)));
  if (cur != comm->cudaDev) cudaSetDevice(cur);
  *out = tp;
  return ncclSuccess;
}

ncclResult_t ncclTpDestroy(ncclTp_t tp) {
  if (!tp) return ncclSuccess;
  cudaDeviceSynchronize();
  for (auto& kv : tp->gathered) {
    if (kv.second) symWindowDeregister(tp->comm, kv.second);
    memFree(kv.first);
  }
  if (tp->accum) memUntrack(tp->comm, tp->accum);
  for (auto& kv : tp->gathered) memUntrack(tp->comm, kv.first);
  if (tp->accumWin) symWindowDeregister(tp->comm, tp->accumWin);
  if (tp->accum) memFree(tp->accum);
  if (tp->blockFlags) cudaFree(tp->blockFlags);
  delete tp;
  return ncclSuccess;
}

ncclResult_t ncclTpAllocGathered(ncclTp_t tp, size_t rows, size_t cols, void** ptr) {
  if (!tp || !ptr) return ncclInvalidArgument;
  void* p = nullptr;
  NCCLCHECK(memAlloc(&p, rows * cols * 2, tp->comm->cudaDev));
  SymWindow* w = nullptr;
  if (tp->comm->nRanks > 1) {
    NCCLCHECK(symWindowRegister(tp->comm, p, rows * cols * 2, &w, NCCL_WIN_COLL_SYMMETRIC));
    if (!w->symmetric) { WARN("ncclTpAllocGathered: window could not be mapped by the peers"); return ncclInternalError; }
  }
  tp->gathered[p] = w;
  memTrack(tp->comm, p, rows * cols * 2, MEM_OFFLOAD, "gathered activations", tp->comm->nRanks > 1 ? &tp->gathered[p] : nullptr, NCCL_WIN_COLL_SYMMETRIC);
  *ptr = p;
  return ncclSuccess;
}

ncclResult_t ncclTpFreeGathered(ncclTp_t tp, void* ptr) {
  if (!tp) return ncclInvalidArgument;
  auto it = tp->gathered.find(ptr);
  if (it == tp->gathered.end()) return ncclInvalidArgument;
  cudaDeviceSynchronize();
  memUntrack(tp->comm, ptr);
  if (it->second) symWindowDeregister(tp->comm, it->second);
  memFree(ptr);
  tp->gathered.erase(it);
  return ncclSuccess;
}

ncclResult_t ncclTpGemm(ncclTp_t tp, const void* A, const void* W, void* C, int M, int N, int K, cudaStream_t stream) {
  if (!tp || !A || !W || !C) return ncclInvalidArgument;
  NCCLCHECK(checkShape(M, N, K, 1));
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.C = C; a.ldc = N; a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_STORE;
  a.rank = tp->comm->rank; a.nRanks = tp->comm->nRanks;
  fillSyncTp(tp->comm, &a.sync);
  return launchGemm(tp, A, W, &a, stream);
}

ncclResult_t ncclTpGemmReduceScatter(ncclTp_t tp, const void* A, const void* W, void* out, int M, int N, int K, cudaStream_t stream) {
  if (!tp || !A || !W || !out) return ncclInvalidArgument;
  ncclComm* comm = tp->comm;
  const int n = comm->nRanks;
  NCCLCHECK(checkShape(M, N, K, n));
  NCCLCHECK(devPlaneCheckStatus(comm));
  if (n > 1) NCCLCHECK(devPlaneOrderStreams(comm, stream));   // the fused kernels use the communicator's barrier slots: one kernel of a communicator at a time
  if (n == 1) return ncclTpGemm(tp, A, W, out, M, N, K, stream);
  const size_t need = (size_t)M * N * 2;
  if (need > tp->accumBytes) { WARN("ncclTpGemmReduceScatter: %d x %d exceeds the context's staging window", M, N); return ncclInvalidArgument; }
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_REDUCE;
  a.rank = comm->rank; a.nRanks = n;
  for (int p = 0; p < n; ++p) a.partial[p] = tp->accumWin->host.peerPtr[p];
  fillSyncTp(comm, &a.sync);
  NCCLCHECK(launchGemm(tp, A, W, &a, stream));
  // kernel completion implies that every rank's partial tiles have landed in this rank's staging slots
  size_t count = (size_t)(M / n) * N;
  int ctas = (int)std::min<size_t>((count / 8 + 255) / 256, (size_t)tp->smCount * 8);
  const void* staged = tp->accum;
  int nSources = n;
  void* args[4] = {(void*)&staged, &out, &count, &nSources};
  CUDACHECK(cudaLaunchKernel(tpReduceKernelFn(), dim3(ctas), dim3(256), args, 0, stream));
  if (comm->devPlane) comm->devPlane->launches++;
  return ncclSuccess;
}

ncclResult_t ncclTpAllGatherGemm(ncclTp_t tp, void* gatheredA, const void* W, void* C, int M, int N, int K, cudaStream_t stream) {
  if (!tp || !gatheredA || !W || !C) return ncclInvalidArgument;
  ncclComm* comm = tp->comm;
  const int n = comm->nRanks;
  NCCLCHECK(checkShape(M, N, K, n));
  NCCLCHECK(devPlaneCheckStatus(comm));
  if (n > 1) NCCLCHECK(devPlaneOrderStreams(comm, stream));   // the fused kernels use the communicator's barrier slots: one kernel of a communicator at a time
  if (n == 1) return ncclTpGemm(tp, gatheredA, W, C, M, N, K, stream);
  auto it = tp->gathered.find(gatheredA);
  if (it == tp->gathered.end() || !it->second) { WARN("ncclTpAllGatherGemm: the activation buffer must come from ncclTpAllocGathered"); return ncclInvalidArgument; }
  if ((size_t)(M / 128) > tp->maxBlocks) { WARN("ncclTpAllGatherGemm: M=%d exceeds the context's row limit", M); return ncclInvalidArgument; }
  TpGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.C = C; a.ldc = N; a.M = M; a.N = N; a.K = K;
  a.mode = TP_MODE_GATHER;
  a.rank = comm->rank; a.nRanks = n;
  for (int p = 0; p < n; ++p) a.peerA[p] = it->second->host.peerPtr[p];
  a.blockFlags = tp->blockFlags;
  a.flagEpoch = ++tp->epoch;
  fillSyncTp(comm, &a.sync);
  return launchGemm(tp, gatheredA, W, &a, stream);
}

}  // extern "C"
