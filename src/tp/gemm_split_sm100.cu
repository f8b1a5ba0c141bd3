// Tensor-parallel bf16 GEMM for outputs with few tiles (decoding, narrow layers): the K dimension of a 128 x 256 tile is split
// over a cluster of S CTAs, so that S times as many SMs stream the operands; plain C = A * W^T, no communication.
//
// Bound by memory when M is small (the weights are read once): at 128 x 8192 x 8192 one CTA per tile left 116 of 148 SMs idle
// and took 52 us for 138 MB, clusters of four take 32. Every CTA runs the producer / MMA roles of gemm_sm100.cu over its share of the K blocks, one tile
// per CTA. Then the cluster adds up: column chunk c (32 columns) belongs to CTA c % S; every CTA copies its fp32 partial sums
// of the other CTAs' chunks from tensor memory into their shared memory (the operand ring is free by then), and after a
// cluster barrier the owner adds them in the order of the K shares, its own among them, rounds once and stores. No workspace,
// and the same result whatever the schedule.
// Waits are bounded and reported as in the other kernels.
#include "gemm_roles.cuh"

namespace b200 {

using namespace sm100;

namespace {
constexpr int BM = kTpBM, BK = kTpBK, UMMA_K = 16;
constexpr int kThreads = 192;
constexpr uint32_t kStageABytes = BM * BK * 2;
constexpr size_t kRingBytes = 4 * (BM + 256) * BK * 2;   // operand ring: as many stages as fit
constexpr size_t kSmemBytes = 1024 + kRingBytes + 256;
constexpr int kChunk = 32;
constexpr uint32_t kChunkBytes = BM * kChunk * 4;
// chunks of one owner x shares of the others, for every width and cluster size
constexpr bool fits() {
  for (int w : {128, 256})
    for (int s = 2; s <= kTpMaxSplit; ++s)
      if ((size_t)((w / kChunk + s - 1) / s) * (s - 1) * kChunkBytes > kRingBytes) return false;
  return true;
}
static_assert(fits(), "partial sums must fit the operand ring");

__device__ __forceinline__ void stSharedCluster16(uint32_t clusterAddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(clusterAddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
}  // namespace

// BN: width of the tiles, 256 or 128
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
tpGemmSplitKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ TpGemmArgs a) {
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  constexpr uint32_t kStageBBytes = BN * BK * 2, kStageBytes = kStageABytes + kStageBBytes;
  constexpr int STAGES = kRingBytes / kStageBytes, kChunks = BN / kChunk;
  uint8_t* ctrl = smem + kRingBytes;
  uint64_t* fullBar = (uint64_t*)ctrl;            // [STAGES]
  uint64_t* emptyBar = fullBar + STAGES;          // [STAGES]
  uint64_t* accFull = emptyBar + STAGES;
  uint32_t* tmemSlot = (uint32_t*)(accFull + 1);
  volatile uint32_t* abortFlag = tmemSlot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int share = (int)clusterCtaRank(), S = a.splitK;
  const int tile = blockIdx.x / S;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbarInit(smemAddr(&fullBar[s]), 1); mbarInit(smemAddr(&emptyBar[s]), 1); }
    mbarInit(smemAddr(accFull), 1);
    *abortFlag = 0;
    mbarInitFence();
    prefetchTensorMap(&tmA);
    prefetchTensorMap(&tmB);
  }
  if (warp == 1) {
    tmemAlloc(smemAddr(tmemSlot), BN);
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;
  pdlEnter();   // the set-up above overlaps the end of the kernel before; operands and results are touched behind it
  const uint32_t ring = smemAddr(smem);

  const int tilesN = a.N / BN;
  const int mBlk = tile / tilesN, nBlk = tile % tilesN;
  const int kBlocks = a.K / BK;
  const int k0 = kBlocks * share / S, k1 = kBlocks * (share + 1) / S;   // the host keeps S <= kBlocks: never empty
  const uint32_t smemA0 = ring, smemB0 = ring + STAGES * kStageABytes;
  auto fail = [&](uint32_t what) {
    *abortFlag = 1;
    tpReportTimeout(a, WAIT_TILE, what);
  };

  if (warp == 0) {
    if (electOne()) {
      uint32_t armed = 0, armedPhase = 0;   // per stage: a copy was issued, and for which phase of its barrier
      for (int kb = k0; kb < k1; ++kb) {
        const int i = kb - k0, s = i % STAGES;
        const uint32_t ph = (i / STAGES) & 1;
        if (!mbarWait(smemAddr(&emptyBar[s]), ph ^ 1)) { fail(1000 + s); break; }
        const uint32_t fb = smemAddr(&fullBar[s]);
        mbarExpectTx(fb, kStageBytes);
        tmaLoad2d(smemA0 + s * kStageABytes, &tmA, kb * BK, mBlk * BM, fb);
        tmaLoad2d(smemB0 + s * kStageBBytes, &tmB, kb * BK, nBlk * BN, fb);
        armed |= 1u << s;
        armedPhase = (armedPhase & ~(1u << s)) | (ph << s);
      }
      if (*abortFlag)
        for (int s = 0; s < STAGES; ++s)
          if ((armed >> s) & 1u) mbarWait(smemAddr(&fullBar[s]), (armedPhase >> s) & 1u, 1u << 20);
    }
  } else if (warp == 1) {
    if (electOne()) {
      const uint32_t idesc = umInstrBf16(BM, BN);
      bool bad = false;
      for (int kb = k0; kb < k1; ++kb) {
        const int i = kb - k0, s = i % STAGES;
        const uint32_t ph = (i / STAGES) & 1;
        if (!mbarWait(smemAddr(&fullBar[s]), ph)) { fail(3000 + s); bad = true; break; }
        tcFenceAfter();
        const uint32_t aAddr = smemA0 + s * kStageABytes, bAddr = smemB0 + s * kStageBBytes;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          ummaBf16(tmemBase, umDescK128(aAddr + k * UMMA_K * 2), umDescK128(bAddr + k * UMMA_K * 2), idesc, (i | k) != 0);
        ummaCommit(smemAddr(&emptyBar[s]));
      }
      if (!bad) ummaCommit(smemAddr(accFull));
    }
  } else {
    if (!mbarWait(smemAddr(accFull), 0) && lane == 0) fail(4000);
  }
  __syncwarp();
  tcFenceBefore();
  // every CTA's MMAs have read their operands (accFull follows them all): the rings are free for partial sums
  clusterSync();
  tcFenceAfter();

  const int q = warp & 3, row = q * 32 + lane;
  const uint32_t tBase = tmemBase + ((uint32_t)(q * 32) << 16);
  // slot of (chunk of this owner, share of another CTA): 16-byte pieces [column / 4][row], so a warp writes and reads 512
  // contiguous bytes
  auto slotOf = [&](int chunk, int from, int owner) {
    const int others = from < owner ? from : from - 1;
    return (uint32_t)((chunk / S) * (S - 1) + others) * kChunkBytes + (uint32_t)row * 16;
  };
  if (warp >= 2) {
    for (int c = 0; c < kChunks; ++c) {
      const int owner = c % S;
      if (owner == share) continue;
      uint32_t r[32];
      tmemLd32(tBase + c * kChunk, r);
      tmemLdWait32(r);
      const uint32_t dst = mapaShared(ring + slotOf(c, share, owner), (uint32_t)owner);
#pragma unroll
      for (int j = 0; j < 8; ++j) stSharedCluster16(dst + j * (BM * 16), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    }
  }
  __syncwarp();
  clusterSync();
  if (warp >= 2) {
    __nv_bfloat16* out = (__nv_bfloat16*)a.C + (size_t)(mBlk * BM + row) * a.ldc + (size_t)nBlk * BN;
    for (int c = share; c < kChunks; c += S) {
      uint32_t own[32];
      tmemLd32(tBase + c * kChunk, own);
      tmemLdWait32(own);
      float sum[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[j] = 0.0f;
      for (int from = 0; from < S; ++from) {
        if (from == share) {
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] += __uint_as_float(own[j]);
        } else {
          const uint8_t* src = smem + slotOf(c, from, share);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = *(const float4*)(src + j * (BM * 16));
            sum[4 * j] += v.x;
            sum[4 * j + 1] += v.y;
            sum[4 * j + 2] += v.z;
            sum[4 * j + 3] += v.w;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 o;
        __nv_bfloat162* p = (__nv_bfloat162*)&o;
#pragma unroll
        for (int k = 0; k < 4; ++k) p[k] = __floats2bfloat162_rn(sum[8 * j + 2 * k], sum[8 * j + 2 * k + 1]);
        *(uint4*)(out + c * kChunk + j * 8) = o;
      }
    }
  }
  tcFenceBefore();
  __syncthreads();
  if (warp == 1) {
    tcFenceAfter();
    tmemDealloc(tmemBase, BN);
  }
}

const void* tpGemmSplitKernelFn(int width) { return width == 128 ? (const void*)tpGemmSplitKernel<128> : (const void*)tpGemmSplitKernel<256>; }
size_t tpGemmSplitSmemBytes() { return kSmemBytes; }
int tpGemmSplitThreads() { return kThreads; }

}  // namespace b200
