// Tensor-parallel bf16 GEMM for outputs with few tiles (decoding, narrow layers): the K dimension is cut into P shares with a sum each,
// which a cluster of S CTAs takes tile by tile, so that S times as many SMs stream the operands; plain C = A * W^T, no communication.
//
// Bound by memory when M is small (the weights are read once): at 128 x 8192 x 8192 one CTA per 128 x 256 tile left 116 of 148 SMs idle
// and took 52 us for 138 MB. Every CTA runs the producer / MMA roles of gemm_sm100.cu over the K blocks of its shares, one tile per CTA. A tile
// of 256 columns has a CTA to each share (P = S); of 128 columns a CTA takes up to four, with an accumulator each: twice the tiles, half
// the CTAs to a tile. P is the same for both widths (tp.cc), so that the width changes neither the sums nor their order.
// Then the cluster adds up: column chunk c (32 columns) belongs to CTA c % S; every CTA copies its fp32 partial sums of the other CTAs'
// chunks from tensor memory into their shared memory, and after a cluster barrier the owner adds them in the order of the K shares, its own
// among them, rounds once and stores. The sums of a CTA's last share go into the owner's operand ring, which is free by then; those of the
// shares before it ("early") into a zone behind the ring, while the next share is multiplied: an exchange of all sums at the end took 4 us
// longer at 128 x 4096 x 4096. No workspace, and the same result whatever the schedule.
// Waits are bounded and reported as in the other kernels.
#include <algorithm>

#include "gemm_roles.cuh"

namespace b200 {

using namespace sm100;

namespace {
constexpr int BM = kTpBM, BK = kTpBK, UMMA_K = 16;
constexpr int kThreads = 192;
constexpr uint32_t kStageABytes = BM * BK * 2;
constexpr size_t kRingBytes = 4 * (BM + 256) * BK * 2;   // operand ring, as many stages as fit, and the zone of the early sums
constexpr size_t kSmemBytes = 1024 + kRingBytes + 256;
constexpr int kChunk = 32;
constexpr uint32_t kChunkBytes = BM * kChunk * 4;
constexpr int kMaxStages = 6;
constexpr int tmemColsOf(int width) { return width == 256 ? 256 : 512; }   // one accumulator, or up to four
}  // namespace

int tpGemmSplitPlan(TpGemmArgs* a, int width) {
  const int S = a->splitK, P = a->shares;
  for (int c = 0; c <= S; ++c) a->firstShare[c] = (uint8_t)(P * c / S);   // as even as they go
  int most = 0;
  for (int c = 0; c < S; ++c) {
    const int chunks = (width / kChunk - c + S - 1) / S, own = a->firstShare[c + 1] - a->firstShare[c];
    a->earlySums[c] = (uint8_t)(P - S - (own - 1));
    if (chunks > 0) most = std::max(most, chunks * a->earlySums[c]);
  }
  a->early = most;
  return most;
}

namespace {
// last sums of one owner's chunks from the other CTAs, for every width and cluster size
constexpr bool fits() {
  for (int w : {128, 256})
    for (int s = 2; s <= kTpMaxSplit; ++s)
      if ((size_t)((w / kChunk + s - 1) / s) * (s - 1) * kChunkBytes > kRingBytes - (w == 128 ? kTpMaxEarly * kChunkBytes : 0)) return false;
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
  constexpr int kChunks = BN / kChunk;
  static_assert(kRingBytes / kStageBytes <= kMaxStages, "not enough barriers");
  static_assert((kRingBytes - kTpMaxEarly * kChunkBytes) / kStageBytes >= 4 || BN != 128, "too few stages beside the early sums");
  uint8_t* ctrl = smem + kRingBytes;
  uint64_t* fullBar = (uint64_t*)ctrl;            // [kMaxStages]
  uint64_t* emptyBar = fullBar + kMaxStages;      // [kMaxStages]
  uint64_t* accFull = emptyBar + kMaxStages;      // [kTpMaxOwnShares]
  uint32_t* tmemSlot = (uint32_t*)(accFull + kTpMaxOwnShares);
  volatile uint32_t* abortFlag = tmemSlot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = (int)clusterCtaRank(), S = a.splitK, P = a.shares;
  const int tile = blockIdx.x / S;
  const uint32_t earlyAt = (uint32_t)kRingBytes - a.early * kChunkBytes;
  const int STAGES = earlyAt / kStageBytes;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbarInit(smemAddr(&fullBar[s]), 1); mbarInit(smemAddr(&emptyBar[s]), 1); }
    for (int j = 0; j < kTpMaxOwnShares; ++j) mbarInit(smemAddr(&accFull[j]), 1);
    *abortFlag = 0;
    mbarInitFence();
    prefetchTensorMap(&tmA);
    prefetchTensorMap(&tmB);
  }
  if (warp == 1) {
    tmemAlloc(smemAddr(tmemSlot), tmemColsOf(BN));
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  if (a.early) clusterSync();   // early sums go into the shared memory of CTAs that have begun
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;
  pdlEnter();   // the set-up above overlaps the end of the kernel before; operands and results are touched behind it
  const uint32_t ring = smemAddr(smem);

  const int tilesN = a.N / BN;
  const int mBlk = tile / tilesN, nBlk = tile % tilesN;
  const int kBlocks = a.K / BK;
  const int p0 = a.firstShare[cta], p1 = a.firstShare[cta + 1];   // shares of this CTA
  // the host keeps S <= P <= kBlocks: neither a CTA nor a share is empty
  auto blockOf = [&](int p) { return kBlocks * p / P; };
  const uint32_t smemA0 = ring, smemB0 = ring + STAGES * kStageABytes;
  auto fail = [&](uint32_t what) {
    *abortFlag = 1;
    tpReportTimeout(a, WAIT_TILE, what);
  };

  const int q = warp & 3, row = q * 32 + lane;
  const uint32_t tBase = tmemBase + ((uint32_t)(q * 32) << 16);
  // Where an owner finds the sums of share p (of CTA `from`, whose last share is `last`) for its n-th chunk: 16-byte pieces
  // [column / 4][row], so a warp writes and reads 512 contiguous bytes
  auto slotOf = [&](int n, int p, int from, bool last, int owner) {
    const bool behind = from > owner;   // the owner's own shares have no slots
    const int slot = last ? n * (S - 1) + from - behind : n * a.earlySums[owner] + p - from - (behind ? a.firstShare[owner + 1] - a.firstShare[owner] - 1 : 0);
    return (last ? 0 : earlyAt) + slot * kChunkBytes + (uint32_t)row * 16;
  };
  // share p's sums of the other CTAs' chunks
  auto handOver = [&](int p) {
    const bool last = p + 1 == p1;
    int owner = 0, n = 0;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      if (owner != cta) {
        uint32_t r[32];
        tmemLd32(tBase + (p - p0) * BN + c * kChunk, r);
        const uint32_t dst = mapaShared(ring + slotOf(n, p, cta, last, owner), (uint32_t)owner);
        tmemLdWait32(r);
#pragma unroll
        for (int j = 0; j < 8; ++j) stSharedCluster16(dst + j * (BM * 16), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
      if (++owner == S) { owner = 0; ++n; }
    }
  };

  if (warp == 0) {
    if (electOne()) {
      uint32_t armed = 0, phases = 0;   // per stage: a copy was issued, and for which phase of its barrier
      int s = 0;
      uint32_t ph = 0;
      for (int kb = blockOf(p0); kb < blockOf(p1); ++kb) {
        if (!mbarWait(smemAddr(&emptyBar[s]), ph ^ 1)) { fail(1000 + s); break; }
        const uint32_t fb = smemAddr(&fullBar[s]);
        mbarExpectTx(fb, kStageBytes);
        tmaLoad2d(smemA0 + s * kStageABytes, &tmA, kb * BK, mBlk * BM, fb);
        tmaLoad2d(smemB0 + s * kStageBBytes, &tmB, kb * BK, nBlk * BN, fb);
        armed |= 1u << s;
        phases = (phases & ~(1u << s)) | (ph << s);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (*abortFlag)
        for (s = 0; s < STAGES; ++s)
          if ((armed >> s) & 1u) mbarWait(smemAddr(&fullBar[s]), (phases >> s) & 1u, 1u << 20);
    }
  } else if (warp == 1) {
    if (electOne()) {
      const uint32_t idesc = umInstrBf16(BM, BN);
      bool bad = false;
      int s = 0;
      uint32_t ph = 0;
      for (int p = p0; p < p1 && !bad; ++p) {
        const uint32_t acc = tmemBase + (p - p0) * BN;
        const int first = blockOf(p), end = blockOf(p + 1);
        for (int kb = first; kb < end; ++kb) {
          if (!mbarWait(smemAddr(&fullBar[s]), ph)) { fail(3000 + s); bad = true; break; }
          tcFenceAfter();
          const uint32_t aAddr = smemA0 + s * kStageABytes, bAddr = smemB0 + s * kStageBBytes;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            ummaBf16(acc, umDescK128(aAddr + k * UMMA_K * 2), umDescK128(bAddr + k * UMMA_K * 2), idesc, kb > first || k > 0);
          ummaCommit(smemAddr(&emptyBar[s]));
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (!bad) ummaCommit(smemAddr(&accFull[p - p0]));
      }
    }
  } else {
    for (int p = p0; p < p1; ++p) {
      if (!__all_sync(~0u, mbarWait(smemAddr(&accFull[p - p0]), 0))) {
        if (lane == 0) fail(4000 + p);
        break;
      }
      tcFenceAfter();
      if (p + 1 < p1) handOver(p);
    }
  }
  __syncwarp();
  tcFenceBefore();
  // every CTA's MMAs have read their operands (the last accFull follows them all): the rings are free for partial sums
  clusterSync();
  tcFenceAfter();
  if (warp >= 2) handOver(p1 - 1);
  __syncwarp();
  clusterSync();
  if (warp >= 2) {
    __nv_bfloat16* out = (__nv_bfloat16*)a.C + (size_t)(mBlk * BM + row) * a.ldc + (size_t)nBlk * BN;
    for (int c = cta, n = 0; c < kChunks; c += S, ++n) {
      float sum[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[j] = 0.0f;
      int from = 0;
      for (int p = 0; p < P; ++p) {
        const bool last = p + 1 == a.firstShare[from + 1];
        if (from == cta) {
          uint32_t own[32];
          tmemLd32(tBase + (p - p0) * BN + c * kChunk, own);
          tmemLdWait32(own);
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] += __uint_as_float(own[j]);
        } else {
          const uint8_t* src = smem + slotOf(n, p, from, last, cta);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = *(const float4*)(src + j * (BM * 16));
            sum[4 * j] += v.x;
            sum[4 * j + 1] += v.y;
            sum[4 * j + 2] += v.z;
            sum[4 * j + 3] += v.w;
          }
        }
        from += last;
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
    tmemDealloc(tmemBase, tmemColsOf(BN));
  }
}

const void* tpGemmSplitKernelFn(int width) { return width == 128 ? (const void*)tpGemmSplitKernel<128> : (const void*)tpGemmSplitKernel<256>; }
size_t tpGemmSplitSmemBytes() { return kSmemBytes; }
int tpGemmSplitThreads() { return kThreads; }

}  // namespace b200
