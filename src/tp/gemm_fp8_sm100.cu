// Block-scaled fp8 (e4m3) tensor-parallel GEMM for sm_100a: C[M,N] = A[M,K] * W[N,K]^T where
// A carries one fp32 scale per row and 128 columns (scaleA[K/128][M]) and W one per 128 x 128
// block (scaleW[K/128][N/128]); accumulation is fp32.
//
// The tensor cores cannot apply fp32 block scales themselves, so accumulation has two levels:
//   level 1  tcgen05.mma kind::f8f6f4 (128xBNx32, BN = 256 or 128) sums one 128-wide K block into
//            a TMEM accumulator; two accumulators alternate block by block;
//   level 2  the epilogue warps read each finished block from TMEM (tcgen05.ld), multiply by
//            scaleA[row] * scaleW[block] and add into fp32 registers, while the tensor cores
//            already work on the next K block in the other accumulator.
// 1920 x 4096 x 7168 57 us with its operands in L2 (59 with weights from memory), 8192 x 8192 x 7168 468 us (2.05 PFLOP/s), against 107 us and 1.2 PFLOP/s of a level 2 that waited for each 32
// columns in turn. What bounds the kernel is the round trip of an accumulator (MMAs, level 2, release) and behind that the operand traffic
// from L2 (48 KiB per K block and SM). So level 2 is a pipeline of its own: 32 columns are fetched while the 32 before them are
// multiplied (packed fp32 pairs), across K blocks too, an accumulator is given back as soon as it is read, and the two scales of the
// next K block are multiplied only when it is there (as one product fetched ahead they held up the block before: 78 us for the first
// shape).
// Plain calls with few tiles take tiles of 128 columns, or a cluster of CTAs to a tile, each with its share of the K blocks, so that
// more SMs work (the rule and its figures are in tp.cc).
// Persistent CTAs of three warpgroups: warp 0 TMA producer (128x128-byte A tiles, BNx128-byte W tiles,
// 128-byte swizzle, ring of four stages, six at 128 columns), warp 1 MMA issuer, warps 4-11 epilogue (each warp owns 32 TMEM
// lanes and one half of the tile's columns: up to 128 fp32 accumulators per thread, for which the first warpgroup hands over its
// registers).
// The fused modes work as in the bf16 kernel (gemm_sm100.cu): REDUCE stores the scaled tile as bf16
// into this rank's slot of the owning rank's staging buffer over NVLink (summed afterwards);
// GATHER has comm CTAs pull remote row blocks with bulk copies and their scales with plain peer
// loads. No load uses cluster multicast; tensor-map TMA loads read local memory only.
// Quantisation kernels for both operand kinds are at the end of the file.
// Every wait is bounded; on expiry the kernel records a status, drains its TMA copies, frees its
// tensor memory and returns.
#include <cuda_fp8.h>

#include "gemm_sm100.cuh"

#include "../kernels/common.cuh"
#include "tp.h"

namespace b200 {

using namespace sm100;

namespace {
constexpr int BM = kTpBM, BK = 128, UMMA_K = 32;
constexpr int kThreads = 384, kEpiWarps = 8;
constexpr uint32_t kTmemCols = 512, kAccCols = 256;   // two accumulators, at fixed columns
constexpr size_t kEpiBufBytes = kEpiWarps * 4096;     // one 32 x 128-byte transpose buffer per epilogue warp
constexpr size_t kRingBytes = 4 * (BM + 256) * BK;    // operand ring: as many stages as fit
constexpr size_t kSmemBytes = 1024 + kRingBytes + 256 + kEpiBufBytes;
constexpr uint32_t kChunkBytes = BM * 32 * 4;         // fp32 partial sums of 32 columns
// partial sums of one owner's chunks from the other shares, for every width and cluster size
constexpr bool exchangeFits() {
  for (int w : {128, 256})
    for (int s = 2; s <= kTpMaxSplit; ++s)
      if ((size_t)((w / 32 + s - 1) / s) * (s - 1) * kChunkBytes > kRingBytes) return false;
  return true;
}
static_assert(exchangeFits(), "partial sums must fit the operand ring");
// registers per thread: 168 at launch; the producer warpgroup keeps 56, the two epilogue warpgroups take 224
constexpr int kRegsLaunch = 168, kRegsProducer = 56, kRegsEpilogue = 224;
static_assert(128 * kRegsProducer + 256 * kRegsEpilogue <= kThreads * kRegsLaunch, "register shares exceed the launch");
__device__ __forceinline__ void stSharedCluster16(uint32_t clusterAddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(clusterAddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
}  // namespace

// FUSED: the modes with a collective. The plain form is compiled without what they keep in registers across the tile loop.
// BN: columns of a tile, 256 or (plain calls with few tiles) 128.
// SPLIT: one tile per cluster of a.splitK CTAs that share its K blocks (see the end of the kernel).
template <bool FUSED, int BN, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
tpGemmFp8Kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ TpGemmArgs a) {
  constexpr uint32_t kStageABytes = BM * BK, kStageBBytes = BN * BK, kStageBytes = kStageABytes + kStageBBytes;
  constexpr int STAGES = kRingBytes / kStageBytes;
  constexpr int kHalf = BN / 2, kChunks = kHalf / 32;   // columns and chunks of 32 columns of an epilogue warp
  // A wait for an accumulator that runs out ends the loop over the K blocks behind the block, whose sums nobody stores. Leaving at once made the
  // compiler move registers: 64 moves per K block and warp beside 64 products (1920 x 4096 x 7168 67.0 us, so 62.1; 8192 x 8192 x 7168 507,
  // 488). Tiles of 128 columns have registers to spare, and shared tiles end anyway: there it cost 1 %, and they leave. The vote on the wait, which is
  // there so that no lane goes on alone, made the loop faster too: 61.5 -> 57.2 and 485 -> 468 us, 4096 x 4096 x 4096 75 -> 71.5.
  constexpr bool kLeave = BN == 128 || SPLIT;
  static_assert(BN == 256 || BN == 128, "a warp's columns lie in one block of W's scales");
  static_assert(!(FUSED && (SPLIT || BN != kTpBN)), "the fused modes use whole tiles");
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t* ctrl = smem + kRingBytes;
  uint64_t* fullBar = (uint64_t*)ctrl;
  uint64_t* emptyBar = fullBar + STAGES;
  uint64_t* accFull = emptyBar + STAGES;
  uint64_t* accEmpty = accFull + 2;
  uint32_t* tmemSlot = (uint32_t*)(accEmpty + 2);
  volatile uint32_t* abortFlag = tmemSlot + 1;
  uint8_t* epiBuf = ctrl + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = a.rank, n = a.nRanks;
  const bool gather = FUSED && a.mode == TP_MODE_GATHER;
  const bool commCta = gather && (int)blockIdx.x >= a.gemmCtas;
  const int share = SPLIT ? (int)clusterCtaRank() : 0, S = SPLIT ? a.splitK : 1;
  const int kBegin = SPLIT ? a.K / BK * share / S : 0;                          // the host keeps S <= K blocks: never empty
  const int kBlocks = (SPLIT ? a.K / BK * (share + 1) / S : a.K / BK) - kBegin;   // of this CTA

  CtaBarrier bar;
  bool ok = true;
  if (FUSED) {
    bar.init(a.sync, rank, n, blockIdx.x);
    ok = bar.sync(false, false);
  }

  if (commCta) {
    // ---- all-gather role: rows (fp8) and their scales, block by block in consumption order
    const int blocksPerRank = a.M / n / BM;
    const size_t blockBytes = (size_t)BM * a.K;
    const int commIdx = blockIdx.x - a.gemmCtas, commN = gridDim.x - a.gemmCtas;
    constexpr int kPipeStages = 6;
    constexpr uint32_t kPipeChunk = 32768;
    static_assert((size_t)kPipeStages * kPipeChunk <= kRingBytes, "copy ring must fit the operand ring");
    uint64_t* pipeBars = fullBar;
    if (threadIdx.x == 0) {
      for (int s = 0; s < kPipeStages; ++s) mbarInit(smemAddr(&pipeBars[s]), 1);
      mbarInitFence();
    }
    __syncthreads();
    uint32_t phaseBits = 0;
    // remote blocks in the order the GEMM consumes them (rank+1 first), dealt round-robin to the comm CTAs
    for (int idx = commIdx; idx < (n - 1) * blocksPerRank && ok; idx += commN) {
      const int src = (rank + 1 + idx / blocksPerRank) % n;
      {
        const int b = idx % blocksPerRank;
        const int mb = src * blocksPerRank + b;
        // scales of these 128 rows: one 512-byte run per K block, plain peer loads by all threads
        const float* sFrom = (const float*)((const char*)a.peerA[src] + a.scaleOffset);
        float* sTo = (float*)((char*)a.peerA[rank] + a.scaleOffset);
        for (int e = threadIdx.x; e < kBlocks * (BM / 4); e += kThreads) {
          const size_t off = (size_t)(e / (BM / 4)) * a.M + (size_t)mb * BM + (size_t)(e % (BM / 4)) * 4;
          st16(sTo + off, ldStream16(sFrom + off));
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          // the rows: bulk copies peer -> shared memory -> local, driven by this one thread
          const char* from = (const char*)a.peerA[src] + (size_t)mb * blockBytes;
          char* to = (char*)a.peerA[rank] + (size_t)mb * blockBytes;
          ok = bulkPipe<kPipeStages, kPipeChunk>(to, from, blockBytes, smemAddr(smem), pipeBars, phaseBits);
          if (ok) {
            fenceProxyAsync();
            __threadfence();
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.blockFlags + mb), "r"(a.flagEpoch) : "memory");
          } else if (a.sync.status[rank] && ldRelaxedSys(a.sync.status[rank]) == DEV_OK) {
            a.sync.status[rank][1] = WAIT_TILE;
            a.sync.status[rank][2] = 5000 + mb;
            a.sync.status[rank][3] = blockIdx.x;
            __threadfence_system();
            stRelaxedSys(a.sync.status[rank], DEV_TIMEOUT);
          }
        }
        ok = __syncthreads_and(ok);
      }
    }
    bar.sync(true, false);
    bar.finish();
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbarInit(smemAddr(&fullBar[s]), 1); mbarInit(smemAddr(&emptyBar[s]), 1); }
    for (int b = 0; b < 2; ++b) { mbarInit(smemAddr(&accFull[b]), 1); mbarInit(smemAddr(&accEmpty[b]), kEpiWarps); }
    *abortFlag = ok ? 0u : 1u;
    mbarInitFence();
    prefetchTensorMap(&tmA);
    prefetchTensorMap(&tmB);
  }
  if (warp == 1) {
    tmemAlloc(smemAddr(tmemSlot), kTmemCols);
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;
  pdlEnter();   // the set-up above overlaps the end of the kernel before; operands and results are touched behind it

  const int tilesN = a.N / BN;
  const int nTiles = (a.M / BM) * tilesN;
  const int gemmCtas = gather ? a.gemmCtas : gridDim.x / S;
  const int tile0 = blockIdx.x / S;
  const uint32_t smemA0 = smemAddr(smem), smemB0 = smemA0 + STAGES * kStageABytes;
  auto fail = [&](uint32_t kind, uint32_t what) {
    *abortFlag = 1;
    if (a.sync.status[rank] && ldRelaxedSys(a.sync.status[rank]) == DEV_OK) {
      a.sync.status[rank][1] = kind;
      a.sync.status[rank][2] = what;
      a.sync.status[rank][3] = blockIdx.x;
      __threadfence_system();
      stRelaxedSys(a.sync.status[rank], DEV_TIMEOUT);
    }
  };

  if (warp < 4) {
    regsGive<kRegsProducer>();
    if (warp == 0 && electOne()) {
      uint32_t kc = 0;
      uint32_t armed = 0, armedPhase = 0;   // per stage: a copy was issued, and for which phase of its barrier
      for (int t = tile0; t < nTiles && !*abortFlag; t += gemmCtas) {
        const TileCoord tc = tileOf(a, t, BM, BN);
        if (gather && tc.owner != rank) {
          const uint32_t* f = a.blockFlags + tc.mBlk;
          bool got = false;
          for (uint32_t spin = 0; spin < (1u << 26); ++spin) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
            if ((int32_t)(v - a.flagEpoch) >= 0) { got = true; break; }
            if (*abortFlag) break;
          }
          if (!got) { fail(WAIT_TILE, (uint32_t)tc.mBlk); break; }
          fenceProxyAsync();
        }
        for (int kb = 0; kb < kBlocks; ++kb, ++kc) {
          const int s = kc % STAGES;
          const uint32_t ph = (kc / STAGES) & 1;
          if (!mbarWait(smemAddr(&emptyBar[s]), ph ^ 1)) { fail(WAIT_TILE, 1000 + s); break; }
          const uint32_t fb = smemAddr(&fullBar[s]);
          mbarExpectTx(fb, kStageBytes);
          tmaLoad2d(smemA0 + s * kStageABytes, &tmA, (kBegin + kb) * BK, tc.mBlk * BM, fb);
          tmaLoad2d(smemB0 + s * kStageBBytes, &tmB, (kBegin + kb) * BK, tc.nBlk * BN, fb);
          armed |= 1u << s;
          armedPhase = (armedPhase & ~(1u << s)) | (ph << s);
        }
      }
      if (*abortFlag) {
        // copies already issued still write into shared memory: wait for them (bounded)
        for (int s = 0; s < STAGES; ++s)
          if ((armed >> s) & 1u) mbarWait(smemAddr(&fullBar[s]), (armedPhase >> s) & 1u, 1u << 20);
      }
    } else if (warp == 1 && electOne()) {
      const uint32_t idesc = umInstrE4m3(BM, BN);
      uint32_t kc = 0;
      for (int t = tile0; t < nTiles && !*abortFlag; t += gemmCtas) {
        bool bad = false;
        for (int kb = 0; kb < kBlocks; ++kb, ++kc) {
          const int buf = kc & 1;
          const uint32_t aph = (kc >> 1) & 1;
          if (!mbarWait(smemAddr(&accEmpty[buf]), aph ^ 1)) { fail(WAIT_TILE, 2000 + buf); bad = true; break; }
          const int s = kc % STAGES;
          const uint32_t ph = (kc / STAGES) & 1;
          if (!mbarWait(smemAddr(&fullBar[s]), ph)) { fail(WAIT_TILE, 3000 + s); bad = true; break; }
          tcFenceAfter();
          const uint32_t dT = tmemBase + buf * kAccCols;
          const uint32_t aAddr = smemA0 + s * kStageABytes, bAddr = smemB0 + s * kStageBBytes;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            ummaF8(dT, umDescK128(aAddr + k * UMMA_K), umDescK128(bAddr + k * UMMA_K), idesc, k != 0);
          ummaCommit(smemAddr(&emptyBar[s]));   // the stage is free once these MMAs have read it
          ummaCommit(smemAddr(&accFull[buf]));  // this K block's partial sums are complete
        }
        if (bad) break;
      }
    }
  } else {
    regsTake<kRegsEpilogue>();
    // ---- epilogue warps: TMEM lanes [32q, 32q+32), columns [kHalf * h, kHalf * (h + 1))
    const int q = warp & 3;
    const int h = (warp - 4) >> 2;
    const int c0 = h * kHalf;
    const float* scaleA = gather ? (const float*)((const char*)a.peerA[rank] + a.scaleOffset) : a.scaleA;
    const int wBlocksN = a.N / 128;
    uint32_t kc = 0;
    uint64_t acc[kChunks * 16];   // fp32 pairs
    for (int t = tile0; t < nTiles; t += gemmCtas) {
      const TileCoord tc = tileOf(a, t, BM, BN);
      const int row0 = tc.mBlk * BM + q * 32;
      const int row = row0 + lane;
      const int wCol = (tc.nBlk * BN + c0) / 128;
#pragma unroll
      for (int j = 0; j < kChunks * 16; ++j) acc[j] = 0;
      // The scales of the next K block travel ahead of the accumulator that needs them.
      // In GATHER mode the scales of remote rows land together with the rows: the flag the TMA
      // producer waited for covers them, and accFull orders this warp after the producer.
      bool bad = __any_sync(0xffffffffu, *abortFlag);
      if (bad) break;
      // Rows gathered from a peer arrive during this kernel: their scales may be read only after
      // the tile's first accumulator is published (the producer saw the block's flag before it
      // issued the TMA loads that fed it), and never through the read-only cache path.
      const bool remoteRows = gather && tc.owner != rank;
      float nextA = 0.0f, nextW = 0.0f;
      auto fetchScales = [&](int kb) {
        nextA = *(const volatile float*)(scaleA + (size_t)(kBegin + kb) * a.M + row);
        nextW = *(const volatile float*)(a.scaleW + (size_t)(kBegin + kb) * wBlocksN + wCol);
      };
      if (!remoteRows) fetchScales(0);
      // sets of 32 columns: one is fetched while the one before is multiplied, across K blocks too
      uint32_t set[2][32];
#pragma unroll
      for (int j = 0; j < 32; ++j) set[1][j] = 0;
      float s = 0.0f;
      auto madd = [&](int c, const uint32_t (&r)[32], float by) {
        const uint64_t s2 = packF32x2(__float_as_uint(by), __float_as_uint(by));
#pragma unroll
        for (int j = 0; j < 16; ++j) fmaF32x2(acc[c * 16 + j], packF32x2(r[2 * j], r[2 * j + 1]), s2);
      };
      for (int kb = 0; kb < kBlocks && (kLeave || !bad); ++kb, ++kc) {
        const int buf = kc & 1;
        const uint32_t aph = (kc >> 1) & 1;
        bad = !__all_sync(0xffffffffu, mbarWait(smemAddr(&accFull[buf]), aph));   // one answer for the warp, which loads together
        if (bad && lane == 0) fail(WAIT_TILE, 4000 + buf);
        if (kLeave && bad) break;
        tcFenceAfter();
        if (remoteRows && kb == 0) fetchScales(0);
        const uint32_t tBase = tmemBase + ((uint32_t)(q * 32) << 16) + buf * kAccCols + c0;
        const float next = nextA * nextW;
        if (kb + 1 < kBlocks) fetchScales(kb + 1);
        tmemLd32(tBase, set[0]);
        madd(kChunks - 1, set[1], s);   // the last columns of the block before this one
        tmemLdWait32(set[0]);
        s = next;
#pragma unroll
        for (int c = 1; c < kChunks; ++c) {
          tmemLd32(tBase + c * 32, set[c & 1]);
          madd(c - 1, set[(c - 1) & 1], s);
          tmemLdWait32(set[c & 1]);
        }
        tcFenceBefore();
        __syncwarp();
        if (lane == 0) mbarArrive(smemAddr(&accEmpty[buf]));
      }
      if (bad) break;
      madd(kChunks - 1, set[1], s);
      if (SPLIT) break;   // one tile, finished with the other shares below
      // final tile: bf16, transposed through shared memory so that every store instruction writes
      // whole 128-byte row segments (see the bf16 kernel); REDUCE targets the owner's staging slot
      {
        __nv_bfloat16* dstBase;
        size_t ld;
        if (FUSED && a.mode == TP_MODE_REDUCE) {
          const int rowsPerRank = a.M / n;
          dstBase = (__nv_bfloat16*)a.partial[tc.owner] + ((size_t)rank * rowsPerRank + (row0 - tc.owner * rowsPerRank)) * a.N + (size_t)tc.nBlk * BN + c0;
          ld = (size_t)a.N;
        } else {
          dstBase = (__nv_bfloat16*)a.C + (size_t)row0 * a.ldc + (size_t)tc.nBlk * BN + c0;
          ld = (size_t)a.ldc;
        }
        uint8_t* wbuf = epiBuf + (size_t)(warp - 4) * 4096;
        auto bf16Pair = [&](int i) -> uint32_t {
          const __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float((uint32_t)acc[i]), __uint_as_float((uint32_t)(acc[i] >> 32)));
          return *(const uint32_t*)&p;
        };
#pragma unroll
        for (int cc = 0; cc < kChunks / 2; ++cc) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int b0 = cc * 32 + j * 4;
            const uint4 o = make_uint4(bf16Pair(b0), bf16Pair(b0 + 1), bf16Pair(b0 + 2), bf16Pair(b0 + 3));
            *(uint4*)(wbuf + lane * 128 + ((j ^ (lane & 7)) * 16)) = o;
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int rr = k * 4 + (lane >> 3), j = lane & 7;
            const uint4 o = *(const uint4*)(wbuf + rr * 128 + ((j ^ (rr & 7)) * 16));
            *(uint4*)((char*)(dstBase + (size_t)rr * ld) + cc * 128 + j * 16) = o;
          }
          __syncwarp();
        }
      }
    }
    if (SPLIT) {
      // Every CTA holds the scaled fp32 sums of its share of the K blocks in registers. Chunk g of 32 columns belongs to CTA g % S: the
      // others put their sums into its operand ring (free: all MMAs of the cluster are behind the first barrier), and the owner
      // adds them in the order of the shares, rounds once and stores. The result does not depend on the schedule.
      const int rowInTile = q * 32 + lane;
      auto slotOf = [&](int g, int from, int owner) {
        const int others = from < owner ? from : from - 1;
        return (uint32_t)((g / S) * (S - 1) + others) * kChunkBytes + (uint32_t)rowInTile * 16;
      };
      __syncwarp();
      clusterSync();
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int g = h * kChunks + c, owner = g % S;
        if (owner == share) continue;
        const uint32_t dst = mapaShared(smemA0 + slotOf(g, share, owner), (uint32_t)owner);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          stSharedCluster16(dst + j * (BM * 16), (uint32_t)acc[c * 16 + 2 * j], (uint32_t)(acc[c * 16 + 2 * j] >> 32), (uint32_t)acc[c * 16 + 2 * j + 1],
                            (uint32_t)(acc[c * 16 + 2 * j + 1] >> 32));
      }
      clusterSync();
      const TileCoord tc = tileOf(a, tile0, BM, BN);
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int g = h * kChunks + c, col = tc.nBlk * BN + g * 32;
        if (g % S != share) continue;
        float sum[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[j] = 0.0f;
        for (int from = 0; from < S; ++from) {
          if (from == share) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              sum[2 * j] += __uint_as_float((uint32_t)acc[c * 16 + j]);
              sum[2 * j + 1] += __uint_as_float((uint32_t)(acc[c * 16 + j] >> 32));
            }
          } else {
            const uint8_t* src = smem + slotOf(g, from, share);
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
        __nv_bfloat16* out = (__nv_bfloat16*)a.C + (size_t)(tc.mBlk * BM + rowInTile) * a.ldc + col;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 o;
          __nv_bfloat162* p = (__nv_bfloat162*)&o;
#pragma unroll
          for (int k = 0; k < 4; ++k) p[k] = __floats2bfloat162_rn(sum[8 * j + 2 * k], sum[8 * j + 2 * k + 1]);
          *(uint4*)(out + j * 8) = o;
        }
      }
    }
  }
  if (SPLIT && warp < 4) {
    __syncwarp();
    clusterSync();
    clusterSync();
  }

  tcFenceBefore();
  __syncthreads();
  if (warp == 1) {
    tcFenceAfter();
    tmemDealloc(tmemBase, kTmemCols);
  }
  if (FUSED) {
    bar.sync(true, false);
    bar.finish();
  }
}

// ------------------------------------------------------------------------------------ quantisation
__device__ __forceinline__ uint32_t packE4m3x4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return (uint32_t)lo | ((uint32_t)hi << 16);
}

// Activations: one scale per row and 128 columns; scales[kb][row]. Eight lanes share a group of 128 columns, 16 columns (two
// 16-byte loads, one 16-byte store) each; a warp covers four rows of one K block, so that it writes four neighbouring scales, and a
// CTA four rows of 16 K blocks, two per thread with all loads ahead of the arithmetic. Bound by memory: 1920 x 7168 take 8.9 us, with one
// warp and 8-byte accesses per group they took 18.
// Needs 16-byte aligned x and q.
constexpr int kQuantRows = 4, kQuantBlocks = 16;
__global__ void __launch_bounds__(256) tpQuantRowsWideKernel(const __nv_bfloat16* x, uint8_t* q, float* scales,
                                                             int rows, int K) {
  pdlEnter();
  const int kBlocks = K / 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = (int)blockIdx.x * kQuantRows + (lane >> 3);
  uint4 raw[2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int kb = (int)blockIdx.y * kQuantBlocks + u * 8 + warp;
    const bool in = row < rows && kb < kBlocks;
    const uint4* p = (const uint4*)(x + (size_t)row * K + (size_t)kb * 128 + (lane & 7) * 16);
    raw[u][0] = in ? ldStream16(p) : make_uint4(0, 0, 0, 0);
    raw[u][1] = in ? ldStream16(p + 1) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int kb = (int)blockIdx.y * kQuantBlocks + u * 8 + warp;
    float v[16];
    float m = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const __nv_bfloat162* p = (const __nv_bfloat162*)&raw[u][h];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[h * 8 + 2 * i] = __bfloat162float(p[i].x);
        v[h * 8 + 2 * i + 1] = __bfloat162float(p[i].y);
        m = fmaxf(m, fmaxf(fabsf(v[h * 8 + 2 * i]), fabsf(v[h * 8 + 2 * i + 1])));
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float s = fmaxf(m, 1e-10f) / 448.0f;
    const float inv = 1.0f / s;
    if (row >= rows || kb >= kBlocks) continue;
    uint4 o;
    o.x = packE4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
    o.y = packE4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
    o.z = packE4m3x4(v[8] * inv, v[9] * inv, v[10] * inv, v[11] * inv);
    o.w = packE4m3x4(v[12] * inv, v[13] * inv, v[14] * inv, v[15] * inv);
    *(uint4*)(q + (size_t)row * K + (size_t)kb * 128 + (lane & 7) * 16) = o;
    if ((lane & 7) == 0) scales[(size_t)kb * rows + row] = s;
  }
}

// The same from 8-byte aligned x into 4-byte aligned q, and for few K blocks. One warp per (row, K block).
__global__ void __launch_bounds__(256) tpQuantRowsKernel(const __nv_bfloat16* x, uint8_t* q, float* scales,
                                                          int rows, int K) {
  pdlEnter();
  const int kBlocks = K / 128;
  const size_t warpId = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const size_t nWarps = ((size_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (size_t w = warpId; w < (size_t)rows * kBlocks; w += nWarps) {
    const int row = (int)(w / kBlocks), kb = (int)(w % kBlocks);
    const size_t off = (size_t)row * K + (size_t)kb * 128 + lane * 4;
    const uint2 raw = *(const uint2*)(x + off);
    const __nv_bfloat162* p = (const __nv_bfloat162*)&raw;
    float v0 = __bfloat162float(p[0].x), v1 = __bfloat162float(p[0].y), v2 = __bfloat162float(p[1].x), v3 = __bfloat162float(p[1].y);
    float m = fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float s = fmaxf(m, 1e-10f) / 448.0f;
    const float inv = 1.0f / s;
    *(uint32_t*)(q + off) = packE4m3x4(v0 * inv, v1 * inv, v2 * inv, v3 * inv);
    if (lane == 0) scales[(size_t)kb * rows + row] = s;
  }
}

// Weights: one scale per 128 x 128 block. One CTA of 256 threads per block; scales[kb][rows/128].
__global__ void __launch_bounds__(256) tpQuantBlocksKernel(const __nv_bfloat16* x, uint8_t* q, float* scales,
                                                            int rows, int K) {
  pdlEnter();
  __shared__ float red[8];
  const int kBlocks = K / 128, rBlocks = rows / 128;
  for (int blk = blockIdx.x; blk < kBlocks * rBlocks; blk += gridDim.x) {
    const int rb = blk / kBlocks, kb = blk % kBlocks;
    // thread t: rows (t / 32) + 8 i, columns 4 (t % 32) .. +3
    float v[16][4];
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const size_t off = (size_t)(rb * 128 + (threadIdx.x >> 5) + 8 * i) * K + (size_t)kb * 128 + (threadIdx.x & 31) * 4;
      const uint2 raw = *(const uint2*)(x + off);
      const __nv_bfloat162* p = (const __nv_bfloat162*)&raw;
      v[i][0] = __bfloat162float(p[0].x); v[i][1] = __bfloat162float(p[0].y); v[i][2] = __bfloat162float(p[1].x); v[i][3] = __bfloat162float(p[1].y);
      m = fmaxf(m, fmaxf(fmaxf(fabsf(v[i][0]), fabsf(v[i][1])), fmaxf(fabsf(v[i][2]), fabsf(v[i][3]))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w]);
    const float s = fmaxf(m, 1e-10f) / 448.0f;
    const float inv = 1.0f / s;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const size_t off = (size_t)(rb * 128 + (threadIdx.x >> 5) + 8 * i) * K + (size_t)kb * 128 + (threadIdx.x & 31) * 4;
      *(uint32_t*)(q + off) = packE4m3x4(v[i][0] * inv, v[i][1] * inv, v[i][2] * inv, v[i][3] * inv);
    }
    if (threadIdx.x == 0) scales[(size_t)kb * rBlocks + rb] = s;
  }
}

const void* tpGemmFp8KernelFn(bool fused, int width, bool split) {
  if (fused) return (const void*)tpGemmFp8Kernel<true, 256, false>;
  if (width == 256) return split ? (const void*)tpGemmFp8Kernel<false, 256, true> : (const void*)tpGemmFp8Kernel<false, 256, false>;
  return split ? (const void*)tpGemmFp8Kernel<false, 128, true> : (const void*)tpGemmFp8Kernel<false, 128, false>;
}
const void* tpQuantRowsWideKernelFn() { return (const void*)tpQuantRowsWideKernel; }
void tpQuantRowsWideGrid(int rows, int K, int* x, int* y) {
  *x = (rows + kQuantRows - 1) / kQuantRows;
  *y = (K / 128 + kQuantBlocks - 1) / kQuantBlocks;
}
const void* tpQuantRowsKernelFn() { return (const void*)tpQuantRowsKernel; }
const void* tpQuantBlocksKernelFn() { return (const void*)tpQuantBlocksKernel; }
size_t tpGemmFp8SmemBytes() { return kSmemBytes; }
int tpGemmFp8Threads() { return kThreads; }

}  // namespace b200
