// Kernels written against the public device API (nccl_device.h) only: they serve as its tests
// and as the fused all-reduce + residual + RMSNorm building block of tensor-parallel decoders.
//   b200DevApiAllReduce   in-place-capable sum all-reduce of a window slice: every CTA owns one
//                         LSA barrier; each pack is loaded from all peers (or through
//                         multimem.ld_reduce) and stored to all peers (or through multimem.st).
//   b200DevApiArRmsNorm   x = sum over ranks of partial[t,:] + residual[t,:]; residual <- x;
//                         out <- x * rsqrt(mean(x^2) + eps) * weight. One-shot (every rank reduces
//                         every row; peer loads or multimem) or two-shot (rows dealt to ranks, the
//                         owner stores residual and out to every rank).
//   b200DevApiLLSum       low-latency all-to-all session: two floats per slot summed over ranks.
// Reference parity: examples/06_device_api (LSA / multimem all-reduce samples) and
// contrib/nccl_ubx allreduce_2shot_* with residual and RMSNorm epilogue.
#include <cuda_bf16.h>

#include <algorithm>

#include "nccl_device.h"
#include "../comm/device_plane.h"
#include "../kernels/common.cuh"
#include "../tp/gemm_sm100.cuh"

namespace {

constexpr int kThreads = 512;

template <typename T>
__global__ void __launch_bounds__(kThreads) devApiAllReduceKernel(ncclDevComm_t dc, ncclWindow_t sendWin, size_t sendOff, ncclWindow_t recvWin,
                                                                   size_t recvOff, size_t count, int multimem, int* status) {
  using V = nccl_device::Vec16<T>;
  ncclCoopCta cta;
  ncclLsaBarrierSession<ncclCoopCta> bar(cta, dc, ncclTeamLsa(dc), blockIdx.x);
  if (bar.sync(0, false, false) != ncclSuccess) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    bar.finish();
    return;
  }
  const int n = dc.lsaSize;
  const size_t packs = count / V::N;   // the host checks count % V::N == 0
  const size_t perRank = (packs + n - 1) / n;
  const size_t lo = min(packs, perRank * dc.lsaRank), hi = min(packs, lo + perRank);
  const char* mcIn = (const char*)ncclGetMultimemPointer(sendWin, sendOff);
  char* mcOut = (char*)ncclGetMultimemPointer(recvWin, recvOff);
  for (size_t i = lo + (size_t)blockIdx.x * kThreads + threadIdx.x; i < hi; i += (size_t)gridDim.x * kThreads) {
    uint4 r;
    if (multimem) {
      r = V::mcLoad(mcIn + i * 16);
      ncclMultimemStore16(mcOut + i * 16, r);
    } else {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int p = 0; p < n; ++p) V::add(acc, *(const uint4*)((const char*)ncclGetLsaPointer(sendWin, sendOff, p) + i * 16));
      r = V::pack(acc);
      for (int p = 0; p < n; ++p) *(uint4*)((char*)ncclGetLsaPointer(recvWin, recvOff, (dc.lsaRank + p) % n) + i * 16) = r;
    }
  }
  if (bar.sync(0, true, false) != ncclSuccess && threadIdx.x == 0) atomicExch(status, 2);
  bar.finish();
}

__device__ __forceinline__ float blockSum(float v, float* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) smem[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < kThreads / 32 ? smem[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) smem[32] = t;
  }
  __syncthreads();
  return smem[32];
}

// mode 0: one-shot, peer loads; 1: one-shot, multimem.ld_reduce; 2: two-shot, peer loads + peer stores
__global__ void __launch_bounds__(kThreads) devApiArRmsNormKernel(ncclDevComm_t dc, ncclWindow_t inWin, size_t inOff, ncclWindow_t resWin, size_t resOff,
                                                                   ncclWindow_t outWin, size_t outOff, const __nv_bfloat16* weight, float eps, int tokens,
                                                                   int hidden, int mode, int* status) {
  using V = nccl_device::Vec16<__nv_bfloat16>;
  __shared__ float red[40];
  ncclCoopCta cta;
  ncclLsaBarrierSession<ncclCoopCta> bar(cta, dc, ncclTeamLsa(dc), blockIdx.x);
  if (bar.sync(0, false, false) != ncclSuccess) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    bar.finish();
    return;
  }
  const int n = dc.lsaSize, me = dc.lsaRank;
  const int packsPerRow = hidden / 8;   // the host checks hidden % 8 == 0 and hidden <= 8 * kThreads * 4
  const size_t rowBytes = (size_t)hidden * 2;
  const int rowStep = mode == 2 ? gridDim.x * n : gridDim.x;
  const int rowStart = mode == 2 ? blockIdx.x * n + me : blockIdx.x;
  char* resLocal = (char*)ncclGetLocalPointer(resWin, resOff);
  char* outLocal = (char*)ncclGetLocalPointer(outWin, outOff);
  const char* mcIn = (const char*)ncclGetMultimemPointer(inWin, inOff);
  for (int t = rowStart; t < tokens; t += rowStep) {
    float x[4][8];
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int pk = threadIdx.x + k * kThreads;
#pragma unroll
      for (int j = 0; j < 8; ++j) x[k][j] = 0.0f;
      if (pk < packsPerRow) {
        const size_t o = t * rowBytes + (size_t)pk * 16;
        if (mode == 1) {
          V::add(x[k], V::mcLoad(mcIn + o));
        } else {
          for (int p = 0; p < n; ++p) V::add(x[k], *(const uint4*)((const char*)ncclGetLsaPointer(inWin, inOff, p) + o));
        }
        V::add(x[k], *(const uint4*)(resLocal + o));
        // the residual stream is kept in bf16: normalise exactly what is stored
        const uint4 packed = V::pack(x[k]);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[k][j] = 0.0f;
        V::add(x[k], packed);
        if (mode == 2) {
          for (int p = 0; p < n; ++p) *(uint4*)((char*)ncclGetLsaPointer(resWin, resOff, (me + p) % n) + o) = packed;
        } else {
          *(uint4*)(resLocal + o) = packed;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += x[k][j] * x[k][j];
      }
    }
    const float inv = rsqrtf(blockSum(ss, red) / (float)hidden + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int pk = threadIdx.x + k * kThreads;
      if (pk < packsPerRow) {
        const size_t o = t * rowBytes + (size_t)pk * 16;
        float w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        V::add(w, *(const uint4*)((const char*)weight + (size_t)pk * 16));
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] *= x[k][j] * inv;
        const uint4 packed = V::pack(w);
        if (mode == 2) {
          for (int p = 0; p < n; ++p) *(uint4*)((char*)ncclGetLsaPointer(outWin, outOff, (me + p) % n) + o) = packed;
        } else {
          *(uint4*)(outLocal + o) = packed;
        }
      }
    }
  }
  if (bar.sync(0, true, false) != ncclSuccess && threadIdx.x == 0) atomicExch(status, 2);
  bar.finish();
}

// One rank: x = partial + residual, residual <- x, out <- rmsnorm(x) * weight, as above without the sources to wait for.
// Bound on the SMs that the caller grants by what each of them moves through shared memory and has in flight: a producer warp
// streams chunks of R neighbouring rows (partial and residual) into a ring of shared memory with bulk copies, groups of G
// threads take one row each from there. 2048 rows of 8192 take 24 us a call on 64 CTAs (5.5 TB/s; the same on 96 and 148): 127 with a CTA
// to a row whose loads wait for the previous row's stores, and 33 while the compiler read the rows word by word, four lanes to a bank (13
// wavefronts for 16 bytes a lane instead of 4): hence addBf16 takes values, and the ring is visibly shared memory. Values are added, squared and scaled in pairs; the gains lie beside the ring, so that 768 threads have the registers they need.
constexpr int kRowPacks = 8;          // 16-byte packs of a row per thread, at most
constexpr int kRowStages = 16;        // chunks in the ring, at most
constexpr size_t kRowRing = 200 << 10;
constexpr int kRowsWide = 768;        // threads of the groups where rows are long and many, kThreads otherwise
constexpr int kRowSmem = (227 << 10) - 1024;   // ring and gains; the rest is static
constexpr int kStatusRing = 6;        // status word: a wait on the ring ran out

// Pairs of values: bf16 is the upper half of fp32.
__device__ __forceinline__ uint64_t unpackBf16x2(uint32_t u) { return b200::sm100::packF32x2(u << 16, u & 0xffff0000u); }
__device__ __forceinline__ uint64_t mulF32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The exact sum rounded once, which is what fp32 gives too: where a sum of two bf16 numbers does not fit into fp32, the smaller one is
// far below a tie of the larger.
__device__ __forceinline__ uint4 addBf16(uint4 a, uint4 b) {
  uint4 r;
  const __nv_bfloat162 *x = (const __nv_bfloat162*)&a, *y = (const __nv_bfloat162*)&b;
  __nv_bfloat162* z = (__nv_bfloat162*)&r;
#pragma unroll
  for (int i = 0; i < 4; ++i) z[i] = __hadd2_rn(x[i], y[i]);
  return r;
}

struct RowArgs {
  const char* partial;
  char* residual;
  char* out;
  const char* weight;
  float eps;
  int tokens, hidden, chunkShift, stages;
  int* status;
};

// FULL: every thread of a group has the same number of packs. W: threads of all groups
template <int G, bool FULL, int W>
__global__ void __launch_bounds__(W + 32, 1) rmsNormRowsKernel(const __grid_constant__ RowArgs a) {
  using namespace b200::sm100;
  constexpr int kGroups = W / G, kWarps = G / 32;
  // the gains, then the ring. Aligned here and not by arithmetic, behind which the compiler no longer knew that it reads shared memory:
  // generic loads of 16 bytes took 13 wavefronts instead of 4
  extern __shared__ __align__(128) uint8_t gains[];
  __shared__ float red[2][W / 32];
  __shared__ uint64_t fullBar[kRowStages], emptyBar[kRowStages];
  __shared__ volatile int gaveUp;
  const int shift = a.chunkShift, R = 1 << shift, chunks = (a.tokens + R - 1) >> shift, packs = a.hidden / 8;
  const size_t rowBytes = (size_t)a.hidden * 2;
  uint8_t* ring = gains + ((rowBytes + 127) & ~(size_t)127);
  const uint32_t half = (uint32_t)(R * rowBytes);   // partial rows, then residual rows
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbarInit(smemAddr(&fullBar[s]), 1);
      mbarInit(smemAddr(&emptyBar[s]), R * kWarps);   // one arrival per row and warp
    }
    gaveUp = 0;
    mbarInitFence();
  }
  __syncthreads();
  b200::pdlEnter();   // the set-up above overlaps the end of the kernel before
  // false: this wait or one of another thread ran out. Nobody waits, copies or stores any longer; the copies still under way are
  // waited for below
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    if (!gaveUp && mbarWait(smemAddr(bar), parity)) return true;
    gaveUp = 1;
    atomicExch(a.status, kStatusRing);
    return false;
  };
  if (threadIdx.x >= W) {
    if (threadIdx.x == W) {
      int i = 0;
      for (int c = blockIdx.x; c < chunks && !gaveUp; c += gridDim.x, ++i) {
        const int s = i % a.stages;
        const uint32_t ph = (i / a.stages) & 1;
        if (!wait(&emptyBar[s], ph ^ 1)) break;   // the slot is still being read
        const int rows = a.tokens - c * R < R ? a.tokens - c * R : R;
        const uint32_t bytes = (uint32_t)(rows * rowBytes);
        const size_t off = (size_t)c * R * rowBytes;
        const uint32_t dst = smemAddr(ring) + (uint32_t)s * 2 * half, fb = smemAddr(&fullBar[s]);
        mbarExpectTx(fb, 2 * bytes);
        bulkLoad(dst, a.partial + off, bytes, fb);
        bulkLoad(dst + half, a.residual + off, bytes, fb);
      }
      if (gaveUp)
        for (int j = i > a.stages ? i - a.stages : 0; j < i; ++j) mbarWait(smemAddr(&fullBar[j % a.stages]), (j / a.stages) & 1, 1u << 20);
    }
  } else {
    // the gains, while the first rows travel
    for (int pk = threadIdx.x; pk < packs; pk += W) *(uint4*)(gains + (size_t)pk * 16) = *(const uint4*)(a.weight + (size_t)pk * 16);
    asm volatile("bar.sync 15, %0;" ::"n"(W) : "memory");
    const int grp = threadIdx.x / G;
    const int tid = threadIdx.x % G, mine = packs / G, lap = a.stages << shift;   // rows of a lap of the ring, whole steps of the group
    auto has = [&](int k) { return FULL ? k < mine : tid + k * G < packs; };
    int m = grp;   // this group's row, counted from the lap's first
    uint32_t phase = 0;
    int parity = 0;
    // row n of this CTA: row n % R of its chunk n / R
    for (int n = grp;; n += kGroups, parity ^= 1) {
      const int c = (int)blockIdx.x + (n >> shift) * (int)gridDim.x;
      if (c >= chunks) break;
      const int r = m & (R - 1), t = c * R + r;
      if (t >= a.tokens) break;
      const int s = m >> shift;
      // a row that did not arrive is left alone: neither read, stored nor released; its group still meets at the barrier. The lanes of a warp
      // vote: each of them polls and reads gaveUp for itself
      const bool ok = __all_sync(0xffffffffu, wait(&fullBar[s], phase));
      if ((m += kGroups) >= lap) {
        m -= lap;
        phase ^= 1;
      }
      const uint8_t* part = ring + (size_t)s * 2 * half + r * rowBytes + tid * 16;
      const size_t at = t * rowBytes + tid * 16;
      char* res = a.residual + at;
      uint4 sum[kRowPacks];
      uint64_t squares = 0;   // two fp32 sums
      if (ok) {
#pragma unroll
        for (int k = 0; k < kRowPacks; ++k) {
          if (has(k)) {
            // the residual stream is kept in bf16: normalise exactly what is stored
            const uint4 x = *(const uint4*)(part + k * G * 16), y = *(const uint4*)(part + half + k * G * 16);
            sum[k] = addBf16(x, y);
            *(uint4*)(res + k * G * 16) = sum[k];
            const uint32_t u[4] = {sum[k].x, sum[k].y, sum[k].z, sum[k].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint64_t x = unpackBf16x2(u[j]);
              fmaF32x2(squares, x, x);
            }
          }
        }
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbarArrive(smemAddr(&emptyBar[s]));   // the warp has read its part of the row
      }
      float ss = __uint_as_float((uint32_t)squares) + __uint_as_float((uint32_t)(squares >> 32));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (kWarps > 1) {
        // one word per warp, two sets by parity: a warp reaches the set again only after the group has met once more
        if ((threadIdx.x & 31) == 0) red[parity][threadIdx.x >> 5] = ss;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(G) : "memory");
        ss = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) ss += red[parity][grp * kWarps + w];
      }
      if (!ok) continue;
      const float inv = rsqrtf(ss / (float)a.hidden + a.eps);
      const uint64_t inv2 = packF32x2(__float_as_uint(inv), __float_as_uint(inv));
      char* out = a.out + at;
      const uint8_t* gain = gains + tid * 16;
#pragma unroll
      for (int k = 0; k < kRowPacks; ++k) {
        if (has(k)) {
          const uint4 gk = *(const uint4*)(gain + k * G * 16);
          const uint32_t u[4] = {sum[k].x, sum[k].y, sum[k].z, sum[k].w}, g[4] = {gk.x, gk.y, gk.z, gk.w};
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t y = mulF32x2(mulF32x2(unpackBf16x2(u[j]), inv2), unpackBf16x2(g[j]));
            const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float((uint32_t)y), __uint_as_float((uint32_t)(y >> 32)));
            o[j] = *(const uint32_t*)&b;
          }
          *(uint4*)(out + k * G * 16) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
  }
  __syncthreads();   // no thread leaves while a copy into this CTA's shared memory is under way
}

// How the kernel above splits a call: threads to a row, rows of a chunk, chunks in the ring.
//
// A wait on a slot's barrier tells two uses of the slot apart by the parity of their phases, so a group may wait for a use only
// when it has seen the one before: nothing orders the copies of two chunks, and a wait that skips a use would take a slot whose
// copy of the lap before is still under way for loaded. Group g takes rows g, g + groups, ... of its CTA, so it sees every use of
// the slots that it reads when a lap of the ring (stages x chunkRows rows) is a whole number of its steps. Both are kept to
// multiples that see to it: four groups get 4 stages of 8192 channels where the ring would hold 6.
struct RowPlan {
  int group, threads, chunkRows, stages;
};

RowPlan rowPlan(int tokens, int hidden, int nCtas) {
  const size_t rowBytes = (size_t)hidden * 2;
  RowPlan p;
  // the fewest threads to a row that hold it, more where there are not enough rows for that many groups
  p.group = 32;
  while (p.group < kThreads && (p.group * kRowPacks < hidden / 8 || (long long)nCtas * (kThreads / p.group) > tokens)) p.group *= 2;
  // Six rows under way in a CTA instead of four where that many fit the ring as well as four do and there are enough of them: 2048 x 8192 24.2 us
  // for 25.5 with 512 threads, 3000 x 7168 30.5 for 33.0, 1000 x 8104 13.8 for 14.1. The other side of the line: 1024 x 5120 10.1 / 9.9, 700 x 6144
  // 8.5 / 8.3, 256 x 8192 5.0 / 4.8.
  p.threads = p.group == 128 && hidden > 6144 && tokens >= 12 * nCtas ? kRowsWide : kThreads;
  // chunks of about 8 KiB (a copy below that costs more to issue than to move), while every CTA still gets several; a power of two
  const int rows = std::min((int)(8192 / rowBytes), tokens / (4 * nCtas));
  p.chunkRows = 1;
  while (2 * p.chunkRows <= rows) p.chunkRows *= 2;
  int step = p.threads / p.group;
  for (int r = p.chunkRows; r > 1 && step % 2 == 0; r /= 2) step /= 2;
  p.stages = (int)std::min<size_t>(kRowStages, kRowRing / (2 * p.chunkRows * rowBytes)) / step * step;
  return p;
}

template <int G, int W = kThreads> const void* rowsKernel(bool full) { return full ? (const void*)rmsNormRowsKernel<G, true, W> : (const void*)rmsNormRowsKernel<G, false, W>; }

ncclResult_t launchRmsNormRows(RowArgs a, int nCtas, cudaStream_t stream) {
  const RowPlan p = rowPlan(a.tokens, a.hidden, nCtas);
  a.chunkShift = __builtin_ctz(p.chunkRows);
  a.stages = p.stages;
  const size_t smem = 128 + (size_t)a.hidden * 4 * p.chunkRows * p.stages + (size_t)a.hidden * 2;
  const bool full = a.hidden / 8 % p.group == 0;
  const void* fn = p.threads == kRowsWide ? rowsKernel<128, kRowsWide>(full) : p.group == 32 ? rowsKernel<32>(full) : p.group == 64 ? rowsKernel<64>(full) :
                   p.group == 128 ? rowsKernel<128>(full) : p.group == 256 ? rowsKernel<256>(full) : rowsKernel<512>(full);
  // The limit belongs to the function, which threads with other shapes launch at the same time: every call sets the same value, the
  // largest ring, and never one below what another is about to launch with.
  void* args[1] = {&a};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute pdl;
  cfg.gridDim = dim3(nCtas);
  cfg.blockDim = dim3(p.threads + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  if (b200::devPlanePdl()) {
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
  }
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmem) == cudaSuccess &&
      cudaLaunchKernelExC(&cfg, fn, args) == cudaSuccess)
    return ncclSuccess;
  (void)cudaGetLastError();   // the call reports it: later checks do not find it again
  return ncclUnhandledCudaError;
}

// Exercises ncclLLA2ASession: every rank contributes two floats per slot; each rank receives the sum.
__global__ void __launch_bounds__(256) devApiLLSumKernel(ncclDevComm_t dc, const float2* in, float2* out, int slots, int* status) {
  ncclCoopCta cta;
  ncclLLA2ASession<ncclCoopCta> ll(cta, dc, ncclTeamLsa(dc), blockIdx.x);
  for (int s = threadIdx.x; s < slots; s += blockDim.x) {
    const float2 v = in[blockIdx.x * slots + s];
    ll.bcast(s, (uint64_t)__float_as_uint(v.x) | ((uint64_t)__float_as_uint(v.y) << 32));
    float2 r;
    if (ll.recvReduceFloat2(s, v, &r) != ncclSuccess) {
      atomicExch(status, 3);
      break;
    }
    out[blockIdx.x * slots + s] = r;
  }
  ll.endEpoch();
}

// Exercises ncclGin: every rank puts `bytes` from its send region into the next rank's receive region,
// bumps signal 0 there, and waits until its own signal 0 has reached the call's sequence number.
__global__ void __launch_bounds__(256) devApiGinRingKernel(ncclDevComm_t dc, ncclWindow_t win, size_t sendOff, size_t recvOff, size_t bytes,
                                                           unsigned long long seq, int* status) {
  ncclCoopCta cta;
  ncclGin gin(dc);
  const ncclTeam_t team = ncclTeamLsa(dc);
  const int next = (dc.lsaRank + 1) % dc.lsaSize;
  if (gin.put(cta, team, next, win, recvOff, win, sendOff, bytes, /*signal*/ 0, /*counter*/ 0) != ncclSuccess) {
    if (threadIdx.x == 0) atomicExch(status, 4);
    return;
  }
  if (threadIdx.x == 0 && gin.waitSignal(0, seq) != ncclSuccess) atomicExch(status, 5);
}

int* statusWord() {
  static thread_local int* w[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!w[dev]) {
    if (cudaMalloc(&w[dev], sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(w[dev], 0, sizeof(int));
  }
  return w[dev];
}

}  // namespace

extern "C" {

// Sum all-reduce of `count` elements (ncclFloat32 or ncclBfloat16) from sendWin+sendOff into
// recvWin+recvOff on every rank. nCtas must not exceed the device communicator's lsaBarrierCount.
ncclResult_t b200DevApiAllReduce(const ncclDevComm_t* dc, ncclWindow_t sendWin, size_t sendOff, ncclWindow_t recvWin, size_t recvOff, size_t count,
                                 ncclDataType_t type, int multimem, int nCtas, cudaStream_t stream) {
  if (!dc || !sendWin || !recvWin || nCtas < 1 || nCtas > dc->lsaBarrierCount) return ncclInvalidArgument;
  if (type != ncclFloat32 && type != ncclBfloat16) return ncclInvalidArgument;
  const size_t per = type == ncclFloat32 ? 4 : 8;
  if (count % per || sendOff % 16 || recvOff % 16) return ncclInvalidArgument;
  if (multimem && (!sendWin->mcPtr || !recvWin->mcPtr)) return ncclInvalidUsage;
  int* st = statusWord();
  if (!st) return ncclUnhandledCudaError;
  if (type == ncclFloat32)
    devApiAllReduceKernel<float><<<nCtas, kThreads, 0, stream>>>(*dc, sendWin->devSelf, sendOff, recvWin->devSelf, recvOff, count, multimem, st);
  else
    devApiAllReduceKernel<__nv_bfloat16><<<nCtas, kThreads, 0, stream>>>(*dc, sendWin->devSelf, sendOff, recvWin->devSelf, recvOff, count, multimem, st);
  return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

ncclResult_t b200DevApiArRmsNorm(const ncclDevComm_t* dc, ncclWindow_t inWin, size_t inOff, ncclWindow_t resWin, size_t resOff, ncclWindow_t outWin,
                                 size_t outOff, const void* weight, float eps, int tokens, int hidden, int mode, int nCtas, cudaStream_t stream) {
  if (!dc || !inWin || !resWin || !outWin || !weight || nCtas < 1 || nCtas > dc->lsaBarrierCount) return ncclInvalidArgument;
  if (hidden % 8 || hidden > 8 * kThreads * 4 || tokens < 0 || mode < 0 || mode > 2) return ncclInvalidArgument;
  if (inOff % 16 || resOff % 16 || outOff % 16 || (uintptr_t)weight % 16) return ncclInvalidArgument;
  if (mode == 1 && !inWin->mcPtr) return ncclInvalidUsage;
  int* st = statusWord();
  if (!st) return ncclUnhandledCudaError;
  if (dc->lsaSize == 1 && mode != 1) {
    if (tokens == 0 || hidden <= 0) return ncclSuccess;   // no rows, or rows without channels: nothing to read or write
    RowArgs a = {(const char*)inWin->peerPtr[inWin->rank] + inOff, (char*)resWin->peerPtr[resWin->rank] + resOff, (char*)outWin->peerPtr[outWin->rank] + outOff, (const char*)weight, eps, tokens, hidden, 0, 0, st};
    return launchRmsNormRows(a, nCtas, stream);
  }
  devApiArRmsNormKernel<<<nCtas, kThreads, 0, stream>>>(*dc, inWin->devSelf, inOff, resWin->devSelf, resOff, outWin->devSelf, outOff,
                                                        (const __nv_bfloat16*)weight, eps, tokens, hidden, mode, st);
  return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

// The split of a one-rank call, for tests: threads to a row, threads of all groups, rows of a chunk, chunks in the ring.
ncclResult_t b200DevApiArRmsNormPlan(int tokens, int hidden, int nCtas, int plan[4]) {
  if (!plan || tokens < 0 || hidden < 8 || hidden % 8 || hidden > 8 * kThreads * 4 || nCtas < 1) return ncclInvalidArgument;
  const RowPlan p = rowPlan(tokens, hidden, nCtas);
  plan[0] = p.group;
  plan[1] = p.threads;
  plan[2] = p.chunkRows;
  plan[3] = p.stages;
  return ncclSuccess;
}

ncclResult_t b200DevApiLLSum(const ncclDevComm_t* dc, const void* in, void* out, int slots, int nCtas, cudaStream_t stream) {
  if (!dc || !in || !out || nCtas < 1 || nCtas > dc->llA2ABlockCount || slots < 1 || slots > dc->llA2ASlotCount) return ncclInvalidArgument;
  int* st = statusWord();
  if (!st) return ncclUnhandledCudaError;
  devApiLLSumKernel<<<nCtas, 256, 0, stream>>>(*dc, (const float2*)in, (float2*)out, slots, st);
  return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

// One CTA; needs a device communicator created with at least one GIN signal and counter.
ncclResult_t b200DevApiGinRing(const ncclDevComm_t* dc, ncclWindow_t win, size_t sendOff, size_t recvOff, size_t bytes, unsigned long long seq,
                               cudaStream_t stream) {
  if (!dc || !win || dc->ginSignalCount < 1 || dc->ginCounterCount < 1) return ncclInvalidArgument;
  int* st = statusWord();
  if (!st) return ncclUnhandledCudaError;
  devApiGinRingKernel<<<1, 256, 0, stream>>>(*dc, win->devSelf, sendOff, recvOff, bytes, seq, st);
  return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

// 0 when no device-API kernel launched by this thread on the current device gave up a wait,
// otherwise the code of the wait (1 entry barrier, 2 exit barrier, 3 low-latency receive, 4 put, 5 signal, 6 a row copied
// into shared memory by the one-rank RMSNorm kernel).
// Synchronises the device and clears the word.
int b200DevApiStatus(void) {
  int* st = statusWord();
  if (!st) return -1;
  int v = -1;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  cudaMemcpy(&v, st, sizeof(int), cudaMemcpyDeviceToHost);
  if (v) cudaMemset(st, 0, sizeof(int));
  return v;
}

}  // extern "C"
