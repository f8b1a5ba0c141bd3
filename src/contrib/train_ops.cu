// Elementwise and row kernels of a decoder's training step, forward and backward: RMSNorm (with the residual addition that
// precedes it), rotary embedding, SwiGLU, and the cross entropy of the output head. Each reads its operands once and writes its
// results once, bf16 in memory and fp32 in between; as chains of framework operations they were 60 to 80 launches per layer with
// an fp32 copy of most operands in memory.
// Sizes in the comments are those of 2048 tokens of a layer with hidden 4096, 32 + 8 heads of 128, ffn 14336, or of a vocabulary of
// 16384; kernel times with cold caches. The SwiGLU backward is bound by memory (55 us, 6.4 TB/s), SwiGLU by memory and its exponential
// (35 us, 5.1 TB/s, the SMs at 72 %), the cross entropy with its gradient by its two exponentials per logit (60 us, the SMs at 80 %; its bytes
// would take 20). The small ones are bound by the latency of a row, two trips to memory with a reduction between them: RMSNorm takes 12 us
// (16 with an addition), its backward 19 and 6 for the gains, the rotation 10 (12 back).
// The reference has no model code; frameworks above it (FSDP, ZeRO) run this between its all-gather and reduce-scatter calls
// (src/collectives.cc: ncclAllGather / ncclReduceScatter).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <initializer_list>

#include "nccl.h"

namespace {

constexpr int kMaxRowThreads = 512;

// By value: bound to memory, a reference was read word by word, 16 bytes apart from lane to lane (2048 rows of 4096, caches flushed: the norm with an
// addition 21.4 us, 19.4 by value, its backward 29.5 and 27.5; kernels that load every operand at once lost nothing).
__device__ __forceinline__ void unpack8(uint4 q, float* f) {
  const __nv_bfloat162* p = (const __nv_bfloat162*)&q;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(p[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 q;
  __nv_bfloat162* p = (__nv_bfloat162*)&q;
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return q;
}

__device__ __forceinline__ float toBf16(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

// Sum over the block, the same value in every thread. `red` has 32 floats; two calls in a row need a different `red`.
__device__ __forceinline__ float blockSum(float v, float* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  const int warps = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = (threadIdx.x & 31) < warps ? red[threadIdx.x & 31] : 0.0f;
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  return v;
}

// ---------------------------------------------------------------------------------------------- RMSNorm
// One CTA per row, V packs of 8 channels per thread kept in registers between the sum of squares and the scaling.
// sum = x + add when `add` (rounded to bf16, and normalised as rounded), h = bf16(sum * rsqrt(mean(sum^2) + eps)) * gain: rounded where
// the model's own operations round, like the activation below, so that the loss is theirs.
template <int V>
__global__ void __launch_bounds__(kMaxRowThreads) rmsNormKernel(const uint4* x, const uint4* add, const uint4* gain, uint4* sum, uint4* h, float* rstd,
                                                               int packs, float eps) {
  __shared__ float red[32];
  const size_t row = (size_t)blockIdx.x * packs;
  float f[V][8], ss = 0.0f;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int p = threadIdx.x + v * blockDim.x;
    if (p < packs) {
      uint4 q = x[row + p];
      unpack8(q, f[v]);
      if (add) {
        float g[8];
        unpack8(add[row + p], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[v][i] += g[i];
        q = pack8(f[v]);
        sum[row + p] = q;
        unpack8(q, f[v]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[v][i] * f[v][i];
    }
  }
  const float r = rsqrtf(blockSum(ss, red) / (float)(packs * 8) + eps);
  if (rstd && threadIdx.x == 0) rstd[blockIdx.x] = r;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int p = threadIdx.x + v * blockDim.x;
    if (p < packs) {
      float g[8];
      unpack8(gain[p], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) g[i] *= toBf16(f[v][i] * r);
      h[row + p] = pack8(g);
    }
  }
}

// dx = res + rstd * (dh * gain - xn * mean(dh * gain * xn)), xn = x * rstd; the sum of dh * xn over the rows of this CTA goes to
// partial[blockIdx.x][channel] in fp32 (added up by colSumKernel in a fixed order). `res` is the gradient that went past the norm.
// The rows are dealt out in turn, so that a thread keeps its channels and the sums stay in registers.
template <int V>
__global__ void __launch_bounds__(kMaxRowThreads) rmsNormBackwardKernel(const uint4* x, const uint4* gain, const float* rstd, const uint4* dh, const uint4* res,
                                                                       uint4* dx, float4* partial, int rows, int packs) {
  __shared__ float red[2][32];
  float dg[V][8];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) dg[v][i] = 0.0f;
  int turn = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, turn ^= 1) {
    const size_t at = (size_t)row * packs;
    const float r = rstd[row];
    float xn[V][8], d[V][8], dot = 0.0f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int p = threadIdx.x + v * blockDim.x;
      if (p < packs) {
        float g[8];
        unpack8(x[at + p], xn[v]);
        unpack8(dh[at + p], d[v]);
        unpack8(gain[p], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xn[v][i] *= r;
          dg[v][i] += d[v][i] * xn[v][i];
          d[v][i] *= g[i];
          dot += d[v][i] * xn[v][i];
        }
      }
    }
    const float mean = blockSum(dot, red[turn]) / (float)(packs * 8);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int p = threadIdx.x + v * blockDim.x;
      if (p < packs) {
        float o[8];
        if (res) {
          unpack8(res[at + p], o);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += r * (d[v][i] - xn[v][i] * mean);
        dx[at + p] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int p = threadIdx.x + v * blockDim.x;
    if (p < packs) {
      float4* to = partial + ((size_t)blockIdx.x * packs + p) * 2;
      to[0] = make_float4(dg[v][0], dg[v][1], dg[v][2], dg[v][3]);
      to[1] = make_float4(dg[v][4], dg[v][5], dg[v][6], dg[v][7]);
    }
  }
}

// out[c] = bf16(sum over n of partial[n][c]): 32 channels per CTA, 32 slices of the rows, added in a fixed order.
__global__ void __launch_bounds__(1024) colSumKernel(const float* partial, __nv_bfloat16* out, int n, int cols) {
  __shared__ float s[32][33];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float acc = 0.0f;
  if (c < cols)
    for (int i = slice; i < n; i += 32) acc += partial[(size_t)i * cols + c];
  s[slice][lane] = acc;
  __syncthreads();
  if (slice == 0 && c < cols) {
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) sum += s[i][lane];
    out[c] = __float2bfloat16_rn(sum);
  }
}

// ---------------------------------------------------------------------------------------------- rotary embedding
// Rotates the pairs (i, i + D/2) of the first `turned` heads of qkv [tokens][heads][D] in place. One CTA per token, so that the
// divisions are of 32 bits; a thread turns 8 pairs at a time.
__global__ void __launch_bounds__(kMaxRowThreads) ropeKernel(uint4* qkv, const float4* cosT, const float4* sinT, int turned, int heads, int half8, int seq) {
  const int tok = blockIdx.x;
  uint4* mine = qkv + (size_t)tok * heads * 2 * half8;
  for (int i = threadIdx.x; i < turned * half8; i += blockDim.x) {
    const int head = i / half8, p = i - head * half8;
    uint4* at = mine + head * 2 * half8 + p;
    const size_t tab = ((size_t)(tok % seq) * half8 + p) * 2;
    float a[8], b[8], c[8], s[8], o[8];
    unpack8(at[0], a);
    unpack8(at[half8], b);
    *(float4*)c = cosT[tab];
    *(float4*)(c + 4) = cosT[tab + 1];
    *(float4*)s = sinT[tab];
    *(float4*)(s + 4) = sinT[tab + 1];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = a[j] * c[j] - b[j] * s[j];
    at[0] = pack8(o);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = b[j] * c[j] + a[j] * s[j];
    at[half8] = pack8(o);
  }
}

// A [batch][head][seq][D] gradient as attention returns it: strides in elements, channels next to each other.
struct HeadGrad {
  const __nv_bfloat16* p;
  long long batch, head, seq;
};

// The inverse rotation of dq and dk, and dv as it is, gathered into dqkv [tokens][heads + 2 kvHeads][D].
__global__ void __launch_bounds__(kMaxRowThreads) ropeBackwardKernel(HeadGrad dq, HeadGrad dk, HeadGrad dv, uint4* dqkv, const float4* cosT, const float4* sinT,
                                                                    int heads, int kvHeads, int half8, int seq) {
  const int all = heads + 2 * kvHeads, tok = blockIdx.x;
  uint4* mine = dqkv + (size_t)tok * all * 2 * half8;
  for (int i = threadIdx.x; i < all * half8; i += blockDim.x) {
    const int head = i / half8, p = i - head * half8;
    const bool isQ = head < heads, isV = head >= heads + kvHeads;
    const HeadGrad& g = isQ ? dq : isV ? dv : dk;
    const int own = isQ ? head : isV ? head - heads - kvHeads : head - heads;
    const uint4* from = (const uint4*)(g.p + (long long)(tok / seq) * g.batch + own * g.head + (long long)(tok % seq) * g.seq) + p;
    uint4 qa = from[0], qb = from[half8];
    if (!isV) {
      const size_t tab = ((size_t)(tok % seq) * half8 + p) * 2;
      float a[8], b[8], c[8], s[8], o[8];
      unpack8(qa, a);
      unpack8(qb, b);
      *(float4*)c = cosT[tab];
      *(float4*)(c + 4) = cosT[tab + 1];
      *(float4*)s = sinT[tab];
      *(float4*)(s + 4) = sinT[tab + 1];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = a[j] * c[j] + b[j] * s[j];
      qa = pack8(o);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = b[j] * c[j] - a[j] * s[j];
      qb = pack8(o);
    }
    uint4* at = mine + head * 2 * half8 + p;
    at[0] = qa;
    at[half8] = qb;
  }
}

// ---------------------------------------------------------------------------------------------- SwiGLU
// gu [rows][gate | up]; act = bf16(silu(gate)) * up.
__global__ void __launch_bounds__(256) swigluKernel(const uint4* gu, uint4* act, int packs) {
  const size_t row = blockIdx.x;
  const int p = blockIdx.y * blockDim.x + threadIdx.x;
  if (p >= packs) return;
  float g[8], u[8];
  unpack8(gu[row * 2 * packs + p], g);
  unpack8(gu[row * 2 * packs + packs + p], u);
#pragma unroll
  for (int i = 0; i < 8; ++i) u[i] *= toBf16(g[i] / (1.0f + expf(-g[i])));
  act[row * packs + p] = pack8(u);
}

// From gate, up and d(act): d(gate) and d(up) over gate and up, and act over d(act) (the gradient of the next weight needs it).
__global__ void __launch_bounds__(256) swigluBackwardKernel(uint4* gu, uint4* dact, int packs) {
  const size_t row = blockIdx.x;
  const int p = blockIdx.y * blockDim.x + threadIdx.x;
  if (p >= packs) return;
  uint4* gp = gu + row * 2 * packs + p;
  uint4* up = gp + packs;
  uint4* dp = dact + row * packs + p;
  const uint4 qg = *gp, qu = *up, qd = *dp;
  float g[8], u[8], d[8];
  unpack8(qg, g);
  unpack8(qu, u);
  unpack8(qd, d);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float sig = 1.0f / (1.0f + expf(-g[i])), silu = g[i] * sig, dd = d[i];
    d[i] = silu * u[i];
    g[i] = dd * u[i] * (sig * (1.0f + g[i] * (1.0f - sig)));
    u[i] = dd * silu;
  }
  *gp = pack8(g);
  *up = pack8(u);
  *dp = pack8(d);
}

// ---------------------------------------------------------------------------------------------- cross entropy
constexpr long long kIgnore = -100;

// count: how many rows are not ignored; ok: whether each of those has a class for its target.
__global__ void __launch_bounds__(1024) countTargetsKernel(const long long* target, int rows, int vocab, float* count, bool* ok) {
  __shared__ float red[2][32];
  float n = 0.0f, bad = 0.0f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    const long long t = target[i];
    n += t != kIgnore;
    bad += t != kIgnore && (t < 0 || t >= vocab);
  }
  n = blockSum(n, red[0]);
  bad = blockSum(bad, red[1]);
  if (threadIdx.x == 0) {
    *count = n;
    *ok = bad == 0.0f;
  }
}

// Running maximum and sum of exp(value - maximum); the comparisons keep a maximum of -inf from turning finite sums into NaN.
__device__ __forceinline__ void mergeExp(float& m, float& s, float m2, float s2) {
  const float top = fmaxf(m, m2);
  s = (m == top ? s : s * expf(m - top)) + (m2 == top ? s2 : s2 * expf(m2 - top));
  m = top;
}

// One CTA per row: log-sum-exp of the row, then d(logits) = (softmax - onehot) / count over the logits (the second read comes from
// L2). rowLoss = log-sum-exp - logit of the target; ignored rows give 0 and no gradient.
__global__ void __launch_bounds__(512) crossEntropyKernel(uint4* logits, const long long* target, const float* count, float* rowLoss, int vocab) {
  __shared__ float sm[16], ss[16], sTarget;
  const int packs = vocab / 8;
  uint4* row = logits + (size_t)blockIdx.x * packs;
  const long long t = target[blockIdx.x];
  const bool counts = t >= 0 && t < vocab;
  if (!counts) {
    for (int p = threadIdx.x; p < packs; p += blockDim.x) row[p] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) rowLoss[blockIdx.x] = 0.0f;
    return;
  }
  if (threadIdx.x == 0) sTarget = __bfloat162float(((const __nv_bfloat16*)row)[t]);
  float m = -INFINITY, s = 0.0f;
  for (int p = threadIdx.x; p < packs; p += blockDim.x) {
    float f[8];
    unpack8(row[p], f);
    float top = f[0], add = 0.0f;
#pragma unroll
    for (int i = 1; i < 8; ++i) top = fmaxf(top, f[i]);
    top = fmaxf(top, m);
#pragma unroll
    for (int i = 0; i < 8; ++i) add += f[i] == -INFINITY ? 0.0f : expf(f[i] - top);
    s = (m == top ? s : s * expf(m - top)) + add;
    m = top;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float m2 = __shfl_xor_sync(~0u, m, o), s2 = __shfl_xor_sync(~0u, s, o);
    mergeExp(m, s, m2, s2);
  }
  if ((threadIdx.x & 31) == 0) {
    sm[threadIdx.x >> 5] = m;
    ss[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  m = sm[threadIdx.x & 15];
  s = ss[threadIdx.x & 15];
#pragma unroll
  for (int o = 8; o; o >>= 1) {
    const float m2 = __shfl_xor_sync(~0u, m, o), s2 = __shfl_xor_sync(~0u, s, o);
    mergeExp(m, s, m2, s2);
  }
  const float logSum = logf(s);
  if (threadIdx.x == 0) rowLoss[blockIdx.x] = logSum - (sTarget - m);
  const float inv = 1.0f / *count;
  for (int p = threadIdx.x; p < packs; p += blockDim.x) {
    float f[8];
    unpack8(row[p], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      f[i] = expf(f[i] - m - logSum);
      if ((long long)p * 8 + i == t) f[i] -= 1.0f;
      f[i] *= inv;
    }
    row[p] = pack8(f);
  }
}

__global__ void __launch_bounds__(1024) meanLossKernel(const float* rowLoss, const float* count, float* loss, int rows) {
  __shared__ float red[32];
  float s = 0.0f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) s += rowLoss[i];
  s = blockSum(s, red);
  if (threadIdx.x == 0) *loss = s / *count;
}

// ---------------------------------------------------------------------------------------------- embedding
// out[id] = sum over the tokens with that id of dx, in fp32 in a fixed order, rounded once; all other rows are zero. Ids repeat (a padding id may
// be half of a batch), so the work is cut by tokens and not by ids: the token positions are ordered by id, a CTA adds the rows of kIdRows
// neighbours, and an id that reaches over several of them leaves fp32 sums that a third kernel adds. With a CTA per id, one row behind the
// other, 2048 tokens of 4096 channels into a table of 16384 rows took 39 us for uniform ids, 1040 with half of them one id and 2060 with all
// of them; now 39, 41 and 43, most of it the table's zeros (8192 tokens: 124, 4120 and 8160 us, now 78, 84 and 90; the framework's kernel with
// its fills and copies 762, 624 and 471).
constexpr int kIdRows = 16, kMaxIds = 8192, kPosBits = 13;
static_assert(kMaxIds == 1 << kPosBits, "positions must fit");
constexpr int kRankTokens = 32;   // of a CTA, four per warp

// keys[rank] = id << 13 | position, ascending, ids outside the table as `vocab`: the rank of a token is the number of ids below its own, and of equal
// ones ahead of it. Every CTA looks at all ids for its kRankTokens tokens (the work grows with the square of the tokens: 2048 hide behind the zeros, 8192 take 40 us). The CTAs behind
// the first `ranking` write the table's zeros meanwhile.
__global__ void __launch_bounds__(256) rankIdsKernel(const long long* ids, unsigned long long* keys, uint4* out, size_t outPacks, int tokens, int vocab, int ranking) {
  extern __shared__ uint32_t id[];
  if ((int)blockIdx.x >= ranking) {
    const size_t step = (size_t)(gridDim.x - ranking) * blockDim.x;
    for (size_t i = (size_t)(blockIdx.x - ranking) * blockDim.x + threadIdx.x; i < outPacks; i += step) out[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  for (int i = threadIdx.x; i < tokens; i += blockDim.x) {
    const long long v = ids[i];
    id[i] = v >= 0 && v < vocab ? (uint32_t)v : (uint32_t)vocab;
  }
  __syncthreads();
  constexpr int N = kRankTokens / 8;
  const int lane = threadIdx.x & 31, t0 = blockIdx.x * kRankTokens + threadIdx.x / 32 * N;
  if (t0 >= tokens) return;
  uint32_t mine[N], rank[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    mine[n] = t0 + n < tokens ? id[t0 + n] : 0;
    rank[n] = 0;
  }
  auto count = [&](int j, const uint32_t (&below)[N]) {
    const uint32_t v = id[j];
#pragma unroll
    for (int n = 0; n < N; ++n) rank[n] += v < below[n];
  };
  uint32_t withEqual[N];
#pragma unroll
  for (int n = 0; n < N; ++n) withEqual[n] = mine[n] + 1;
  const int block = t0 / 32 * 32;   // of the tokens themselves (N divides 32)
  int j = lane;
#pragma unroll 4
  for (; j < block; j += 32) count(j, withEqual);
  if (j < tokens) {
#pragma unroll
    for (int n = 0; n < N; ++n) rank[n] += id[j] < mine[n] + (j < t0 + n);
  }
#pragma unroll 4
  for (j += 32; j < tokens; j += 32) count(j, mine);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const uint32_t r = __reduce_add_sync(~0u, rank[n]);
    if (lane == n && t0 + n < tokens) keys[r] = (unsigned long long)mine[n] << kPosBits | (unsigned)(t0 + n);
  }
}

// CTA (c, slice): positions [c * kIdRows, ...) of the order, 128 packs of channels at most. Sums of an id that begins and ends here go to `out`;
// partial[c][0] takes what belongs to an id that began before, partial[c][1] the begin of one that goes on.
__global__ void __launch_bounds__(128) embeddingSumKernel(const unsigned long long* keys, const uint4* dx, uint4* out, float4* partial, int tokens, int vocab, int packs) {
  constexpr int U = 8;   // rows on their way
  __shared__ unsigned long long key[kIdRows + 2];   // with the neighbours on both sides
  const int first = blockIdx.x * kIdRows, rows = min(kIdRows, tokens - first);
  for (int i = threadIdx.x; i < rows + 2; i += blockDim.x) {
    const int at = first + i - 1;
    key[i] = at >= 0 && at < tokens ? keys[at] : ~0ull;
  }
  __syncthreads();
  const int p = blockIdx.y * blockDim.x + threadIdx.x;
  if (p >= packs) return;
  auto idOf = [&](int r) { return key[r + 1] >> kPosBits; };
  bool began = idOf(-1) == idOf(0);   // before this CTA
  float acc[8] = {};
  for (int r0 = 0; r0 < rows; r0 += U) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r0 + u < rows) v[u] = dx[(size_t)(key[r0 + u + 1] & (kMaxIds - 1)) * packs + p];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u;
      if (r >= rows) break;
      float f[8];
      unpack8(v[u], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
      const unsigned long long id = idOf(r);
      const bool goesOn = idOf(r + 1) == id;
      if (goesOn && r + 1 < rows) continue;
      if (id < (unsigned long long)vocab) {
        if (began || goesOn) {
          float4* to = partial + (((size_t)blockIdx.x * 2 + (began ? 0 : 1)) * packs + p) * 2;
          to[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
          to[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        } else {
          out[id * packs + p] = pack8(acc);
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
      began = false;
    }
  }
}

// CTA (c, slice): the id that begins in positions [c * kIdRows, ...) and goes on behind them, if there is one: 8 warps take its sums in
// turn, 256 channels each, and their results are added in order.
constexpr int kJoinQuads = 2;   // of a thread
__global__ void __launch_bounds__(256) embeddingJoinKernel(const unsigned long long* keys, const float4* partial, uint2* out, int tokens, int vocab, int hidden) {
  __shared__ float4 sums[7][kJoinQuads][32];
  const int c = blockIdx.x, last = (c + 1) * kIdRows - 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;   // never the last chunk: last + 1 < tokens
  const unsigned long long id = keys[last] >> kPosBits;
  if (id >= (unsigned long long)vocab || keys[last + 1] >> kPosBits != id) return;
  if (c > 0 && keys[c * kIdRows - 1] >> kPosBits == id) return;   // began before
  int more = 0;   // chunks that it goes on into
  for (int k = c + 1 + threadIdx.x, got = 256; got == 256; k += 256) more += got = __syncthreads_count(k * kIdRows < tokens && keys[k * kIdRows] >> kPosBits == id);
  const int quads = hidden / 4, q0 = blockIdx.y * 32 * kJoinQuads + lane;
  float4 acc[kJoinQuads];
#pragma unroll
  for (int k = 0; k < kJoinQuads; ++k) acc[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
  for (int i = warp; i <= more; i += 8) {
    const float4* from = partial + ((size_t)(c + i) * 2 + (i == 0)) * quads + q0;
#pragma unroll
    for (int k = 0; k < kJoinQuads; ++k) {
      if (q0 + k * 32 >= quads) break;
      const float4 v = from[k * 32];
      acc[k].x += v.x;
      acc[k].y += v.y;
      acc[k].z += v.z;
      acc[k].w += v.w;
    }
  }
  if (warp) {
#pragma unroll
    for (int k = 0; k < kJoinQuads; ++k) sums[warp - 1][k][lane] = acc[k];
  }
  __syncthreads();
  if (warp) return;
#pragma unroll
  for (int k = 0; k < kJoinQuads; ++k) {
    if (q0 + k * 32 >= quads) break;
    for (int w = 0; w < 7; ++w) {
      acc[k].x += sums[w][k][lane].x;
      acc[k].y += sums[w][k][lane].y;
      acc[k].z += sums[w][k][lane].z;
      acc[k].w += sums[w][k][lane].w;
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[k].x, acc[k].y), hi = __floats2bfloat162_rn(acc[k].z, acc[k].w);
    out[id * quads + q0 + k * 32] = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
  }
}

// ---------------------------------------------------------------------------------------------- launches
bool aligned16(std::initializer_list<const void*> ps) {
  uintptr_t all = 0;
  for (const void* p : ps) all |= (uintptr_t)p;
  return all % 16 == 0;
}

ncclResult_t launched() { return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError; }

int smCount() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  return sms;
}

// Threads of a CTA that owns rows of `packs` packs, and packs per thread: 1, 2 or 4; 0 for rows that are too long.
int rowShape(int packs, int* threads) {
  const int v = packs <= kMaxRowThreads ? 1 : packs <= 2 * kMaxRowThreads ? 2 : packs <= 4 * kMaxRowThreads ? 4 : 0;
  if (v) *threads = ((packs + v - 1) / v + 31) / 32 * 32;
  return v;
}

int itemThreads(int items) { return std::min(kMaxRowThreads, (items + 31) / 32 * 32); }

}  // namespace

// h = rmsnorm(x + add) * gain over rows of `hidden` channels (a multiple of 8, at most 16384); `sum` takes x + add when add is given, rstd
// [rows] (or null) what the backward needs.
extern "C" ncclResult_t b200RmsNorm(const void* x, const void* add, const void* gain, void* sum, void* h, float* rstd, int rows, int hidden, float eps,
                                    cudaStream_t stream) {
  int threads = 0;
  if (!x || !gain || !h || (add && !sum) || rows < 0 || hidden <= 0 || hidden % 8 || !aligned16({x, add, gain, sum, h})) return ncclInvalidArgument;
  const int packs = hidden / 8, v = rowShape(packs, &threads);
  if (!v) return ncclInvalidArgument;
  if (rows == 0) return ncclSuccess;
  auto fn = v == 1 ? rmsNormKernel<1> : v == 2 ? rmsNormKernel<2> : rmsNormKernel<4>;
  fn<<<rows, threads, 0, stream>>>((const uint4*)x, (const uint4*)add, (const uint4*)gain, (uint4*)sum, (uint4*)h, rstd, packs, eps);
  return launched();
}

// CTAs (and rows of fp32 partial sums) that b200RmsNormBackward uses.
extern "C" int b200RmsNormBackwardCtas(int rows) { return std::max(1, std::min(rows, smCount() * 2)); }

// partial: [b200RmsNormBackwardCtas(rows)][hidden] fp32.
extern "C" ncclResult_t b200RmsNormBackward(const void* x, const void* gain, const float* rstd, const void* dh, const void* res, void* dx, void* dgain,
                                            float* partial, int rows, int hidden, cudaStream_t stream) {
  int threads = 0;
  if (!x || !gain || !rstd || !dh || !dx || !dgain || !partial || rows <= 0 || hidden <= 0 || hidden % 8) return ncclInvalidArgument;
  if (!aligned16({x, gain, dh, res, dx, partial})) return ncclInvalidArgument;
  const int packs = hidden / 8, v = rowShape(packs, &threads), ctas = b200RmsNormBackwardCtas(rows);
  if (!v) return ncclInvalidArgument;
  auto fn = v == 1 ? rmsNormBackwardKernel<1> : v == 2 ? rmsNormBackwardKernel<2> : rmsNormBackwardKernel<4>;
  fn<<<ctas, threads, 0, stream>>>((const uint4*)x, (const uint4*)gain, rstd, (const uint4*)dh, (const uint4*)res, (uint4*)dx, (float4*)partial, rows, packs);
  colSumKernel<<<(hidden + 31) / 32, 1024, 0, stream>>>(partial, (__nv_bfloat16*)dgain, ctas, hidden);
  return launched();
}

// qkv [tokens][heads + 2 kvHeads][headDim] in place; cos and sin [seq][headDim / 2] fp32. headDim is a multiple of 16.
extern "C" ncclResult_t b200Rope(void* qkv, const float* cosT, const float* sinT, int tokens, int seq, int heads, int kvHeads, int headDim, cudaStream_t stream) {
  if (!qkv || !cosT || !sinT || tokens < 0 || seq <= 0 || heads <= 0 || kvHeads <= 0 || headDim <= 0 || headDim % 16 || !aligned16({qkv, cosT, sinT}))
    return ncclInvalidArgument;
  const int turned = heads + kvHeads, half8 = headDim / 16;
  if (tokens == 0) return ncclSuccess;
  ropeKernel<<<tokens, itemThreads(turned * half8), 0, stream>>>((uint4*)qkv, (const float4*)cosT, (const float4*)sinT, turned, heads + 2 * kvHeads, half8, seq);
  return launched();
}

// strides: batch, head and token stride of dq, dk and dv in elements, each a multiple of 8.
extern "C" ncclResult_t b200RopeBackward(const void* dq, const void* dk, const void* dv, const long long* strides, void* dqkv, const float* cosT, const float* sinT,
                                         int tokens, int seq, int heads, int kvHeads, int headDim, cudaStream_t stream) {
  if (!dq || !dk || !dv || !strides || !dqkv || !cosT || !sinT || tokens < 0 || seq <= 0 || heads <= 0 || kvHeads <= 0 || headDim <= 0 || headDim % 16)
    return ncclInvalidArgument;
  if (!aligned16({dq, dk, dv, dqkv, cosT, sinT})) return ncclInvalidArgument;
  HeadGrad g[3];
  const void* p[3] = {dq, dk, dv};
  for (int i = 0; i < 3; ++i) {
    g[i] = {(const __nv_bfloat16*)p[i], strides[3 * i], strides[3 * i + 1], strides[3 * i + 2]};
    if ((g[i].batch | g[i].head | g[i].seq) % 8) return ncclInvalidArgument;
  }
  const int half8 = headDim / 16;
  if (tokens == 0) return ncclSuccess;
  ropeBackwardKernel<<<tokens, itemThreads((heads + 2 * kvHeads) * half8), 0, stream>>>(g[0], g[1], g[2], (uint4*)dqkv, (const float4*)cosT, (const float4*)sinT,
                                                                                       heads, kvHeads, half8, seq);
  return launched();
}

// act [rows][ffn] = silu(gate) * up of gu [rows][gate | up]; ffn is a multiple of 8.
extern "C" ncclResult_t b200SwiGlu(const void* gu, void* act, int rows, int ffn, cudaStream_t stream) {
  if (!gu || !act || rows < 0 || ffn <= 0 || ffn % 8 || !aligned16({gu, act})) return ncclInvalidArgument;
  if (rows == 0) return ncclSuccess;
  swigluKernel<<<dim3(rows, (ffn / 8 + 255) / 256), 256, 0, stream>>>((const uint4*)gu, (uint4*)act, ffn / 8);
  return launched();
}

// gu becomes d(gate) | d(up), dact becomes act.
extern "C" ncclResult_t b200SwiGluBackward(void* gu, void* dact, int rows, int ffn, cudaStream_t stream) {
  if (!gu || !dact || rows < 0 || ffn <= 0 || ffn % 8 || !aligned16({gu, dact})) return ncclInvalidArgument;
  if (rows == 0) return ncclSuccess;
  swigluBackwardKernel<<<dim3(rows, (ffn / 8 + 255) / 256), 256, 0, stream>>>((uint4*)gu, (uint4*)dact, ffn / 8);
  return launched();
}

// Floats that b200EmbeddingBackward needs for `work`, 0 for more tokens than it takes.
extern "C" size_t b200EmbeddingBackwardWork(int tokens, int hidden) {
  return tokens > 0 && tokens <= kMaxIds ? ((size_t)tokens * 2 + 3) / 4 * 4 + (size_t)(tokens + kIdRows - 1) / kIdRows * 2 * hidden : 0;
}

// Gradient of an embedding table [vocab][hidden]: rows of the ids that occur are written over, all others become zero. Ids outside the table are
// left out.
extern "C" ncclResult_t b200EmbeddingBackward(const long long* ids, const void* dx, void* out, float* work, int tokens, int vocab, int hidden, cudaStream_t stream) {
  if (!ids || !dx || !out || !work || tokens <= 0 || tokens > kMaxIds || vocab <= 0 || hidden <= 0 || hidden % 8 || !aligned16({dx, out, work})) return ncclInvalidArgument;
  unsigned long long* keys = (unsigned long long*)work;
  float4* partial = (float4*)(work + ((size_t)tokens * 2 + 3) / 4 * 4);
  const int packs = hidden / 8, chunks = (tokens + kIdRows - 1) / kIdRows, threads = std::min(128, (packs + 31) / 32 * 32);
  const int ranking = (tokens + kRankTokens - 1) / kRankTokens;
  const size_t outPacks = (size_t)vocab * packs;
  const int zeroing = (int)std::min<size_t>((outPacks + 2047) / 2048, 1 << 30);   // neighbours write neighbouring pages at about the same time
  rankIdsKernel<<<ranking + zeroing, 256, tokens * 4, stream>>>(ids, keys, (uint4*)out, outPacks, tokens, vocab, ranking);
  embeddingSumKernel<<<dim3(chunks, (packs + threads - 1) / threads), threads, 0, stream>>>(keys, (const uint4*)dx, (uint4*)out, partial, tokens, vocab, packs);
  if (chunks > 1)
    embeddingJoinKernel<<<dim3(chunks - 1, (hidden / 4 + 32 * kJoinQuads - 1) / (32 * kJoinQuads)), 256, 0, stream>>>(keys, partial, (uint2*)out, tokens, vocab, hidden);
  return launched();
}

// Mean cross entropy of logits [rows][vocab] (bf16, vocab a multiple of 8) over the rows whose target is not -100; logits become their
// gradient. work: rows + 1 floats. *ok (device): whether every target is in range. Rows of targets that are not get no gradient and add
// nothing to the loss, but count in its mean.
extern "C" ncclResult_t b200CrossEntropy(void* logits, const long long* target, float* loss, float* work, void* ok, int rows, int vocab, cudaStream_t stream) {
  if (!logits || !target || !loss || !work || !ok || rows <= 0 || vocab <= 0 || vocab % 8 || !aligned16({logits})) return ncclInvalidArgument;
  countTargetsKernel<<<1, 1024, 0, stream>>>(target, rows, vocab, work + rows, (bool*)ok);
  crossEntropyKernel<<<rows, 512, 0, stream>>>((uint4*)logits, target, work + rows, work, vocab);
  meanLossKernel<<<1, 1024, 0, stream>>>(work, work + rows, loss, rows);
  return launched();
}
