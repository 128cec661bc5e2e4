// Cross entropy over a (shard of the) vocabulary: row statistics, loss terms and the in-place gradient.
//
// Replaces, for sm_100a, the ATen kernels the reference reaches (train.py:46-49 cross entropy). All of them are bound by memory:
// 16-byte accesses, fp32 math.
//
// Compiled without --use_fast_math (build.py: PRECISE), which would turn logf into an approximation: the log-sum-exp of a row is the
// fp32 sum of its maximum and the accurate fp32 logarithm whether it is taken here or, where the statistics of several vocabulary
// shards are merged first, by torch.log. (The exponentials are the fast ones, by name.)
#include "vec8.cuh"

namespace pt {

constexpr int CE_THREADS = 512;

__global__ void __launch_bounds__(CE_THREADS)
ce_stats_kernel(const bf16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ rowmax,
                float* __restrict__ sumexp, float* __restrict__ tgt, int V, long long ld, long long vocab_start) {
  __shared__ float red_m[32], red_s[32];
  pdl_enter();
  const long long row = blockIdx.x;
  const bf16* l = logits + row * ld;
  float m = -INFINITY, s = 0.f;
  const int nchunk = (ld % 8 == 0) ? V / 8 : 0;  // rows are 16-byte aligned only when ld is a multiple of 8
  for (int c = threadIdx.x; c < nchunk; c += CE_THREADS) {
    float v[8];
    unpack8(*reinterpret_cast<const bf16x8*>(l + c * 8), v);
    float cm = v[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) cm = fmaxf(cm, v[j]);
    const float nm = fmaxf(m, cm);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += __expf(v[j] - nm);
    s = s * __expf(m - nm) + acc;
    m = nm;
  }
  for (int i = nchunk * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    const float v = __bfloat162float(l[i]);
    const float nm = fmaxf(m, v);
    s = s * __expf(m - nm) + __expf(v - nm);
    m = nm;
  }
  // merge (m, s) pairs: warp, then block
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o);
    const float os = __shfl_xor_sync(0xffffffffu, s, o);
    const float nm = fmaxf(m, om);
    s = (nm == -INFINITY) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red_m[warp] = m;
    red_s[warp] = s;
  }
  __syncthreads();
  if (warp == 0) {
    m = lane < CE_THREADS / 32 ? red_m[lane] : -INFINITY;
    s = lane < CE_THREADS / 32 ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o);
      const float os = __shfl_xor_sync(0xffffffffu, s, o);
      const float nm = fmaxf(m, om);
      s = (nm == -INFINITY) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
      m = nm;
    }
    if (lane == 0) {
      rowmax[row] = m;
      sumexp[row] = s;
      const long long t = targets[row] - vocab_start;
      tgt[row] = (t >= 0 && t < V) ? __bfloat162float(l[t]) : 0.f;
    }
  }
}

// A row's maximum and sum of exponentials from the per-tile pairs the LM-head GEMM's epilogue left (one warp). The sum of two lanes'
// products is rounded in another order in each, so the lanes' results differ in the last bits: the row's is that of lane 0.
__device__ __forceinline__ float2 merge_tiles(const float2* __restrict__ part, int tiles) {
  float m = -INFINITY, s = 0.f;
  for (int t = threadIdx.x & 31; t < tiles; t += 32) {
    const float2 p = part[t];
    const float nm = fmaxf(m, p.x);
    s = (nm == -INFINITY) ? 0.f : s * __expf(m - nm) + p.y * __expf(p.x - nm);
    m = nm;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o);
    const float os = __shfl_xor_sync(0xffffffffu, s, o);
    const float nm = fmaxf(m, om);
    s = (nm == -INFINITY) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  return make_float2(m, s);
}
// log-sum-exp of a row, in every lane, to the bit what rowmax + torch.log(sumexp) of ce_combine_kernel's results gives (no contraction
// into the logarithm's last step)
__device__ __forceinline__ float lse_of(float2 ms) { return __shfl_sync(0xffffffffu, __fadd_rn(ms.x, logf(ms.y)), 0); }

// Loss terms lse - target logit from the tile pairs alone: one warp per row. A target outside [0, V) counts as logit 0, as in
// ce_stats_kernel (the GEMM's epilogue did not write its slot).
__global__ void __launch_bounds__(256)
ce_loss_kernel(const float2* __restrict__ part, const long long* __restrict__ targets, const float* __restrict__ tgt,
               float* __restrict__ terms, long long T, int tiles, int V, long long vocab_start) {
  pdl_enter();
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= T) return;
  const float z = lse_of(merge_tiles(part + row * tiles, tiles));
  if ((threadIdx.x & 31) == 0) {
    const long long t = targets[row] - vocab_start;
    terms[row] = z - (t >= 0 && t < V ? tgt[row] : 0.f);
  }
}

// In-place gradient (softmax - onehot) * scale of a row of logits per CTA; bound by reading and writing the logits. TILES: the
// row's log-sum-exp comes straight from the tile pairs of the LM-head GEMM and its loss term is left in `terms`, instead of from `lse`. Every
// warp of the CTA merges the pairs for itself (8 bytes per 256 columns, 1.5 KB a row of 49152 and 4 KB of 128256, from L2 but for the first).
// Measured, us, 2048 x 49152 / 2048 x 128256 behind a GEMM with K = 64: GEMM and this kernel 186 / 479; GEMM, clearing and merging kernel and the
// gradient from a given lse 182 / 461 (the gradient alone 69.5 / 180, at the copy rate 62 / 163), without the logarithm, the differences and their
// sum, which were launches of their own.
template <bool TILES>
__global__ void __launch_bounds__(CE_THREADS)
ce_grad_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets, const float* __restrict__ lse,
               int V, long long ld, float scale, long long vocab_start, const float2* __restrict__ part, int tiles,
               const float* __restrict__ tgt, float* __restrict__ terms) {
  pdl_enter();
  const long long row = blockIdx.x;
  bf16* l = logits + row * ld;
  const float z = TILES ? lse_of(merge_tiles(part + row * tiles, tiles)) : lse[row];
  const long long t = targets[row] - vocab_start;
  if (TILES && threadIdx.x == 0) terms[row] = z - (t >= 0 && t < V ? tgt[row] : 0.f);
  const int nchunk = (ld % 8 == 0) ? V / 8 : 0;
  for (int c = threadIdx.x; c < nchunk; c += CE_THREADS) {
    float v[8];
    unpack8(*reinterpret_cast<const bf16x8*>(l + c * 8), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(v[j] - z);
      if ((long long)(c * 8 + j) == t) p -= 1.f;
      v[j] = p * scale;
    }
    *reinterpret_cast<bf16x8*>(l + c * 8) = pack8(v);
  }
  for (int i = nchunk * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    float p = __expf(__bfloat162float(l[i]) - z);
    if ((long long)i == t) p -= 1.f;
    l[i] = __float2bfloat16(p * scale);
  }
}

// Merge the per-tile (max, sum-exp) pairs the LM-head GEMM's epilogue left in part[T, tiles]: one warp per row.
__global__ void __launch_bounds__(256)
ce_combine_kernel(const float2* __restrict__ part, float* __restrict__ rowmax, float* __restrict__ sumexp, long long T, int tiles) {
  pdl_enter();
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= T) return;
  const float2 ms = merge_tiles(part + row * tiles, tiles);
  if (lane == 0) {
    rowmax[row] = ms.x;
    sumexp[row] = ms.y;
  }
}

}  // namespace pt

using namespace pt;

extern "C" int pt_ce_stats(const void* logits, const long long* targets, float* rowmax, float* sumexp, float* tgt,
                           long long T, int V, long long ld, long long vocab_start, cudaStream_t st) {
  if (T == 0) return 0;
  launch_pdl(ce_stats_kernel, dim3((unsigned)T), dim3(CE_THREADS), 0, st, (const bf16*)logits, targets, rowmax, sumexp, tgt, V, ld,
             vocab_start);
  return check_launch();
}

extern "C" int pt_ce_combine(const void* part, float* rowmax, float* sumexp, long long T, int tiles, cudaStream_t st) {
  if (T == 0) return 0;
  launch_pdl(ce_combine_kernel, dim3((unsigned)((T + 7) / 8)), dim3(256), 0, st, (const float2*)part, rowmax, sumexp, T, tiles);
  return check_launch();
}

extern "C" int pt_ce_grad(void* logits, const long long* targets, const float* lse, long long T, int V, long long ld,
                          float scale, long long vocab_start, cudaStream_t st) {
  if (T == 0) return 0;
  launch_pdl(ce_grad_kernel<false>, dim3((unsigned)T), dim3(CE_THREADS), 0, st, (bf16*)logits, targets, lse, V, ld, scale, vocab_start,
             nullptr, 0, nullptr, nullptr);
  return check_launch();
}

// Loss terms (lse - target logit) of T rows from the tile pairs and target logits of pt_gemm_bf16_ce; with `logits` also the in-place
// gradient (softmax - onehot) * scale. One launch instead of the merging kernel, the logarithm, the differences, their sum and the
// clearing of `tgt` as launches of their own.
extern "C" int pt_ce_finish(void* logits, const void* part, int tiles, const long long* targets, const float* tgt, float* terms,
                            long long T, int V, long long ld, float scale, long long vocab_start, cudaStream_t st) {
  if (T == 0) return 0;
  if (logits != nullptr)
    launch_pdl(ce_grad_kernel<true>, dim3((unsigned)T), dim3(CE_THREADS), 0, st, (bf16*)logits, targets, nullptr, V, ld, scale,
               vocab_start, (const float2*)part, tiles, tgt, terms);
  else
    launch_pdl(ce_loss_kernel, dim3((unsigned)((T + 7) / 8)), dim3(256), 0, st, (const float2*)part, targets, tgt, terms, T, tiles, V,
               vocab_start);
  return check_launch();
}
