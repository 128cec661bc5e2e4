// Memory-bound kernels of the model: RMSNorm (+residual) fwd/bwd, RoPE, SwiGLU, embedding, fp32 gradient accumulation,
// multi-tensor AdamW, attention-partial merge, add.
//
// They replace, for sm_100a, the Triton/ATen kernels the reference reaches (picotron/model.py:54-65 RMSNorm,
// :136-137 RoPE, :186 SiLU*mul, :251 embedding; data_parallel.py:131 grad accumulation; train.py:209,235 AdamW;
// context_parallel.py:157-187 LSE merge).
// All of them are bandwidth-bound: 16-byte vector accesses, fp32 math, one pass over HBM per tensor.
#include "vec8.cuh"

#include <type_traits>
#include "noalloc.h"

namespace pt {

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < THREADS / 32) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

// ---------------------------------------------------------------------------------------------
// RMSNorm: block size and column chunks per thread of the partial-sum backward below (H % 8 == 0, H <= 8 * THREADS * MAXC)
// ---------------------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_MAXC = 4;

// ---------------------------------------------------------------------------------------------
// RMSNorm backward. dx = rstd * (w*dy - xhat * mean(xhat * w*dy)) (+ dres);  dw = sum_rows dy * xhat.
// A persistent grid walks the rows; every CTA keeps its dw partial in registers and writes it to
// `partial[grid, H]` (scratch), a second kernel sums the partials.
// ---------------------------------------------------------------------------------------------
template <int MAXC>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                   const float* __restrict__ rstd_in, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                   float* __restrict__ partial, int T, int H) {
  __shared__ float red[32];
  const int nchunk = H / 8;
  float wv[MAXC][8];
  float dwacc[MAXC][8];
#pragma unroll
  for (int i = 0; i < MAXC; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
    if (c < nchunk) unpack8(*reinterpret_cast<const bf16x8*>(w + c * 8), wv[i]);
  }
  for (long long row = blockIdx.x; row < T; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float xh[MAXC][8], wdy[MAXC][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < MAXC; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c < nchunk) {
        float xv[8], dv[8];
        unpack8(*reinterpret_cast<const bf16x8*>(x + row * H + c * 8), xv);
        unpack8(*reinterpret_cast<const bf16x8*>(dy + row * H + c * 8), dv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[i][j] = xv[j] * rstd;
          wdy[i][j] = dv[j] * wv[i][j];
          dot += xh[i][j] * wdy[i][j];
          dwacc[i][j] += dv[j] * xh[i][j];
        }
      }
    }
    dot = block_sum<NORM_THREADS>(dot, red);
    const float cmean = dot / (float)H;
#pragma unroll
    for (int i = 0; i < MAXC; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c < nchunk) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (wdy[i][j] - xh[i][j] * cmean) * rstd;
        if (dres != nullptr) {
          float r[8];
          unpack8(*reinterpret_cast<const bf16x8*>(dres + row * H + c * 8), r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        *reinterpret_cast<bf16x8*>(dx + row * H + c * 8) = pack8(o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MAXC; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nchunk) {
      float4* dst = reinterpret_cast<float4*>(partial + (long long)blockIdx.x * H + c * 8);
      dst[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
      dst[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
    }
  }
}

// out[col] = sum_p partial[p, col]. Block = 32 columns x 8 row-slices; grid = ceil(H / 32).
__global__ void __launch_bounds__(256)
reduce_partials_kernel(const float* __restrict__ partial, float* __restrict__ out, int nparts, int H) {
  __shared__ float red[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (col < H)
    for (int p = ry; p < nparts; p += 8) s += partial[(long long)p * H + col];
  red[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && col < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i][cx];
    out[col] = t;
  }
}

// ---------------------------------------------------------------------------------------------
// RoPE, NeoX (half-split) layout, in place on the first n_rot heads of every row of a packed
// [T, row_stride] activation. cos/sin: fp32 [S, d/2]. Row t is at position t % S.
// One thread handles 8 consecutive elements of the first half and their partners in the second half.
// ---------------------------------------------------------------------------------------------
__global__ void rope_kernel(bf16* __restrict__ qkv, const float* __restrict__ cosT, const float* __restrict__ sinT,
                            long long total, int n_rot, int d, int S, long long row_stride, float sign) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int half = d / 2;
  const int cpp = half / 8;  // chunks per head
  const int c = (int)(idx % cpp);
  const long long hr = idx / cpp;
  const int head = (int)(hr % n_rot);
  const long long row = hr / n_rot;
  const int pos = (int)(row % S);
  bf16* p1 = qkv + row * row_stride + (long long)head * d + c * 8;
  bf16* p2 = p1 + half;
  float a[8], b[8], cs[8], sn[8];
  unpack8(*reinterpret_cast<const bf16x8*>(p1), a);
  unpack8(*reinterpret_cast<const bf16x8*>(p2), b);
  const float4* c4 = reinterpret_cast<const float4*>(cosT + (long long)pos * half + c * 8);
  const float4* s4 = reinterpret_cast<const float4*>(sinT + (long long)pos * half + c * 8);
  float4 t;
  t = c4[0]; cs[0] = t.x; cs[1] = t.y; cs[2] = t.z; cs[3] = t.w;
  t = c4[1]; cs[4] = t.x; cs[5] = t.y; cs[6] = t.z; cs[7] = t.w;
  t = s4[0]; sn[0] = t.x; sn[1] = t.y; sn[2] = t.z; sn[3] = t.w;
  t = s4[1]; sn[4] = t.x; sn[5] = t.y; sn[6] = t.z; sn[7] = t.w;
  float o1[8], o2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float s = sn[j] * sign;
    o1[j] = a[j] * cs[j] - b[j] * s;
    o2[j] = b[j] * cs[j] + a[j] * s;
  }
  *reinterpret_cast<bf16x8*>(p1) = pack8(o1);
  *reinterpret_cast<bf16x8*>(p2) = pack8(o2);
}

// ---------------------------------------------------------------------------------------------
// SwiGLU on packed [T, 2I] pre-activations (gate | up)
// ---------------------------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ out, long long total8, int I8) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total8) return;
  const long long row = idx / I8;
  const int c = (int)(idx % I8);
  const bf16* g = gu + row * (long long)(I8 * 16) + c * 8;
  float gv[8], uv[8], o[8];
  unpack8(*reinterpret_cast<const bf16x8*>(g), gv);
  unpack8(*reinterpret_cast<const bf16x8*>(g + I8 * 8), uv);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sig = 1.f / (1.f + __expf(-gv[j]));
    o[j] = gv[j] * sig * uv[j];
  }
  *reinterpret_cast<bf16x8*>(out + row * (long long)(I8 * 8) + c * 8) = pack8(o);
}

__global__ void swiglu_bwd_kernel(const bf16* __restrict__ gu, const bf16* __restrict__ da, bf16* __restrict__ dgu,
                                  long long total8, int I8) {
  pdl_enter();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total8) return;
  const long long row = idx / I8;
  const int c = (int)(idx % I8);
  const long long off = row * (long long)(I8 * 16) + c * 8;
  float gv[8], uv[8], dv[8], dg[8], du[8];
  unpack8(*reinterpret_cast<const bf16x8*>(gu + off), gv);
  unpack8(*reinterpret_cast<const bf16x8*>(gu + off + I8 * 8), uv);
  unpack8(*reinterpret_cast<const bf16x8*>(da + row * (long long)(I8 * 8) + c * 8), dv);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sig = 1.f / (1.f + __expf(-gv[j]));
    const float silu = gv[j] * sig;
    dg[j] = dv[j] * uv[j] * (sig * (1.f + gv[j] * (1.f - sig)));
    du[j] = dv[j] * silu;
  }
  *reinterpret_cast<bf16x8*>(dgu + off) = pack8(dg);
  *reinterpret_cast<bf16x8*>(dgu + off + I8 * 8) = pack8(du);
}

// ---------------------------------------------------------------------------------------------
// (vocab-parallel) embedding: rows for ids in [vocab_start, vocab_start + rows), zeros otherwise
// ---------------------------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ w,
                                     bf16* __restrict__ out, int H8, long long rows, long long vocab_start) {
  pdl_enter();
  const long long tok = blockIdx.x;
  const long long id = ids[tok] - vocab_start;
  const bool ok = id >= 0 && id < rows;
  const uint4* src = reinterpret_cast<const uint4*>(w + (ok ? id : 0) * (long long)(H8 * 8));
  uint4* dst = reinterpret_cast<uint4*>(out + tok * (long long)(H8 * 8));
  for (int c = threadIdx.x; c < H8; c += blockDim.x) dst[c] = ok ? src[c] : make_uint4(0, 0, 0, 0);
}

// dw[id] += dy of every token with that id. Bound by the reductions at L2 (fp32, 4 bytes a column): 16-byte ones where the destination
// allows it. One thread per 8 columns of a token, whatever the width (a CTA per token left 184 of 256 threads idle at 576 columns).
// 4096 x 2048 into 49152 rows: 54 us with scalar reductions, 25 us with vector ones (3.4 TB/s of the 84 MB read and reduced).
template <bool VEC>
__global__ void __launch_bounds__(256)
embedding_bwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ dy, float* __restrict__ dw, long long T, int H8,
                     long long rows, long long vocab_start) {
  pdl_enter();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long tok = i / H8;
  if (tok >= T) return;
  const int c = (int)(i - tok * H8);
  const long long id = ids[tok] - vocab_start;
  if (id < 0 || id >= rows) return;
  float* dst = dw + (id * H8 + c) * 8;
  float v[8];
  unpack8(*reinterpret_cast<const bf16x8*>(dy + i * 8), v);
  if (VEC) {
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + j), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3])
                   : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) atomicAdd(dst + j, v[j]);
  }
}

// ---------------------------------------------------------------------------------------------
// fp32 += bf16 ; bf16 add
// ---------------------------------------------------------------------------------------------
__global__ void accumulate_kernel(float* __restrict__ acc, const bf16* __restrict__ g, long long n) {
  const long long i8 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i8 + 8 <= n) {
    float v[8];
    unpack8(*reinterpret_cast<const bf16x8*>(g + i8), v);
    float4* a = reinterpret_cast<float4*>(acc + i8);
    float4 a0 = a[0], a1 = a[1];
    a0.x += v[0]; a0.y += v[1]; a0.z += v[2]; a0.w += v[3];
    a1.x += v[4]; a1.y += v[5]; a1.z += v[6]; a1.w += v[7];
    a[0] = a0;
    a[1] = a1;
  } else {
    for (long long i = i8; i < n; ++i) acc[i] += __bfloat162float(g[i]);
  }
}

__global__ void accumulate_f32_kernel(float* __restrict__ acc, const float* __restrict__ g, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) acc[i] += g[i];
}

__global__ void add_kernel(const bf16* __restrict__ a, const bf16* __restrict__ b, bf16* __restrict__ out, long long n) {
  pdl_enter();
  const long long i8 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i8 + 8 <= n) {
    float x[8], y[8];
    unpack8(*reinterpret_cast<const bf16x8*>(a + i8), x);
    unpack8(*reinterpret_cast<const bf16x8*>(b + i8), y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    *reinterpret_cast<bf16x8*>(out + i8) = pack8(x);
  } else {
    for (long long i = i8; i < n; ++i) out[i] = __float2bfloat16(__bfloat162float(a[i]) + __bfloat162float(b[i]));
  }
}

// ---------------------------------------------------------------------------------------------
// multi-tensor AdamW (decoupled weight decay), fp32 gradients, fp32 or bf16 moments, optional fp32 master
// ---------------------------------------------------------------------------------------------
// Bound by memory: 30 bytes per parameter (gradient, moments and master in; moments, master and bf16 weight out). One launch
// takes up to 256 tensors (their table travels as a kernel parameter), one block one chunk of 4096 elements of one tensor,
// found by bisection of the chunk prefix sums, so that the grid fills the chip whatever the tensors' sizes; 16-byte accesses
// where every pointer of the tensor allows them. Clipping + AdamW of 667M parameters (two layers of the 7B shape with its
// embedding and head): 6.72 -> 4.42 ms when the gradients are scaled (42 bytes per parameter, 0.98 of the copy rate), 6.77 -> 3.69 ms
// when there is nothing to clip (34 bytes, 0.95). (Before: launches of at most 320 blocks, 4-byte accesses, and a library multiply
// at 3.1 TB/s for the clipping, also by 1.)
constexpr int ADAM_MAX_TENSORS = 256;
constexpr int ADAM_THREADS = 256;
constexpr int ADAM_CHUNK = 4096;

struct AdamTensor {
  void* param;
  const float* grad;
  float* m;
  float* v;
  float* master;
  long long numel;
};
struct AdamArgs {
  AdamTensor t[ADAM_MAX_TENSORS];
  unsigned first_block[ADAM_MAX_TENSORS + 1];      // first block of each tensor; [count] = grid size
  unsigned char vec[ADAM_MAX_TENSORS];             // 1: every pointer is aligned for 4-element accesses
  int count;
};
static_assert(sizeof(AdamArgs) <= 32000, "kernel parameter limit");

// (Explicit fused operations: left to the compiler, the whole and the partial chunks of a tensor were rounded differently.)
__device__ __forceinline__ void adam_update(float& w, float& m, float& v, float g, float lr, float beta1, float beta2, float eps,
                                            float wd, float bc1, float bc2_sqrt) {
  m = fmaf(g, 1.f - beta1, m * beta1);
  v = fmaf(g * g, 1.f - beta2, v * beta2);
  w = fmaf(w, 1.f - lr * wd, -((lr / bc1) * (m / (sqrtf(v) / bc2_sqrt + eps))));
}

template <bool PARAM_BF16>
__global__ void __launch_bounds__(ADAM_THREADS)
adamw_kernel(const __grid_constant__ AdamArgs args, float lr, float beta1, float beta2, float eps, float wd,
             float bc1, float bc2_sqrt) {
  int lo = 0, hi = args.count;                     // the tensor of this block: first_block[lo] <= blockIdx.x < first_block[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (args.first_block[mid] <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  const AdamTensor& t = args.t[lo];
  const long long base = (long long)(blockIdx.x - args.first_block[lo]) * ADAM_CHUNK;
  const long long end = min(base + ADAM_CHUNK, t.numel);
  if (args.vec[lo] && end - base == ADAM_CHUNK) {
    constexpr int ITERS = ADAM_CHUNK / (4 * ADAM_THREADS);
#pragma unroll 2
    for (int k = 0; k < ITERS; ++k) {
      const long long i = base + (long long)(k * ADAM_THREADS + threadIdx.x) * 4;
      const float4 g = __ldcs(reinterpret_cast<const float4*>(t.grad + i));
      float4 m = __ldcs(reinterpret_cast<const float4*>(t.m + i));
      float4 v = __ldcs(reinterpret_cast<const float4*>(t.v + i));
      float4 w;
      if (t.master != nullptr) {
        w = __ldcs(reinterpret_cast<const float4*>(t.master + i));
      } else if (PARAM_BF16) {
        const uint2 q = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(t.param) + i);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.y));
        w = make_float4(a.x, a.y, b.x, b.y);
      } else {
        w = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(t.param) + i);
      }
      adam_update(w.x, m.x, v.x, g.x, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
      adam_update(w.y, m.y, v.y, g.y, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
      adam_update(w.z, m.z, v.z, g.z, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
      adam_update(w.w, m.w, v.w, g.w, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
      __stcs(reinterpret_cast<float4*>(t.m + i), m);
      __stcs(reinterpret_cast<float4*>(t.v + i), v);
      if (t.master != nullptr) __stcs(reinterpret_cast<float4*>(t.master + i), w);
      if (PARAM_BF16) {
        uint2 q;
        q.x = pack_bf16(w.x, w.y);
        q.y = pack_bf16(w.z, w.w);
        *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(t.param) + i) = q;
      } else {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(t.param) + i) = w;
      }
    }
    return;
  }
  for (long long i = base + threadIdx.x; i < end; i += ADAM_THREADS) {
    float w;
    if (t.master != nullptr) w = t.master[i];
    else if (PARAM_BF16) w = __bfloat162float(reinterpret_cast<bf16*>(t.param)[i]);
    else w = reinterpret_cast<float*>(t.param)[i];
    float m = t.m[i], v = t.v[i];
    adam_update(w, m, v, t.grad[i], lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
    t.m[i] = m;
    t.v[i] = v;
    if (t.master != nullptr) t.master[i] = w;
    if (PARAM_BF16) reinterpret_cast<bf16*>(t.param)[i] = __float2bfloat16(w);
    else reinterpret_cast<float*>(t.param)[i] = w;
  }
}

// x *= *coef over a contiguous fp32 buffer (gradient clipping). Bound by memory: 8 bytes per element; a coefficient of exactly
// 1 (nothing to clip) leaves the buffer untouched without reading it.
constexpr int SCALE_CHUNK = 8192;
__global__ void __launch_bounds__(256) scale_kernel(float* __restrict__ x, const float* __restrict__ coef, long long n) {
  const float c = *coef;
  if (c == 1.f) return;
  const long long base = (long long)blockIdx.x * SCALE_CHUNK;
  const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  if (aligned && base + SCALE_CHUNK <= n) {
#pragma unroll
    for (int k = 0; k < SCALE_CHUNK / 1024; ++k) {
      float4* q = reinterpret_cast<float4*>(x + base) + k * 256 + threadIdx.x;
      float4 v = __ldcs(q);
      v.x *= c; v.y *= c; v.z *= c; v.w *= c;
      __stcs(q, v);
    }
  } else {
    for (long long i = base + threadIdx.x; i < n && i < base + SCALE_CHUNK; i += 256) x[i] *= c;
  }
}

// ---------------------------------------------------------------------------------------------
// merge of two attention partials (ring attention): out fp32 [B,S,h,d], lse fp32 [B,h,S]
//   out -= sigmoid(bl - l) * (out - block_out);   l -= logsigmoid(l - bl)
// ---------------------------------------------------------------------------------------------
__global__ void merge_attention_kernel(float* __restrict__ out, float* __restrict__ lse, const bf16* __restrict__ bo,
                                       const float* __restrict__ bl, int B, int S, int h, int d) {
  // one warp per (b, s, head)
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long total = (long long)B * S * h;
  if (wid >= total) return;
  const int head = (int)(wid % h);
  const long long bs = wid / h;
  const int s = (int)(bs % S);
  const int b = (int)(bs / S);
  const long long li = ((long long)b * h + head) * S + s;
  const float l = lse[li], nb = bl[li];
  const float sig = 1.f / (1.f + __expf(l - nb));          // sigmoid(nb - l)
  float* o = out + wid * d;
  const bf16* n = bo + wid * d;
  for (int j = lane; j < d; j += 32) o[j] -= sig * (o[j] - __bfloat162float(n[j]));
  __syncwarp();
  if (lane == 0) {
    // l - logsigmoid(l - nb) = l + log(1 + exp(nb - l)) computed stably
    const float mx = fmaxf(l, nb);
    lse[li] = mx + __logf(__expf(l - mx) + __expf(nb - mx));
  }
}

}  // namespace pt

// ===============================================================================================
// C launch API (raw pointers; the Python bindings validate shapes and dtypes)
// ===============================================================================================
using namespace pt;

// ---------------------------------------------------------------------------------------------
// RMSNorm kernels of the training step. Bound by memory: 4 (forward), 8 (with the residual add) and 8 (backward) bytes per
// element. A TEAM of 32, 64, 128 or 256 threads holds one row, at most 4 16-byte chunks per thread, so that a row is one batch
// of loads, one reduction among the team's own warps and one batch of stores, and a CTA of 256 threads works on 256 / TEAM
// independent rows. Forward: one row per team and a CTA for every 256 / TEAM rows. Backward: three CTAs per SM (two where a thread
// holds more than two chunks) walk the rows; a thread's columns never change, so the weight gradient is summed in registers, then
// over the CTA's teams in shared memory, and added to the destination once per CTA.
//   forward :  x_new = x (+ delta); rstd = rsqrt(mean(x_new^2) + eps); y = x_new * rstd * w
//   backward:  dx = rstd * (w*dy - xhat * mean(xhat*w*dy)) (+ dres);  dw_acc += sum_rows dy * xhat   (fp32 reductions)
// H % 8 == 0, H <= 8 * 4 * TEAM. (Before, the whole CTA held four rows at a time: at H = 576 two thirds of its threads had no
// column, and every four rows waited for one CTA barrier. Measured then
// and now, us, launch included: forward / with add / backward of 8192 x 576: 15.2 -> 11.3 / 17.5 -> 15.0 / 27.6 -> 17.5;
// 4096 x 960: 12.3 -> 10.2 / 14.4 / 20.6 -> 16.4; 4096 x 2048: 14.3 / 20.5 -> 18.5 / 24.6 -> 22.6; wide rows gain nothing: 4096 x
// 4096: 20.5 -> 21.4 / 30.7 / 41.9 -> 43.0, 32768 x 2048: 56.3 -> 59.4 / 95.1 -> 94.2 / 110.6 -> 104.4.)
// The backward's next rows travel through shared memory while one is reduced (its rows were one load latency after the other). Without /
// with, us, inputs not in L2: 8192 x 256: 7.3 -> 6.8, 8192 x 512: 9.9 -> 9.3, 8192 x 576: 12.1 -> 10.6, 8192 x 960: 17.9 -> 14.3, 2048 x 2048: 10.6 -> 9.6,
// 32768 x 2048: 96.8 -> 81.1 (6.6 TB/s), 8192 x 4096: 60.1 -> 54.4, 8192 x 8192: 107.8 -> 93.4; few rows have nothing to fetch ahead (512 x 2048:
// 5.7 -> 5.2, 512 x 264: 2.7 -> 2.8).
// ---------------------------------------------------------------------------------------------
constexpr int ROWS_THREADS = 256;

// Sum over a row. Its order is the same for every team size: the 16-byte chunks c, c + 256, ... go to one running sum, 32
// neighbouring running sums are added by a warp (butterfly), and the eight warp sums so obtained as
// (((0 + 1) + (2 + 3)) + (4 + 5)) + (6 + 7). So a thread of a small team keeps a running sum per chunk (`acc_of`), each reduced by
// itself: results do not depend on how a row is dealt to threads. `red` has 8 floats per team and parity of `it`.
template <int TEAM> __host__ __device__ constexpr int acc_of(int i) { return i % (ROWS_THREADS / TEAM); }
template <int TEAM, int NC> __host__ __device__ constexpr int accs() { return NC < ROWS_THREADS / TEAM ? NC : ROWS_THREADS / TEAM; }

// Warp sums of four values at once, each as warp_sum gives it: the first two steps of the butterflies share their shuffles,
// because a lane needs to go on with only one of the values. Value a ends up in the lanes [8 a, 8 a + 8).
__device__ __forceinline__ float warp_sums4(float v0, float v1, float v2, float v3) {
  constexpr unsigned FULL = 0xffffffffu;
  const bool b16 = threadIdx.x & 16, b8 = threadIdx.x & 8;
  const float k0 = (b16 ? v2 : v0) + __shfl_xor_sync(FULL, b16 ? v0 : v2, 16);
  const float k1 = (b16 ? v3 : v1) + __shfl_xor_sync(FULL, b16 ? v1 : v3, 16);
  float k = (b8 ? k1 : k0) + __shfl_xor_sync(FULL, b8 ? k0 : k1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(FULL, k, o);
  return k;
}

template <int TEAM, int NA>
__device__ __forceinline__ float row_sum(float (&v)[NA], float* red, int it) {
  constexpr int WARPS = TEAM / 32;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float k = 0.f;
  if constexpr (NA > 2) {
    k = warp_sums4(v[0], v[1], v[2], NA > 3 ? v[NA - 1] : 0.f);
  } else {
#pragma unroll
    for (int a = 0; a < NA; ++a) v[a] = warp_sum(v[a]);
  }
  if constexpr (WARPS == 1) {
#pragma unroll
    for (int a = 0; a < NA; ++a) s[a] = NA > 2 ? __shfl_sync(0xffffffffu, k, a * 8) : v[a];
  } else {
    const int warp = (threadIdx.x % TEAM) >> 5, team = threadIdx.x / TEAM, lane = threadIdx.x & 31;
    float* buf = red + ((it & 1) * (ROWS_THREADS / TEAM) + team) * 8;
    if constexpr (NA > 2) {
      if (lane % 8 == 0 && lane / 8 < NA) buf[lane / 8 * WARPS + warp] = k;
    } else if (lane == 0) {
#pragma unroll
      for (int a = 0; a < NA; ++a) buf[a * WARPS + warp] = v[a];
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(TEAM) : "memory");
#pragma unroll
    for (int i = 0; i < NA * WARPS; ++i) s[i] = buf[i];
  }
  return (((s[0] + s[1]) + (s[2] + s[3])) + (s[4] + s[5])) + (s[6] + s[7]);
}

template <bool ADD, int TEAM, int NC>
__global__ void __launch_bounds__(ROWS_THREADS)
rmsnorm_fwd_rows_kernel(const bf16* __restrict__ x, const bf16* __restrict__ delta, const bf16* __restrict__ w,
                        bf16* __restrict__ x_new, bf16* __restrict__ y, float* __restrict__ rstd_out, int T, int H, float eps) {
  __shared__ __align__(16) float red[ROWS_THREADS / TEAM * 8];
  pdl_enter();
  const int nchunk = H / 8, tid = threadIdx.x % TEAM;
  const long long row = (long long)blockIdx.x * (ROWS_THREADS / TEAM) + threadIdx.x / TEAM;
  if (row >= T) return;                              // (a whole team: its barrier is its own)
  bf16x8 px[NC], pd[NC], wv[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = tid + i * TEAM;
    if (c < nchunk) {
      px[i] = *reinterpret_cast<const bf16x8*>(x + row * H + c * 8);
      if (ADD) pd[i] = *reinterpret_cast<const bf16x8*>(delta + row * H + c * 8);
      wv[i] = *reinterpret_cast<const bf16x8*>(w + c * 8);
    }
  }
  float ss[accs<TEAM, NC>()] = {};
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = tid + i * TEAM;
    if (c < nchunk) {
      float v[8];
      unpack8(px[i], v);
      if (ADD) {
        float d[8];
        unpack8(pd[i], d);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += d[j];
        px[i] = pack8(v);                              // the rounded residual stream is what the backward sees
        *reinterpret_cast<bf16x8*>(x_new + row * H + c * 8) = px[i];
        unpack8(px[i], v);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss[acc_of<TEAM>(i)] += v[j] * v[j];
    }
  }
  const float rstd = rsqrtf(row_sum<TEAM>(ss, red, 0) / (float)H + eps);
  if (tid == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = tid + i * TEAM;
    if (c < nchunk) {
      float v[8], ww[8], o[8];
      unpack8(px[i], v);
      unpack8(wv[i], ww);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[j] * rstd * ww[j];
      *reinterpret_cast<bf16x8*>(y + row * H + c * 8) = pack8(o);
    }
  }
}

// Backward: a team has the next rows' operands on their way into shared memory (cp.async, every thread the chunks it will use itself, so
// no barrier is needed) while it works on one. Rows in flight per team, and the bytes that takes per CTA. Two are enough where three CTAs
// of several teams share an SM; a third would take 221 of its 228 KB (three / two, us: 8192 x 512: 10.6 / 9.3, 32768 x 264: 23.2 / 21.8, 2048 x 2048: 11.0 / 9.6);
// a CTA that is one team wants three (8192 x 4096: 54.4 / 58.4), rows of one chunk a thread four (8192 x 64: 4.8 / 5.4 with two).
template <int TEAM, int NC> __host__ __device__ constexpr int bwd_stages() { return NC <= 1 ? 4 : NC == 2 && TEAM == ROWS_THREADS ? 3 : 2; }
template <int TEAM, int NC> __host__ __device__ constexpr int bwd_smem() {
  const int pipe = bwd_stages<TEAM, NC>() * 3 * NC * ROWS_THREADS * 16, comb = TEAM < ROWS_THREADS ? ROWS_THREADS * NC * 32 : 0;
  return pipe > comb ? pipe : comb;
}
__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(g) : "memory");
}

template <int TEAM, int NC>
__global__ void __launch_bounds__(ROWS_THREADS, NC <= 2 ? 3 : 2)
rmsnorm_bwd_rows_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                        const float* __restrict__ rstd_in, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                        float* __restrict__ dw_acc, int T, int H) {
  constexpr int TEAMS = ROWS_THREADS / TEAM;
  __shared__ __align__(16) float red[2 * TEAMS * 8];
  constexpr int STAGES = bwd_stages<TEAM, NC>();
  extern __shared__ __align__(16) uint4 pipe[];      // [stage][x, dy, dres][chunk][thread]; after the rows the teams' sums
  pdl_enter();
  const int nchunk = H / 8, tid = threadIdx.x % TEAM, team = threadIdx.x / TEAM;
  bf16x8 wv[NC];
  float dwacc[NC][8];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = tid + i * TEAM;
    if (c < nchunk) wv[i] = *reinterpret_cast<const bf16x8*>(w + c * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
  }
  const long long step = (long long)gridDim.x * TEAMS;
  auto fetch = [&](long long row, int stage) {
    if (row < T) {
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const int c = tid + i * TEAM;
        if (c < nchunk) {
          uint4* const q = pipe + (stage * 3 * NC + i) * ROWS_THREADS + threadIdx.x;
          cp_async16(q, x + row * H + c * 8);
          cp_async16(q + NC * ROWS_THREADS, dy + row * H + c * 8);
          if (dres != nullptr) cp_async16(q + 2 * NC * ROWS_THREADS, dres + row * H + c * 8);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  long long row = (long long)blockIdx.x * TEAMS + team;
#pragma unroll
  for (int st = 0; st + 1 < STAGES; ++st) fetch(row + st * step, st);
  float rstd_next = row < T ? rstd_in[row] : 0.f;
  int stage = 0;
  for (int it = 0; row < T; row += step, ++it) {
    fetch(row + (STAGES - 1) * step, stage == 0 ? STAGES - 1 : stage - 1);
    const float rstd = rstd_next;
    if (row + step < T) rstd_next = rstd_in[row + step];
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
    // (read again for the second pass, instead of held in registers)
    const uint4* const cur = pipe + stage * 3 * NC * ROWS_THREADS + threadIdx.x;
    auto operand = [&](int which, int i) {
      uint4 v;
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                   : "r"(smem_u32(cur + (which * NC + i) * ROWS_THREADS)) : "memory");
      return *reinterpret_cast<const bf16x8*>(&v);
    };
    stage = stage + 1 == STAGES ? 0 : stage + 1;
    float dot[accs<TEAM, NC>()] = {};
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int c = tid + i * TEAM;
      if (c < nchunk) {
        float xv[8], dv[8], ww[8];
        unpack8(operand(0, i), xv);
        unpack8(operand(1, i), dv);
        unpack8(wv[i], ww);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = xv[j] * rstd;
          dot[acc_of<TEAM>(i)] += xh * dv[j] * ww[j];
          dwacc[i][j] += dv[j] * xh;
        }
      }
    }
    const float cmean = row_sum<TEAM>(dot, red, it) / (float)H;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int c = tid + i * TEAM;
      if (c < nchunk) {
        float xv[8], dv[8], ww[8], o[8];
        unpack8(operand(0, i), xv);
        unpack8(operand(1, i), dv);
        unpack8(wv[i], ww);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (dv[j] * ww[j] - xv[j] * rstd * cmean) * rstd;
        if (dres != nullptr) {
          float rr[8];
          unpack8(operand(2, i), rr);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rr[j];
        }
        *reinterpret_cast<bf16x8*>(dx + row * H + c * 8) = pack8(o);
      }
    }
  }
  auto red_add = [&](float* dst, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
  };
  if constexpr (TEAMS == 1) {
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int c = tid + i * TEAM;
      if (c < nchunk) {
        red_add(dw_acc + c * 8, make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]));
        red_add(dw_acc + c * 8 + 4, make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]));
      }
    }
  } else {
    float* const comb = reinterpret_cast<float*>(pipe);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      float4* q = reinterpret_cast<float4*>(comb + (team * TEAM * NC + tid + i * TEAM) * 8);
      q[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
      q[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
    }
    __syncthreads();
    for (int c4 = threadIdx.x; c4 < H / 4; c4 += ROWS_THREADS) {
      float4 v = *reinterpret_cast<const float4*>(comb + c4 * 4);
#pragma unroll
      for (int t = 1; t < TEAMS; ++t) {
        const float4 u = *reinterpret_cast<const float4*>(comb + t * TEAM * NC * 8 + c4 * 4);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
      }
      red_add(dw_acc + c4 * 4, v);
    }
  }
}

// Calls f(team, chunks per thread) as constants for the forward. With many rows the smallest team whose threads hold a row with at
// most four chunks each; with few rows a larger one, as long as its CTAs are at most four per SM, because then the latency of one
// row's loads and sums is all there is. Measured forward / with add (us): 1803 x 576: 32 threads 3.9 / 6.1, 64 threads 2.7 / 3.7;
// 256 x 576: 1.7 / 2.2 and with 256 threads 1.4 / 1.7; 512 x 2048: 64 threads 4.5 / 6.9, 256 threads 2.6 / 3.6; and with many rows
// 8192 x 576: 32 threads 6.7 / 9.7, 64 threads 7.9 / 10.5.
template <int TEAM, typename F>
static void with_chunks(int nchunk, F f) {
#define PT_TEAM(NC) f(std::integral_constant<int, TEAM>{}, std::integral_constant<int, NC>{})
  if (nchunk <= TEAM) PT_TEAM(1);
  else if (nchunk <= 2 * TEAM) PT_TEAM(2);
  else if (nchunk <= 3 * TEAM) PT_TEAM(3);
  else PT_TEAM(4);
#undef PT_TEAM
}
template <typename F>
static void with_forward_team(int T, int H, int num_sms, F f) {
  const int nchunk = H / 8;
  int team = nchunk <= 128 ? 32 : nchunk <= 256 ? 64 : nchunk <= 512 ? 128 : 256;
  while (team < 256 && (long long)T * (2 * team) <= 4LL * num_sms * ROWS_THREADS) team *= 2;
  if (team == 32) with_chunks<32>(nchunk, f);
  else if (team == 64) with_chunks<64>(nchunk, f);
  else if (team == 128) with_chunks<128>(nchunk, f);
  else with_chunks<256>(nchunk, f);
}

// The same for the backward, whose weight-gradient sums favour few, long-lived CTAs. A wide row takes two chunks per thread: half
// the registers make room for a third CTA per SM (4096 x 2048: 26.6 us with four chunks, 22.6 with two; 32768 x 2048: 119 and 104),
// while narrow rows are better off without barriers (8192 x 576: 16.4 us with 32 threads per row, 18.5 with 64).
template <typename F>
static void with_backward_team(int H, F f) {
  const int nchunk = H / 8;
#define PT_TEAM(TEAM, NC) f(std::integral_constant<int, TEAM>{}, std::integral_constant<int, NC>{})
  if (nchunk <= 32) PT_TEAM(32, 1);
  else if (nchunk <= 64) PT_TEAM(32, 2);
  else if (nchunk <= 96) PT_TEAM(32, 3);
  else if (nchunk <= 128) PT_TEAM(32, 4);
  else if (nchunk <= 256) PT_TEAM(128, 2);
  else if (nchunk <= 512) PT_TEAM(256, 2);
  else PT_TEAM(256, 4);
#undef PT_TEAM
}

extern "C" int pt_rmsnorm_fwd(const void* x, const void* delta, const void* w, void* x_new, void* y, float* rstd,
                              int T, int H, float eps, cudaStream_t st) {
  if (H % 8 || H > 8 * ROWS_THREADS * 4) return -10;
  if (T == 0) return 0;
  static int num_sms = 0;
  if (num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  with_forward_team(T, H, num_sms, [&](auto team, auto nc) {
    constexpr int TEAM = decltype(team)::value, NC = decltype(nc)::value, ROWS = ROWS_THREADS / TEAM;
    const dim3 grid((unsigned)((T + ROWS - 1) / ROWS));
    if (delta != nullptr)
      launch_pdl(rmsnorm_fwd_rows_kernel<true, TEAM, NC>, grid, dim3(ROWS_THREADS), 0, st, (const bf16*)x, (const bf16*)delta,
                 (const bf16*)w, (bf16*)x_new, (bf16*)y, rstd, T, H, eps);
    else
      launch_pdl(rmsnorm_fwd_rows_kernel<false, TEAM, NC>, grid, dim3(ROWS_THREADS), 0, st, (const bf16*)x, (const bf16*)delta,
                 (const bf16*)w, (bf16*)x_new, (bf16*)y, rstd, T, H, eps);
  });
  return check_launch();
}

// number of dw partial rows the backward needs in `partial` ([rows, H] fp32 scratch)
extern "C" int pt_rmsnorm_bwd_partial_rows(int T, int num_sms) {
  int g = 4 * num_sms;
  return T < g ? T : g;
}

static void launch_rmsnorm_bwd(int grid, const void* dy, const void* x, const void* w, const float* rstd,
                               const void* dres, void* dx, float* partial, int T, int H, cudaStream_t st) {
  const int mc = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
#define PT_NORM_BWD(MC)                                                                                      \
  rmsnorm_bwd_kernel<MC><<<grid, NORM_THREADS, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd, \
                                                        (const bf16*)dres, (bf16*)dx, partial, T, H)
  if (mc <= 1) PT_NORM_BWD(1); else if (mc <= 2) PT_NORM_BWD(2); else PT_NORM_BWD(4);
#undef PT_NORM_BWD
}

extern "C" int pt_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                              void* dx, float* dw, float* partial, int T, int H, int num_sms, cudaStream_t st) {
  if (H % 8 || H > 8 * NORM_THREADS * NORM_MAXC) return -10;
  if (T == 0) return 0;
  const int grid = pt_rmsnorm_bwd_partial_rows(T, num_sms);
  launch_rmsnorm_bwd(grid, dy, x, w, rstd, dres, dx, partial, T, H, st);
  reduce_partials_kernel<<<(H + 31) / 32, 256, 0, st>>>(partial, dw, grid, H);
  return check_launch(2);
}

// RMSNorm backward that ADDS dw into `dw_acc` (fp32 [H], e.g. the weight's gradient-bucket slice) with vector
// reductions instead of writing per-CTA partials and summing them in a second kernel. Summation order of dw is
// not fixed from run to run. Returns 1 (nothing launched) when the shape is not covered: H % 8 != 0, H > 8192 or a
// dw_acc that is not 16-byte aligned.
extern "C" int pt_rmsnorm_bwd_acc(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                                  void* dx, float* dw_acc, int T, int H, int num_sms, cudaStream_t st) {
  if (H % 8 || H > 8 * ROWS_THREADS * 4 || (reinterpret_cast<uintptr_t>(dw_acc) & 15)) return 1;
  if (T == 0) return 0;
  bool failed = false;
  with_backward_team(H, [&](auto team, auto nc) {
    constexpr int TEAM = decltype(team)::value, NC = decltype(nc)::value, ROWS = ROWS_THREADS / TEAM;
    const int want = (T + ROWS - 1) / ROWS, cap = (NC <= 2 ? 3 : 2) * num_sms;
    auto kern = rmsnorm_bwd_rows_kernel<TEAM, NC>;
    constexpr int SMEM = bwd_smem<TEAM, NC>();
    static PerDevice opted_in;
    const int rc = opted_in.get(current_device(), [&] {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess) return 1;
      cudaGetLastError();
      return -3;
    });
    if (rc <= 0) {
      failed = true;
      return;
    }
    launch_pdl(kern, dim3((unsigned)(want < cap ? want : cap)), dim3(ROWS_THREADS), SMEM, st,
               (const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd, (const bf16*)dres, (bf16*)dx, dw_acc, T, H);
  });
  if (failed) return -3;
  return check_launch();
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of pt_rmsnorm_bwd (contract in noalloc.h): the dw partials live in a file-scope
// device array instead of a caller-provided scratch buffer. In host code `g_noalloc_partial` is only a
// stand-in for the symbol; its device address is resolved once per device with cudaGetSymbolAddress.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_noalloc_partial[PT_NOALLOC_MAX_ROWS * PT_NOALLOC_MAX_H];
static float* g_noalloc_partial_addr[64] = {nullptr};

extern "C" int pt_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                      const void* dres, void* dx, float* dw, int T, int H, cudaStream_t st) {
  if (T <= 0 || H <= 0 || H % 8) return PT_NOALLOC_ERR_BAD_SHAPE;
  if (H > PT_NOALLOC_MAX_H) return PT_NOALLOC_ERR_TOO_LARGE;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return PT_NOALLOC_ERR_SYMBOL;
  if (g_noalloc_partial_addr[dev] == nullptr) {
    // first call on this device: look the array up while this device is current
    float* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_noalloc_partial) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return PT_NOALLOC_ERR_SYMBOL;
    }
    g_noalloc_partial_addr[dev] = p;
  }
  float* partial = g_noalloc_partial_addr[dev];
  const int grid = T < PT_NOALLOC_MAX_ROWS ? T : PT_NOALLOC_MAX_ROWS;   // one partial row per CTA
  launch_rmsnorm_bwd(grid, dy, x, w, rstd, dres, dx, partial, T, H, st);
  reduce_partials_kernel<<<(H + 31) / 32, 256, 0, st>>>(partial, dw, grid, H);
  return check_launch(2) == 0 ? PT_NOALLOC_OK : PT_NOALLOC_ERR_LAUNCH;
}

extern "C" const char* pt_noalloc_strerror(int code) {
  switch (code) {
    case PT_NOALLOC_OK: return "ok";
    case PT_NOALLOC_ERR_BAD_SHAPE: return "bad shape: T must be positive and H a positive multiple of 8";
    case PT_NOALLOC_ERR_TOO_LARGE: return "problem too large for the built-in scratch array: H exceeds PT_NOALLOC_MAX_H (4096)";
    case PT_NOALLOC_ERR_SYMBOL: return "could not resolve the device address of the built-in scratch array";
    case PT_NOALLOC_ERR_LAUNCH: return "kernel launch failed";
    default: return "unknown code";
  }
}

extern "C" int pt_rope(void* qkv, const float* cosT, const float* sinT, long long T, int n_rot, int d, int S,
                       long long row_stride, int inverse, cudaStream_t st) {
  if (d % 16 || row_stride % 8) return -10;
  const long long total = T * n_rot * (d / 16);
  if (total == 0) return 0;
  rope_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>((bf16*)qkv, cosT, sinT, total, n_rot, d, S, row_stride,
                                                              inverse ? -1.f : 1.f);
  return check_launch();
}

extern "C" int pt_swiglu_fwd(const void* gu, void* out, long long T, int I, cudaStream_t st) {
  if (I % 8) return -10;
  const long long total = T * (I / 8);
  if (total == 0) return 0;
  swiglu_fwd_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const bf16*)gu, (bf16*)out, total, I / 8);
  return check_launch();
}

extern "C" int pt_swiglu_bwd(const void* gu, const void* da, void* dgu, long long T, int I, cudaStream_t st) {
  if (I % 8) return -10;
  const long long total = T * (I / 8);
  if (total == 0) return 0;
  launch_pdl(swiglu_bwd_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, st, (const bf16*)gu, (const bf16*)da,
             (bf16*)dgu, total, I / 8);
  return check_launch();
}

extern "C" int pt_embedding_fwd(const long long* ids, const void* w, void* out, long long T, int H, long long rows,
                                long long vocab_start, cudaStream_t st) {
  if (H % 8) return -10;
  if (T == 0) return 0;
  launch_pdl(embedding_fwd_kernel, dim3((unsigned)T), dim3(256), 0, st, ids, (const bf16*)w, (bf16*)out, H / 8, rows, vocab_start);
  return check_launch();
}

extern "C" int pt_embedding_bwd(const long long* ids, const void* dy, float* dw, long long T, int H, long long rows,
                                long long vocab_start, cudaStream_t st) {
  if (H % 8) return -10;
  if (T == 0 || H == 0) return 0;
  const dim3 grid((unsigned)((T * (H / 8) + 255) / 256));
  if ((reinterpret_cast<uintptr_t>(dw) & 15) == 0)
    launch_pdl(embedding_bwd_kernel<true>, grid, dim3(256), 0, st, ids, (const bf16*)dy, dw, T, H / 8, rows, vocab_start);
  else
    launch_pdl(embedding_bwd_kernel<false>, grid, dim3(256), 0, st, ids, (const bf16*)dy, dw, T, H / 8, rows, vocab_start);
  return check_launch();
}

extern "C" int pt_accumulate(float* acc, const void* g, long long n, int g_is_f32, cudaStream_t st) {
  if (n == 0) return 0;
  if (g_is_f32)
    accumulate_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(acc, (const float*)g, n);
  else
    accumulate_kernel<<<(unsigned)((n / 8 + 1 + 255) / 256), 256, 0, st>>>(acc, (const bf16*)g, n);
  return check_launch();
}

extern "C" int pt_add(const void* a, const void* b, void* out, long long n, cudaStream_t st) {
  if (n == 0) return 0;
  launch_pdl(add_kernel, dim3((unsigned)((n / 8 + 1 + 255) / 256)), dim3(256), 0, st, (const bf16*)a, (const bf16*)b, (bf16*)out, n);
  return check_launch();
}

// AdamW over `count` tensors. params: bf16 (param_is_bf16) or fp32. grads/m/v fp32. masters[i] may be null.
extern "C" int pt_adamw_multi(void** params, const float** grads, float** ms, float** vs, float** masters,
                              const long long* numels, int count, int param_is_bf16, int step, float lr, float beta1,
                              float beta2, float eps, float wd, cudaStream_t st) {
  const float bc1 = 1.f - powf(beta1, (float)step);
  const float bc2_sqrt = sqrtf(1.f - powf(beta2, (float)step));
  AdamArgs args;
  args.count = 0;
  long long blocks = 0;
  auto flush = [&]() -> int {
    if (args.count == 0) return 0;
    args.first_block[args.count] = (unsigned)blocks;
    if (param_is_bf16)
      adamw_kernel<true><<<(unsigned)blocks, ADAM_THREADS, 0, st>>>(args, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
    else
      adamw_kernel<false><<<(unsigned)blocks, ADAM_THREADS, 0, st>>>(args, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt);
    args.count = 0;
    blocks = 0;
    return check_launch();
  };
  for (int i = 0; i < count; ++i) {
    const long long n = numels[i];
    if (n == 0) continue;
    const long long chunks = (n + ADAM_CHUNK - 1) / ADAM_CHUNK;
    if (args.count == ADAM_MAX_TENSORS || (args.count > 0 && blocks + chunks > 0x7fffffffLL))
      if (int rc = flush()) return rc;
    const uintptr_t f32s = (uintptr_t)grads[i] | (uintptr_t)ms[i] | (uintptr_t)vs[i] | (uintptr_t)masters[i];
    const int k = args.count++;
    args.t[k] = AdamTensor{params[i], grads[i], ms[i], vs[i], masters[i], n};
    args.vec[k] = (f32s & 15) == 0 && ((uintptr_t)params[i] & (param_is_bf16 ? 7 : 15)) == 0;
    args.first_block[k] = (unsigned)blocks;
    blocks += chunks;
  }
  return flush();
}

extern "C" int pt_scale(float* x, const float* coef, long long n, cudaStream_t st) {
  if (n == 0) return 0;
  scale_kernel<<<(unsigned)((n + SCALE_CHUNK - 1) / SCALE_CHUNK), 256, 0, st>>>(x, coef, n);
  return check_launch();
}

extern "C" int pt_merge_attention(float* out, float* lse, const void* bo, const float* bl, int B, int S, int h, int d,
                                  cudaStream_t st) {
  const long long warps = (long long)B * S * h;
  if (warps == 0) return 0;
  merge_attention_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(out, lse, (const bf16*)bo, bl, B, S, h, d);
  return check_launch();
}
