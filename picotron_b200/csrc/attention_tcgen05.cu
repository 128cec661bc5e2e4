// Flash attention forward and backward for sm_100a: tcgen05 MMAs with TMEM accumulators, TMA-fed tiles,
// native GQA, head_dim 64 or 128, causal or full, arbitrary sequence lengths (tails are masked).
//
// Replaces flash_attn_func (FlashAttention-2, mma.sync) at picotron/model.py:33-37,154 and the materialised
// block attention of ring attention (picotron/context_parallel/context_parallel.py:112-155): the same kernels
// compute one ring block when they are given the global log-sum-exp / delta.
//
// Tensors: q [B,Sq,hq,d], k/v [B,Sk,hkv,d] with packed (head, d) and an arbitrary token stride, so slices of
// the packed qkv activation are read in place through 4-D tensor maps {d, head, token, batch}.
// "causal" masks kv index > q index, both counted from the start of their tensors.
//
// Forward, one CTA per (128 query rows, head, batch); two CTAs share an SM so that one CTA's MMAs overlap the
// other's softmax:
//   warp 4    TMA producer: Q once, then K and V blocks through 2-stage rings
//   warp 5    MMA issuer:  S = Q K^T  (TMEM, BN fp32 columns), later  O_j = P_j V_j  (TMEM, d columns)
//   warps 0-3 softmax: thread t owns query row t = TMEM lane t. Online softmax in the exp2 domain, P_j written
//             as bf16 back into tensor memory as the A operand of the second MMA, which accumulates the output there.
//             Tensor memory spares the swizzled stores, a proxy fence and the wait before them: 1 x 32768, 32 / 8 heads,
//             d = 64: 7.67 -> 6.03 ms; 4 x 1024, 32 heads, d = 64: 66 -> 60 us, d = 128: 75 -> 68 us. Bound by the latency
//             of a block's chain and by the 1,024 cycles that 128 x 128 ex2 take per SM (two blocks: ~3,300 cycles).
//
// Backward, one CTA per (128-key block, kv head, batch) looping over the query heads of the group and the query blocks that see
// this key block, pipelined over the steps (attn_bwd_kernel):
//   S^T = K Q^T and dP^T = V dO^T into TMEM; threads (one key each) form P^T = exp2(S^T*c - lse), stored as bf16 into TMEM, and
//   dS^T = P^T*(dP^T - delta)*scale, stored as bf16 into swizzled shared memory; then dV += P^T dO, dK += dS^T Q (TMEM
//   accumulators that live for the whole CTA) and dQ = dS K, which four warps add to an fp32 workspace with TMA reduce-adds. Eight
//   (d = 128) or sixteen (d = 64) warps compute.
//   A small kernel computes delta = rowsum(dO*O) beforehand and another converts the fp32 dQ to bf16.
#include "common.cuh"
#include "tensormap.cuh"

#include <algorithm>
#include <type_traits>

extern "C" void pt_count_launches(int n);
extern "C" void* pt_status_word();

namespace pt {
namespace attn {

typedef __nv_bfloat16 bf16;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;
constexpr unsigned KID_FWD = 3, KID_BWD = 4;

inline KernelStatus* status_word_attn() { return reinterpret_cast<KernelStatus*>(pt_status_word()); }

static unsigned long long* g_attn_prof = nullptr;   // device buffer of 16 counters while phase profiling is on

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// byte offset of the 16-byte unit holding columns [8u, 8u+8) of row r inside one [rows][64] bf16 chunk
// stored with the 128-byte swizzle (what TMA writes and UMMA descriptors of layout type SWIZZLE_128B read)
__device__ __forceinline__ uint32_t sw128_offset(int r, int u) { return (uint32_t)(r * 128 + ((u ^ (r & 7)) << 4)); }

// ---------------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------------
template <int D, int BN>
struct FwdCfg {
  static constexpr int BM = 128;
  static constexpr int DCH = D / 64;
  static constexpr int Q_BYTES = BM * D * 2;
  static constexpr int KV_BYTES = BN * D * 2;
  static constexpr int STAGES = 2;
  static constexpr int TILES = Q_BYTES + 2 * STAGES * KV_BYTES;
  static constexpr int SMEM = TILES + 256;            // + barriers; the block starts 1024-byte aligned
  static constexpr int TMEM_COLS = 256;
  static constexpr int S_COL = 0, O_COL = BN, P_COL = BN + D;
  static_assert(BN + D + BN / 2 <= TMEM_COLS, "TMEM budget");
};

struct FwdBars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_free, p_ready, o_full;
  uint32_t tmem_base;
  int abort_flag;
};

// K/V may come in up to 8 segments of Sk keys each (the sequence chunks of the context-parallel ranks; a segment's
// tensor map may point into a peer GPU's memory). Keys of segment i precede keys of segment i+1; `causal` applies the
// diagonal mask inside the LAST segment only, every earlier segment is fully visible.
constexpr int MAX_SEGS = 8;
struct KVSegs {
  CUtensorMap k[MAX_SEGS];
  CUtensorMap v[MAX_SEGS];
};

struct AttnParams {
  int B, Sq, Sk, hq, hkv;
  int causal;
  float scale;
  int n_segs;
  unsigned long long* prof;   // optional phase counters (see pt_attention_set_profile); nullptr = not measured
};

// Phase counters of the kernels' consumer threads, in SM clock cycles, summed over all CTAs (one thread of each CTA measures):
//   [0] bwd: waiting for S and dP    [1] bwd: TMEM read, exponentials, P/dS stores    [2] bwd, drain warps: waiting for dQ
//   [3] bwd, drain warps: dQ drain   [4] bwd: steps          [5] bwd: lifetime of the compute loop    [6] bwd: CTAs
//   [8] fwd: S read + row maximum    [9] fwd: wait for O / rescale, P store   [10] fwd: exponentials   [11] fwd: blocks
//   [12] fwd: lifetime of the softmax loop   [13] fwd: CTAs   [14] fwd: waiting for S
// Measured only by the PROF instantiations of the kernels, which are launched while a counter buffer is set; the regular
// instantiations contain none of this code.
__device__ __forceinline__ long long prof_clock(bool on) { return on ? clock64() : 0; }

template <int D, int BN, bool PROF>
__global__ void __launch_bounds__(192, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ KVSegs segs, const __grid_constant__ CUtensorMap tm_o,
                float* __restrict__ LSE, AttnParams p, KernelStatus* status) {
  using Cfg = FwdCfg<D, BN>;
  pdl_launch_dependents();
  // no static shared memory in this kernel: the dynamic block starts at the (1024-byte aligned) window base
  extern __shared__ __align__(1024) uint8_t smem[];
  FwdBars& bars = *reinterpret_cast<FwdBars*>(smem + Cfg::TILES);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + Cfg::Q_BYTES;
  uint8_t* sV = sK + Cfg::STAGES * Cfg::KV_BYTES;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_qb = (p.Sq + Cfg::BM - 1) / Cfg::BM;
  // Work order. Causal: the heaviest query blocks of ALL heads first (longest job first), so that the last CTAs to start are
  // the lightest; head by head, the last head's heavy blocks ran alone at the end. Measured forward / backward (us): 8192 x 32
  // heads, d = 128: 620 -> 527 / 2578 -> 2164; 8 x 1024 x 9 heads, d = 64: 54 -> 44 / 130 -> 104. Full attention has equal
  // blocks and stays head by head, for the L2.
  const unsigned bh_count = (unsigned)(p.hq * p.B);
  const unsigned qi = p.causal ? blockIdx.x / bh_count : blockIdx.x % (unsigned)num_qb;
  const unsigned bh = p.causal ? blockIdx.x % bh_count : blockIdx.x / (unsigned)num_qb;
  const int qb = num_qb - 1 - (int)qi;
  const int head = (int)(bh % (unsigned)p.hq);
  const int b = (int)(bh / (unsigned)p.hq);
  const int kv_head = head / (p.hq / p.hkv);
  const int q0 = qb * Cfg::BM;
  const int bps = (p.Sk + BN - 1) / BN;                              // key blocks per segment
  const int last_end = p.causal ? min(p.Sk, q0 + Cfg::BM) : p.Sk;    // keys of the last segment this tile can see
  const int nblk = (p.n_segs - 1) * bps + (last_end + BN - 1) / BN;

  auto load_kv = [&](int st, uint8_t* ring, const CUtensorMap& map, uint64_t* bar, int kv0) {
    mbar_expect_tx(bar, Cfg::KV_BYTES);
#pragma unroll
    for (int c = 0; c < Cfg::DCH; ++c) tma_load_4d(ring + st * Cfg::KV_BYTES + c * (BN * 128), &map, bar, c * 64, kv_head, kv0, b);
  };

  if (warp == 4 && elect_one()) {
    mbar_init(&bars.q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars.k_full[s], 1);
      mbar_init(&bars.k_empty[s], 1);
      mbar_init(&bars.v_full[s], 1);
      mbar_init(&bars.v_empty[s], 1);
    }
    mbar_init(&bars.s_full, 1);
    mbar_init(&bars.s_free, 4);          // one arrival per softmax warp
    mbar_init(&bars.p_ready, 4);
    mbar_init(&bars.o_full, 1);
    bars.abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&segs.k[0]);
    tma_prefetch_desc(&segs.v[0]);
    tma_prefetch_desc(&tm_o);
    // The first loads leave before the other warps are let go: they travel under the tensor-memory allocation and the first barrier.
    pdl_wait();
    mbar_expect_tx(&bars.q_full, Cfg::Q_BYTES);
#pragma unroll
    for (int c = 0; c < Cfg::DCH; ++c) tma_load_4d(sQ + c * (Cfg::BM * 128), &tm_q, &bars.q_full, c * 64, head, q0, b);
    if (nblk > 0) {
      load_kv(0, sK, segs.k[0], &bars.k_full[0], 0);
      load_kv(0, sV, segs.v[0], &bars.v_full[0], 0);
    }
  }
  if (warp == 5) {
    tmem_alloc(&bars.tmem_base, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();                      // barrier init and tensor-memory allocation overlapped the predecessor's tail
  const uint32_t tmem_base = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;

  if (warp == 4) {
    // ------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int seg = 0, kv0 = 0;                          // (the first block's: above)
      for (int j = 1; j < nblk; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if ((kv0 += BN) >= p.Sk) {
          kv0 = 0;
          ++seg;
        }
        if (!mbar_wait(&bars.k_empty[st], ph ^ 1, abort_flag)) { report_error(status, KID_FWD, 1); break; }
        load_kv(st, sK, segs.k[seg], &bars.k_full[st], kv0);
        if (!mbar_wait(&bars.v_empty[st], ph ^ 1, abort_flag)) { report_error(status, KID_FWD, 2); break; }
        load_kv(st, sV, segs.v[seg], &bars.v_full[st], kv0);
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(Cfg::BM, BN, false, false);
      constexpr uint32_t idesc_o = make_idesc_bf16(Cfg::BM, D, false, true);
      bool ok = mbar_wait(&bars.q_full, 0, abort_flag);
      if (!ok) report_error(status, KID_FWD, 3);
      const uint64_t q_km = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
      // S_{j+1} = Q K_{j+1}^T is issued as soon as the softmax threads have copied S_j out of tensor memory (s_free),
      // i.e. before P_j exists, so it runs under the exponentials of block j instead of after them.
      auto issue_s = [&](int j) -> bool {
        const int st = j & 1;
        if (!mbar_wait(&bars.k_full[st], (j >> 1) & 1, abort_flag)) { report_error(status, KID_FWD, 4); return false; }
        tcgen05_fence_after();
        const uint64_t k_km = make_smem_desc_sw128(smem_u32(sK + st * Cfg::KV_BYTES), 16, 1024);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_bf16(tmem_base + Cfg::S_COL, smem_desc_advance(q_km, (kk >> 2) * (Cfg::BM * 128) + (kk & 3) * 32),
                    smem_desc_advance(k_km, (kk >> 2) * (BN * 128) + (kk & 3) * 32), idesc_s, kk > 0 ? 1u : 0u);
        umma_commit(&bars.s_full);
        umma_commit(&bars.k_empty[st]);
        return true;
      };
      if (ok && nblk > 0) ok = issue_s(0);
      for (int j = 0; j < nblk && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (j + 1 < nblk) {
          if (!mbar_wait(&bars.s_free, j & 1, abort_flag)) { report_error(status, KID_FWD, 10); break; }
          if (!issue_s(j + 1)) break;
        }
        if (!mbar_wait(&bars.p_ready, j & 1, abort_flag)) { report_error(status, KID_FWD, 5); break; }
        if (!mbar_wait(&bars.v_full[st], ph, abort_flag)) { report_error(status, KID_FWD, 6); break; }
        tcgen05_fence_after();
        const uint64_t v_mn = make_smem_desc_sw128(smem_u32(sV + st * Cfg::KV_BYTES), BN * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
          umma_bf16_ts(tmem_base + Cfg::O_COL, tmem_base + Cfg::P_COL + kk * 8, smem_desc_advance(v_mn, kk * 2048), idesc_o,
                       (j > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&bars.o_full);
        umma_commit(&bars.v_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------------------------------------ softmax (warps 0..3)
    // The running output stays in TMEM (the PV MMAs accumulate onto it). Probabilities are taken relative to a
    // reference maximum m_ref that is only moved -- and O rescaled in TMEM -- when the true row maximum has
    // grown by more than 2^8 since the last move, so exp2 never exceeds 256 and the per-block TMEM round trips
    // shrink to one batched read of S.
    const int t = threadIdx.x;                       // query row inside the tile == TMEM lane
    const int row = q0 + t;
    const uint32_t t_lane = tmem_base + (uint32_t(warp * 32) << 16);
    const float sl2 = p.scale * LOG2E;
    constexpr float kRescaleThreshold = 8.f;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    const bool prof_on = PROF && p.prof != nullptr && threadIdx.x == 0;
    long long pacc[4] = {0, 0, 0, 0};
    const long long pstart = prof_clock(prof_on);
    int seg = 0, col0 = 0;                           // the block's segment and first key in it
    for (int j = 0; j < nblk; ++j) {
      const long long pt0 = prof_clock(prof_on);
      if (!mbar_wait(&bars.s_full, j & 1, abort_flag)) { if (lane == 0) report_error(status, KID_FWD, 7); ok = false; break; }
      tcgen05_fence_after();
      const long long pt1 = prof_clock(prof_on);
      uint32_t s[BN];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32b_x32_at(t_lane + Cfg::S_COL + c * 32, s, c * 32);
      tmem_ld_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.s_free);                   // S_j is in registers: the next S may overwrite it
      const bool diag = p.causal && seg == p.n_segs - 1;
      const bool need_mask = (diag && col0 + BN - 1 > q0) || (col0 + BN > p.Sk);
      // four independent running maxima / sums: a single one is a 128-deep chain of dependent instructions
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
        const int vis = min(p.Sk - col0, diag ? row - col0 + 1 : BN);         // the first `vis` columns are visible
#pragma unroll
        for (int e = 0; e < BN; ++e) {
          s[e] = e < vis ? s[e] : __float_as_uint(-INFINITY);
          mx4[e & 3] = fmaxf(mx4[e & 3], __uint_as_float(s[e]));
        }
      } else {
#pragma unroll
        for (int e = 0; e < BN; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], __uint_as_float(s[e]));
      }
      if ((col0 += BN) >= p.Sk) {                                 // (the next block's)
        col0 = 0;
        ++seg;
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float m_blk = mx * sl2;
      const long long pt2 = prof_clock(prof_on);
      // move the reference? (first finite maximum, or growth beyond the threshold)
      const bool move = m_blk > m_ref + kRescaleThreshold || (m_ref == -INFINITY && m_blk > -INFINITY);
      float alpha = 1.f;
      if (move) {
        alpha = fast_exp2(m_ref - m_blk);            // m_ref == -inf -> 0
        m_ref = m_blk;
        l *= alpha;
      }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
      // Sum of a row: its neighbour pairs in four running sums (two packed registers), every fourth pair each. The order is part of
      // the result: a last bit of it moves every later bf16 rounding of a deep model. (Packed sums of even and odd elements were
      // one instruction less per four elements: 5,830 instead of 5,970 us at 32768, d = 64; 500 instead of 507 at 8192, d = 128.)
      uint64_t lsum[2] = {0, 0};
      uint32_t pk[BN / 2];                                        // P_j of this row, bf16 pairs
      const uint64_t sl2_2 = pair_of(sl2, sl2), neg_m = pair_of(-m_use, -m_use);
#pragma unroll
      for (int e = 0; e < BN; e += 4) {
        const uint64_t x0 = fma2(pair_of(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sl2_2, neg_m);
        const uint64_t x1 = fma2(pair_of(__uint_as_float(s[e + 2]), __uint_as_float(s[e + 3])), sl2_2, neg_m);
        const float p0 = fast_exp2(lo_of(x0)), p1 = fast_exp2(hi_of(x0));      // masked: exp2(-inf) = 0
        const float p2 = fast_exp2(lo_of(x1)), p3 = fast_exp2(hi_of(x1));
        lsum[(e >> 2) & 1] = add2(lsum[(e >> 2) & 1], pair_of(p0 + p1, p2 + p3));
        pk[e >> 1] = pack_bf16(p0, p1);
        pk[(e >> 1) + 1] = pack_bf16(p2, p3);
      }
      l += (lo_of(lsum[0]) + hi_of(lsum[0])) + (lo_of(lsum[1]) + hi_of(lsum[1]));
      const long long pt3 = prof_clock(prof_on);
      if (j > 0) {
        // P_{j-1} and O (tensor memory) may be touched once the MMA O += P_{j-1} V_{j-1} has completed
        if (!mbar_wait(&bars.o_full, (j - 1) & 1, abort_flag)) { if (lane == 0) report_error(status, KID_FWD, 8); ok = false; break; }
        tcgen05_fence_after();                                    // (also for the store of P_j below)
        if (__any_sync(0xffffffffu, move)) {
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_lane + Cfg::O_COL + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
            tmem_st_32x32b_x32(t_lane + Cfg::O_COL + c * 32, r);
          }
          tmem_st_wait();
        }
      }
#pragma unroll
      for (int c = 0; c < BN / 64; ++c) tmem_st_32x32b_x32_at(t_lane + Cfg::P_COL + c * 32, pk, c * 32);
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.p_ready);
      if (prof_on) {
        const long long pt4 = clock64();
        pacc[0] += pt2 - pt1; pacc[1] += pt4 - pt3; pacc[2] += pt3 - pt2; pacc[3] += pt1 - pt0;
      }
    }
    if (prof_on) {
      atomicAdd(&p.prof[8], (unsigned long long)pacc[0]);
      atomicAdd(&p.prof[9], (unsigned long long)pacc[1]);
      atomicAdd(&p.prof[10], (unsigned long long)pacc[2]);
      atomicAdd(&p.prof[14], (unsigned long long)pacc[3]);
      atomicAdd(&p.prof[11], (unsigned long long)nblk);
      atomicAdd(&p.prof[12], (unsigned long long)(clock64() - pstart));
      atomicAdd(&p.prof[13], 1ull);
    }
    if (ok && mbar_wait(&bars.o_full, (nblk - 1) & 1, abort_flag)) {
      tcgen05_fence_after();
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      // O goes to TMA through the place of Q, which the last S was the last to read: 32 rows of 64 columns (128 bytes, swizzled) a piece.
      // (Stored by every thread for itself, they were 16-byte pieces of 32 rows an instruction.)
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint8_t* const stg = sQ + (warp * (D / 64) + c) * 4096;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_lane + Cfg::O_COL + c * 64 + h * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < 4; ++u)
            *reinterpret_cast<uint4*>(stg + sw128_offset(lane, h * 4 + u)) =
                make_uint4(pack_bf16(__uint_as_float(r[8 * u]) * inv_l, __uint_as_float(r[8 * u + 1]) * inv_l),
                           pack_bf16(__uint_as_float(r[8 * u + 2]) * inv_l, __uint_as_float(r[8 * u + 3]) * inv_l),
                           pack_bf16(__uint_as_float(r[8 * u + 4]) * inv_l, __uint_as_float(r[8 * u + 5]) * inv_l),
                           pack_bf16(__uint_as_float(r[8 * u + 6]) * inv_l, __uint_as_float(r[8 * u + 7]) * inv_l));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (elect_one()) {
          if (q0 + warp * 32 < p.Sq) tma_store_4d(&tm_o, stg, c * 64, head, q0 + warp * 32, b);
          tma_store_commit();
        }
      }
      if (row < p.Sq)
        LSE[((long long)b * p.hq + head) * p.Sq + row] = (l > 0.f) ? (m_ref * LN2 + __logf(l)) : -INFINITY;
      if (elect_one()) tma_store_wait<0>();
    } else if (ok && lane == 0) {
      report_error(status, KID_FWD, 9);
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 5) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------
// backward helpers: delta = rowsum(dO * O) and fp32 -> bf16 conversion of dQ
// ---------------------------------------------------------------------------------------------------------
// D / 8 threads per (b, s, head) row, 16 bytes of dO and of O per thread, reduced with shuffles inside the group. The fp32
// workspace that dQ is accumulated in is cleared on the way (a fill of its own was one more launch and as many bytes).
template <int D>
__global__ void __launch_bounds__(256)
delta_kernel(const bf16* __restrict__ dO, const bf16* __restrict__ O, float* __restrict__ delta, float* __restrict__ dq_ws, int B,
             int S, int h) {
  constexpr int TPR = D / 8;
  pdl_enter();
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)B * S * h;
  const long long rid = tid / TPR;
  const int part = (int)(tid % TPR);
  const long long r = rid < total ? rid : total - 1;            // clamp: every lane takes part in the shuffles
  const uint4 a = *reinterpret_cast<const uint4*>(dO + r * D + part * 8);
  const uint4 o = *reinterpret_cast<const uint4*>(O + r * D + part * 8);
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, ow[4] = {o.x, o.y, o.z, o.w};
  if (rid < total) {
    float4* z = reinterpret_cast<float4*>(dq_ws + r * D + part * 8);
    z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i]));
    const float2 fo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ow[i]));
    acc += fa.x * fo.x + fa.y * fo.y;
  }
#pragma unroll
  for (int off = TPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (part == 0 && rid < total) {
    const int head = (int)(rid % h);
    const long long bs = rid / h;
    const int s = (int)(bs % S), b = (int)(bs / S);
    delta[((long long)b * h + head) * S + s] = acc;
  }
}

// dq_ws: fp32 [B*Sq, hq*d] contiguous -> dq bf16 with token stride dq_row
__global__ void convert_dq_kernel(const float* __restrict__ ws, bf16* __restrict__ dq, long long tokens, int width,
                                  long long dq_row) {
  pdl_enter();
  const long long i4 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 >= tokens * width) return;
  const long long tok = i4 / width;
  const int col = (int)(i4 % width);
  const float4 v = *reinterpret_cast<const float4*>(ws + i4);
  uint2 o;
  o.x = pack_bf16(v.x, v.y);
  o.y = pack_bf16(v.z, v.w);
  *reinterpret_cast<uint2*>(dq + tok * dq_row + col) = o;
}

// Same conversion with the inverse RoPE of dq folded in (the backward of rotating q): a thread converts 4 columns of the
// first half of a head and their partners in the second half; token t is at position t % seq.
__global__ void convert_dq_rope_kernel(const float* __restrict__ ws, bf16* __restrict__ dq, long long tokens, int heads, int d,
                                       long long dq_row, const float* __restrict__ cosT, const float* __restrict__ sinT,
                                       int seq) {
  pdl_enter();
  const int half = d / 2, per_head = half / 4;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= tokens * heads * per_head) return;
  const int j = (int)(idx % per_head) * 4;
  const long long th = idx / per_head;
  const int head = (int)(th % heads);
  const long long tok = th / heads;
  const int pos = (int)(tok % seq);
  const float* src = ws + (tok * heads + head) * d + j;
  const float4 a = *reinterpret_cast<const float4*>(src);
  const float4 b = *reinterpret_cast<const float4*>(src + half);
  const float4 c = *reinterpret_cast<const float4*>(cosT + (long long)pos * half + j);
  const float4 sn = *reinterpret_cast<const float4*>(sinT + (long long)pos * half + j);
  uint2 o1, o2;
  o1.x = pack_bf16(a.x * c.x + b.x * sn.x, a.y * c.y + b.y * sn.y);
  o1.y = pack_bf16(a.z * c.z + b.z * sn.z, a.w * c.w + b.w * sn.w);
  o2.x = pack_bf16(b.x * c.x - a.x * sn.x, b.y * c.y - a.y * sn.y);
  o2.y = pack_bf16(b.z * c.z - a.z * sn.z, b.w * c.w - a.w * sn.w);
  bf16* dst = dq + tok * dq_row + (long long)head * d + j;
  *reinterpret_cast<uint2*>(dst) = o1;
  *reinterpret_cast<uint2*>(dst + half) = o2;
}

// ---------------------------------------------------------------------------------------------------------
// backward main kernel
// ---------------------------------------------------------------------------------------------------------
template <int D>
struct BwdCfg {
  static constexpr int BM = 128;   // query rows per inner step
  static constexpr int BN = 128;   // keys per CTA
  static constexpr int DCH = D / 64;
  static constexpr int TILE_BYTES = 128 * D * 2;         // Q, dO, K, V tiles
  static constexpr int DS_BYTES = BM * BN * 2;           // dS^T tile (P^T never leaves tensor memory)
  static constexpr int QSTAGES = (D == 64) ? 3 : 2;      // S of step i+1 is computed while dK of step i still reads Q_i
  static constexpr int OSTAGES = (D == 64) ? 3 : 1;      // dO ring; d = 128: dO_i is free after dV_i, half a step before its next use
  // The dQ tile of a step is staged in shared memory, 32 rows x 32 fp32 columns at a time (two buffers per drain warp), and
  // added to the fp32 workspace by TMA reduces (per-thread vector atomics saturate L2).
  static constexpr int DQ_BYTES = 4 * 2 * 32 * 32 * 4;
  static constexpr int STAT_BYTES = 2 * 2 * BM * 4;      // two stages of (lse, delta) of 128 query rows
  static constexpr int TILES = 2 * TILE_BYTES + (QSTAGES + OSTAGES) * TILE_BYTES + DS_BYTES + DQ_BYTES + STAT_BYTES;
  static constexpr int SMEM = TILES + 256;               // + barriers; the block starts 1024-byte aligned
  static constexpr int TMEM_COLS = 512;
  // d = 64: everything has columns of its own. d = 128: P^T reuses the columns S^T was read from (each part of a row its own
  // part of them) and dQ those of dP^T, so S and dP of the next step wait for dV and for the dQ drain.
  static constexpr bool SHARE = (D == 128);
  static constexpr int S_COL = 0, DP_COL = 128, DV_COL = 256, DK_COL = 256 + D;
  static constexpr int DQ_COL = SHARE ? DP_COL : 256 + 2 * D;
  static constexpr int P_COL = SHARE ? S_COL : 256 + 3 * D;
  // (the parts' P^T lie 128 / PARTS columns apart with SHARE, half of that without)
  static_assert(DQ_COL + D <= 512 && DK_COL + D <= 512 && P_COL + (SHARE ? 128 : 64) <= 512, "TMEM budget");
  static_assert(SMEM <= 232448, "shared memory budget");
};

struct BwdBars {
  uint64_t kv_full, q_full[3], q_empty[3], do_full[3], do_empty[3], st_full[2], st_empty[2];
  uint64_t s_full, s_read, p_ready, p_free, dp_full, dp_read, ds_ready, ds_free, dq_full, dq_read, acc_full;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(BwdBars) <= 256, "barrier block");

struct BwdParams {
  int B, Sq, Sk, hq, hkv;
  int causal;
  float scale;
  long long dk_row, dv_row;      // token strides (elements) of dk / dv
  int n_segs;
  long long seg_stride;          // elements between the dk (dv) outputs of consecutive segments
  // optional inverse RoPE of the dK output (the backward of rotating k): fp32 [rope_seq, d/2] tables, key i is at
  // position i % rope_seq. Only with one segment and bf16 outputs; nullptr = dK is written as computed.
  const float* cosT;
  const float* sinT;
  int rope_seq;
  int tma_out;                   // dk and dv are stored through their tensor maps (bf16, one segment)
  int parts;                     // CTAs (of one cluster) that share a key block's query heads, see bwd_head_parts
  unsigned long long* prof;      // optional phase counters, as AttnParams::prof
};

// A step's 128 query columns are dealt to PARTS warps per TMEM lane quarter (32 keys), W columns each: warps 0 .. 4 PARTS - 1 compute, then
// four drain dQ, then TMA producer, MMA issuer, row statistics and an idle warp. Registers per thread are even at launch and then
// redistributed between the warpgroups (PARTS x compute + drain + the rest).
// Four parts for d = 64, two for d = 128. Cycles per step with two / four: d = 64, 1 x 32768, 32 / 8 heads 3,127 / 2,791, 4 x 1024, 32 heads
// 3,620 / 3,370; us: 13,260 / 13,050 (the clock falls as the power cap is reached) and 119 / 114.5; d = 128: 1 x 8192, 32 / 8 heads 1,299 /
// 1,420 us, 4 x 1024, 32 heads 200 / 207. With d = 64 the compute warps' latencies are the step, and twice as many of them hide more;
// with d = 128 the MMAs are half of it, and the smaller batches of tensor-memory reads and the barriers that every MMA waits for
// count more.
constexpr int BWD_REGS = 128, BWD_REGS_COMPUTE = 160, BWD_REGS_DRAIN = 96, BWD_REGS_REST = 96;
constexpr int BWD4_REGS = 80, BWD4_REGS_COMPUTE = 88, BWD4_REGS_DRAIN = 72, BWD4_REGS_REST = 56;
template <int PARTS>
struct BwdWarps {
  static constexpr int W = 128 / PARTS, COMPUTE = 4 * PARTS, THREADS = 32 * (COMPUTE + 8);
  static constexpr int REGS = PARTS == 4 ? BWD4_REGS : BWD_REGS, REGS_COMPUTE = PARTS == 4 ? BWD4_REGS_COMPUTE : BWD_REGS_COMPUTE;
  static constexpr int REGS_DRAIN = PARTS == 4 ? BWD4_REGS_DRAIN : BWD_REGS_DRAIN, REGS_REST = PARTS == 4 ? BWD4_REGS_REST : BWD_REGS_REST;
  static_assert(PARTS * REGS_COMPUTE + REGS_DRAIN + REGS_REST <= (PARTS + 2) * REGS, "setmaxnreg must not ask for more than the launch gave");
  static_assert(THREADS * REGS <= 65536, "register file");
};
// What a CTA works on: a key block of a key/value head, with the query heads of its group and the query blocks that see it.
struct BwdWork {
  int seg, k0, kv_head, b, part, head0, qb_first, steps_per_head, steps;       // part: of the key block's CTAs; head0: its first query head
  bool diag;
};
template <bool SPLIT>
__device__ __forceinline__ BwdWork bwd_work(const BwdParams& p, int BM, int BN, unsigned block) {
  const unsigned parts = SPLIT ? p.parts : 1, cta = block / parts;
  const unsigned bps = (unsigned)(p.Sk + BN - 1) / BN;    // key blocks per segment
  const unsigned num_kb = bps * p.n_segs, heads = (unsigned)(p.hkv * p.B);
  // causal: the first (heaviest) key blocks of all heads first, full attention: head by head (see the forward)
  const unsigned kbg = p.causal ? cta / heads : cta % num_kb, bh = p.causal ? cta % heads : cta / num_kb;
  BwdWork w;
  w.seg = (int)(kbg / bps);
  w.k0 = (int)(kbg - w.seg * bps) * BN;
  w.diag = p.causal && w.seg == p.n_segs - 1;             // the causal diagonal runs through the last segment only
  w.kv_head = (int)(bh % (unsigned)p.hkv);
  w.b = (int)(bh / (unsigned)p.hkv);
  w.qb_first = w.diag ? w.k0 / BM : 0;                    // first query block that sees key k0
  w.steps_per_head = (p.Sq + BM - 1) / BM - w.qb_first;
  const int heads_here = p.hq / p.hkv / (int)parts;
  w.part = (int)(block % parts);
  w.head0 = (w.kv_head * (int)parts + w.part) * heads_here;
  w.steps = w.steps_per_head > 0 ? w.steps_per_head * heads_here : 0;
  return w;
}
template <int D> constexpr int bwd_parts() { return D == 64 ? 4 : 2; }
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Bytes of one CTA's dV and dK sums (fp32) on their way to the first CTA of the cluster: [dV, dK][4 columns][128 keys][4].
template <int D> constexpr int BWD_SUM_BYTES = 2 * 128 * D * 4;
// A compute thread's share of them to `to` (shared::cluster address).
template <int D, int PARTS>
__device__ __forceinline__ void bwd_send_sums(uint32_t tmem_base, uint32_t to) {
  using Cfg = BwdCfg<D>;
  constexpr int SUBS = PARTS / 2;
  unsigned thread;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(thread));
  const int part = thread >> 7, which = part / SUBS, sub = part % SUBS;
  const uint32_t from = tmem_base + (((thread >> 5) & 3) * 32 << 16) + (which == 0 ? Cfg::DV_COL : Cfg::DK_COL);
#pragma unroll 1
  for (int c = sub; c < D / 32; c += SUBS) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(from + c * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int u = 0; u < 8; ++u)
      asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + ((which * (D / 4) + c * 8 + u) * 128 + (thread & 127)) * 16),
                   "r"(r[4 * u]), "r"(r[4 * u + 1]), "r"(r[4 * u + 2]), "r"(r[4 * u + 3])
                   : "memory");
  }
}

// What bounds it: a step (128 keys x 128 queries) is a chain S -> exp -> dP -> dS -> dQ -> drain of hand-offs between the
// tensor core and the compute warps, each of a few hundred cycles; run one after the other they cost 5,400 (d = 64) and
// 7,900 (d = 128) cycles per step against ~1,300 / 2,600 of MMA and ~1,100 of special-function work. So the chain is pipelined
// over steps: S_{i+1} and dP_{i+1} run under the arithmetic of step i, dQ_i / dK_i under the exponentials of step i+1, and
// dQ_i is drained by warps of their own. The scores are computed TRANSPOSED (lane = key): then P^T is written straight back to
// tensor memory as the A operand of dV += P^T dO, and only dS^T goes through shared memory (which the MMAs read all the time).
// Measured (us; 1 x 32768, 32 / 8 heads, d = 64; 1 x 8192, 32 / 8 heads, d = 128): 21,500 -> 16,200 and 2,160 -> 1,410.
template <int D, bool OUT_F32, bool PROF, bool SPLIT, int PARTS>
__device__ __forceinline__ void attn_bwd_body(const CUtensorMap& tm_q, const KVSegs& segs, const CUtensorMap& tm_do, const CUtensorMap& tm_dq,
                                              const CUtensorMap& tm_dk, const CUtensorMap& tm_dv,
                                              const float* __restrict__ LSE, const float* __restrict__ DELTA, void* __restrict__ dK_,
                                              void* __restrict__ dV_, const BwdParams& p, KernelStatus* status) {
  using Cfg = BwdCfg<D>;
  using Warps = BwdWarps<PARTS>;
  constexpr int W = Warps::W, CW = Warps::COMPUTE;
  constexpr int P_PART = Cfg::SHARE ? W : W / 2;          // tensor-memory columns between the parts' P^T
  pdl_launch_dependents();
  // no static shared memory in this kernel: the dynamic block starts at the (1024-byte aligned) window base
  extern __shared__ __align__(1024) uint8_t smem[];
  BwdBars& bars = *reinterpret_cast<BwdBars*>(smem + Cfg::TILES);
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::TILE_BYTES;
  uint8_t* sQ = sV + Cfg::TILE_BYTES;
  uint8_t* sdO = sQ + Cfg::QSTAGES * Cfg::TILE_BYTES;
  uint8_t* sdS = sdO + Cfg::OSTAGES * Cfg::TILE_BYTES;                // dS^T: two chunks of [128 keys][64 queries], 128B swizzle
  uint8_t* sDQ = sdS + Cfg::DS_BYTES;                                 // per drain warp two of [32 rows][32 fp32], 128B swizzle
  float* sStat = reinterpret_cast<float*>(sDQ + Cfg::DQ_BYTES);       // [stage][-lse * log2(e) | -delta * scale][128]

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const BwdWork work = bwd_work<SPLIT>(p, Cfg::BM, Cfg::BN, blockIdx.x);
  const int seg = work.seg, kv_head = work.kv_head, head0 = work.head0, b = work.b, k0 = work.k0, qb_first = work.qb_first, steps_per_head = work.steps_per_head,
            total_steps = work.steps;
  const bool diag = work.diag;
  const bool tm_out = !OUT_F32 && p.tma_out;
  auto load_q = [&](int it, int head, int q0) {
    const int qs = it % Cfg::QSTAGES;
    mbar_expect_tx(&bars.q_full[qs], Cfg::TILE_BYTES);
#pragma unroll
    for (int c = 0; c < Cfg::DCH; ++c)
      tma_load_4d(sQ + qs * Cfg::TILE_BYTES + c * (Cfg::BM * 128), &tm_q, &bars.q_full[qs], c * 64, head, q0, b);
  };
  auto load_do = [&](int it, int head, int q0) {
    const int os = it % Cfg::OSTAGES;
    mbar_expect_tx(&bars.do_full[os], Cfg::TILE_BYTES);
#pragma unroll
    for (int c = 0; c < Cfg::DCH; ++c)
      tma_load_4d(sdO + os * Cfg::TILE_BYTES + c * (Cfg::BM * 128), &tm_do, &bars.do_full[os], c * 64, head, q0, b);
  };

  if (warp == CW + 4 && elect_one()) {
    mbar_init(&bars.kv_full, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(&bars.q_full[s], 1);
      mbar_init(&bars.q_empty[s], 1);
      mbar_init(&bars.do_full[s], 1);
      mbar_init(&bars.do_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars.st_full[s], 32);
      mbar_init(&bars.st_empty[s], CW);
    }
    mbar_init(&bars.s_full, 1);
    mbar_init(&bars.s_read, CW);        // compute -> MMA: one arrival per warp
    mbar_init(&bars.p_ready, CW);
    mbar_init(&bars.p_free, 1);
    mbar_init(&bars.dp_full, 1);
    mbar_init(&bars.dp_read, CW);
    mbar_init(&bars.ds_ready, CW);
    mbar_init(&bars.ds_free, 1);
    mbar_init(&bars.dq_full, 1);
    mbar_init(&bars.dq_read, 4);
    mbar_init(&bars.acc_full, 1);
    bars.abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&segs.k[seg]);
    tma_prefetch_desc(&segs.v[seg]);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_dq);
    if (tm_out) {
      tma_prefetch_desc(&tm_dk);
      tma_prefetch_desc(&tm_dv);
    }
    // The first loads leave before the other warps are let go: they travel under the tensor-memory allocation and the first barrier.
    pdl_wait();
    if (total_steps > 0) {
      mbar_expect_tx(&bars.kv_full, 2 * Cfg::TILE_BYTES);
#pragma unroll
      for (int c = 0; c < Cfg::DCH; ++c) {
        tma_load_4d(sK + c * (Cfg::BN * 128), &segs.k[seg], &bars.kv_full, c * 64, kv_head, k0, b);
        tma_load_4d(sV + c * (Cfg::BN * 128), &segs.v[seg], &bars.kv_full, c * 64, kv_head, k0, b);
      }
      load_q(0, head0, qb_first * Cfg::BM);
      load_do(0, head0, qb_first * Cfg::BM);
    }
  }
  if (warp == CW + 5) {
    tmem_alloc(&bars.tmem_base, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();                      // barrier init and tensor-memory allocation overlapped the predecessor's tail
  const uint32_t tmem_base = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;

  if (warp >= CW + 4) regs_dec<Warps::REGS_REST>();
  if (warp == CW + 4) {
    // ------------------------------------------------------------------------------ TMA producer
    if (total_steps > 0 && elect_one()) {
      for (int it = 1; it < total_steps; ++it) {           // (the first step's and K, V: above)
        const int head = head0 + it / steps_per_head, q0 = (qb_first + it % steps_per_head) * Cfg::BM;
        if (!mbar_wait(&bars.q_empty[it % Cfg::QSTAGES], ((it / Cfg::QSTAGES) & 1) ^ 1, abort_flag)) { report_error(status, KID_BWD, 1); break; }
        load_q(it, head, q0);
        if (!mbar_wait(&bars.do_empty[it % Cfg::OSTAGES], ((it / Cfg::OSTAGES) & 1) ^ 1, abort_flag)) { report_error(status, KID_BWD, 11); break; }
        load_do(it, head, q0);
      }
    }
  } else if (warp == CW + 5) {
    // ------------------------------------------------------------------------------ MMA issuer
    if (total_steps > 0 && elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);   // S^T, dP^T: [key, query], K-major operands
      constexpr uint32_t idesc_kv = make_idesc_bf16(128, D, false, true);     // dV, dK: A = P^T (TMEM) / dS^T (K-major), B = dO / Q (MN-major)
      constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, true, true);      // dQ: A = dS^T seen as dS (MN-major), B = K (MN-major)
      bool ok = mbar_wait(&bars.kv_full, 0, abort_flag);
      if (!ok) report_error(status, KID_BWD, 2);
      // Base descriptors, built once: "km" = K-major view (LBO 16), "mn" = MN-major view (LBO = 64-column chunk).
      const uint32_t k_addr = smem_u32(sK), ds_addr = smem_u32(sdS);
      const uint64_t k_km = make_smem_desc_sw128(k_addr, 16, 1024), k_mn = make_smem_desc_sw128(k_addr, 128 * 128, 1024);
      const uint64_t v_km = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t ds_mn = make_smem_desc_sw128(ds_addr, 128 * 128, 1024), ds_km = make_smem_desc_sw128(ds_addr, 16, 1024);
      const uint64_t q_km0 = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), q_mn0 = make_smem_desc_sw128(smem_u32(sQ), 128 * 128, 1024);
      const uint64_t do_km0 = make_smem_desc_sw128(smem_u32(sdO), 16, 1024), do_mn0 = make_smem_desc_sw128(smem_u32(sdO), 128 * 128, 1024);
      // S^T = K Q^T of step `it`
      auto issue_s = [&](int it) -> bool {
        const int qs = it % Cfg::QSTAGES;
        if (!mbar_wait(&bars.q_full[qs], (it / Cfg::QSTAGES) & 1, abort_flag)) { report_error(status, KID_BWD, 3); return false; }
        tcgen05_fence_after();
        const uint64_t q_km = smem_desc_advance(q_km0, qs * Cfg::TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
          umma_bf16(tmem_base + Cfg::S_COL, smem_desc_advance(k_km, off), smem_desc_advance(q_km, off), idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars.s_full);
        return true;
      };
      // dP^T = V dO^T of step `it`
      auto issue_dp = [&](int it) -> bool {
        const int os = it % Cfg::OSTAGES;
        if (!mbar_wait(&bars.do_full[os], (it / Cfg::OSTAGES) & 1, abort_flag)) { report_error(status, KID_BWD, 12); return false; }
        tcgen05_fence_after();
        const uint64_t do_km = smem_desc_advance(do_km0, os * Cfg::TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
          umma_bf16(tmem_base + Cfg::DP_COL, smem_desc_advance(v_km, off), smem_desc_advance(do_km, off), idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars.dp_full);
        return true;
      };
      ok = ok && issue_s(0);
      if (!Cfg::SHARE) ok = ok && issue_dp(0);
      for (int it = 0; it < total_steps && ok; ++it) {
        const uint32_t par = it & 1;
        const bool next = it + 1 < total_steps;
        if (!Cfg::SHARE && next) {        // the compute warps hold S of this step in registers: the next one may overwrite it
          if (!mbar_wait(&bars.s_read, par, abort_flag)) { report_error(status, KID_BWD, 4); break; }
          if (!issue_s(it + 1)) break;
        }
        if (Cfg::SHARE) {                 // dP shares its columns with dQ of the previous step
          if (it > 0 && !mbar_wait(&bars.dq_read, par ^ 1, abort_flag)) { report_error(status, KID_BWD, 6); break; }
          if (!issue_dp(it)) break;
        }
        // dV += P^T dO : M = 128 keys, N = D, reduction over the 128 query rows
        if (!mbar_wait(&bars.p_ready, par, abort_flag)) { report_error(status, KID_BWD, 5); break; }
        tcgen05_fence_after();
        const uint64_t do_mn = smem_desc_advance(do_mn0, (it % Cfg::OSTAGES) * Cfg::TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma_bf16_ts(tmem_base + Cfg::DV_COL, tmem_base + Cfg::P_COL + kk / (W / 16) * P_PART + kk % (W / 16) * 8,
                       smem_desc_advance(do_mn, kk * 2048), idesc_kv, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&bars.p_free);
        umma_commit(&bars.do_empty[it % Cfg::OSTAGES]);
        if (next) {
          if (Cfg::SHARE) {               // S overwrites P: dV must have read it
            if (!mbar_wait(&bars.p_free, par, abort_flag)) { report_error(status, KID_BWD, 13); break; }
            if (!issue_s(it + 1)) break;
          } else {
            if (!mbar_wait(&bars.dp_read, par, abort_flag)) { report_error(status, KID_BWD, 14); break; }
            if (!issue_dp(it + 1)) break;
          }
        }
        if (!mbar_wait(&bars.ds_ready, par, abort_flag)) { report_error(status, KID_BWD, 15); break; }
        if (!Cfg::SHARE && it > 0 && !mbar_wait(&bars.dq_read, par ^ 1, abort_flag)) { report_error(status, KID_BWD, 16); break; }
        tcgen05_fence_after();
        // dQ = dS K : M = 128 query rows, N = D, reduction over the 128 keys (first: its drain is the longer way)
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma_bf16(tmem_base + Cfg::DQ_COL, smem_desc_advance(ds_mn, kk * 2048), smem_desc_advance(k_mn, kk * 2048), idesc_dq,
                    kk > 0 ? 1u : 0u);
        umma_commit(&bars.dq_full);
        // dK += dS^T Q : M = 128 keys, N = D, reduction over the 128 query rows
        const uint64_t q_mn = smem_desc_advance(q_mn0, (it % Cfg::QSTAGES) * Cfg::TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma_bf16(tmem_base + Cfg::DK_COL, smem_desc_advance(ds_km, (kk >> 2) * (128 * 128) + (kk & 3) * 32),
                    smem_desc_advance(q_mn, kk * 2048), idesc_kv, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&bars.ds_free);
        umma_commit(&bars.q_empty[it % Cfg::QSTAGES]);
      }
      if (ok) umma_commit(&bars.acc_full);
    }
  } else if (warp == CW + 6) {
    // ------------------------------------------------------------------------------ row statistics (lse, delta) of a step's queries
    int q_at = qb_first * Cfg::BM, head = head0;
    for (int it = 0; it < total_steps; ++it) {
      const int st = it & 1;
      const int q0 = q_at;
      const long long base = ((long long)b * p.hq + head) * p.Sq;
      if ((q_at += Cfg::BM) >= p.Sq) {
        q_at = qb_first * Cfg::BM;
        ++head;
      }
      float l[4], dl[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = q0 + lane + 32 * i;
        // rows beyond Sq: exp2(0 - inf) = 0
        l[i] = row < p.Sq ? -LSE[base + row] * LOG2E : -INFINITY;
        dl[i] = row < p.Sq ? -DELTA[base + row] * p.scale : 0.f;
      }
      if (!mbar_wait(&bars.st_empty[st], ((it >> 1) & 1) ^ 1, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 17); break; }
      float* dst = sStat + st * 2 * Cfg::BM;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dst[lane + 32 * i] = l[i];
        dst[Cfg::BM + lane + 32 * i] = dl[i];
      }
      mbar_arrive(&bars.st_full[st]);
    }
  } else if (warp >= CW && warp < CW + 4) {
    // ------------------------------------------------------------------------------ dQ of every step -> fp32 workspace
    // Warp w owns 32 query rows: it stages 32 columns at a time in one of its two buffers and hands them to TMA reduce-adds.
    regs_dec<Warps::REGS_DRAIN>();
    const int quarter = warp & 3;
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16) + Cfg::DQ_COL;
    uint8_t* stg = sDQ + quarter * 8192;
    const bool prof_on = PROF && p.prof != nullptr && threadIdx.x == CW * 32;
    long long pacc[2] = {0, 0};
    int q_at = qb_first * Cfg::BM, head = head0;
    for (int it = 0; it < total_steps; ++it) {
      const int row0 = q_at + quarter * 32, head_here = head;
      if ((q_at += Cfg::BM) >= p.Sq) {
        q_at = qb_first * Cfg::BM;
        ++head;
      }
      const long long pt0 = prof_clock(prof_on);
      if (!mbar_wait(&bars.dq_full, it & 1, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 9); break; }
      tcgen05_fence_after();
      const long long pt1 = prof_clock(prof_on);
      constexpr int DR = PARTS == 4 ? 32 : 64;              // columns read at a time: what the registers hold
#pragma unroll
      for (int r_ = 0; r_ < D / DR; ++r_) {
        uint32_t r[DR];
#pragma unroll
        for (int h = 0; h < DR / 32; ++h) tmem_ld_32x32b_x32_at(t_lane + r_ * DR + h * 32, r, h * 32);
        tmem_ld_wait();
        if (r_ == D / DR - 1) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.dq_read);
        }
#pragma unroll
        for (int h = 0; h < DR / 32; ++h) {
          uint8_t* const buf = stg + ((r_ * (DR / 32) + h) & 1) * 4096;
          if (elect_one()) tma_store_wait_read<1>();          // the reduce before the last has finished reading this buffer
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<uint4*>(buf + sw128_offset(lane, u)) =
                make_uint4(r[h * 32 + 4 * u], r[h * 32 + 4 * u + 1], r[h * 32 + 4 * u + 2], r[h * 32 + 4 * u + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (row0 < p.Sq) tma_reduce_add_4d(&tm_dq, buf, r_ * DR + h * 32, head_here, row0, b);
            tma_store_commit();
          }
        }
      }
      if (prof_on) { const long long pt2 = clock64(); pacc[0] += pt1 - pt0; pacc[1] += pt2 - pt1; }
    }
    if (elect_one()) tma_store_wait<0>();
    if (prof_on) {
      atomicAdd(&p.prof[2], (unsigned long long)pacc[0]);
      atomicAdd(&p.prof[3], (unsigned long long)pacc[1]);
    }
  } else if (warp < CW) {
    // ------------------------------------------------------------------------------ compute threads (warps 0 .. 4 PARTS - 1)
    regs_inc<Warps::REGS_COMPUTE>();
    // The PARTS threads t, t + 128, ... share key k0 + t (TMEM lane t): part i owns query columns i W .. (i + 1) W - 1 of a step; the
    // first half of the parts writes dV, the other dK (SUBS threads per row). Nothing has to be exchanged between them.
    constexpr int SUBS = PARTS / 2;
    const int t = threadIdx.x & 127;
    const int part = threadIdx.x >> 7;
    // dS^T of this thread: W / 8 16-byte units of row t, the first at ds_off, the others an exclusive-or of their number away
    const uint32_t ds_off = ((unsigned)(part * W) >> 6) * (128 * 128) + sw128_offset(t, ((unsigned)(part * W) & 63u) >> 3);
    const int quarter = warp & 3;
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    const uint64_t sl2_2 = pair_of(p.scale * LOG2E, p.scale * LOG2E), scale_2 = pair_of(p.scale, p.scale);
    const int key = k0 + t;
    bool ok = total_steps > 0;
    const bool prof_on = PROF && p.prof != nullptr && threadIdx.x == 0;
    long long pacc[2] = {0, 0};
    const long long pstart = prof_clock(prof_on);
    int q_at = qb_first * Cfg::BM;                         // first query of the step (the steps go through them once per head)
    for (int it = 0; it < total_steps; ++it) {
      const long long pt0 = prof_clock(prof_on);
      const uint32_t par = it & 1;
      // first query of this thread's columns (a division a step is slower, but four parts have no register for the counter)
      const int qcol0 = (PARTS == 4 ? (qb_first + it % steps_per_head) * Cfg::BM : q_at) + part * W;
      if (PARTS != 4 && (q_at += Cfg::BM) >= p.Sq) q_at = qb_first * Cfg::BM;
      const bool need_mask = (diag && k0 + Cfg::BN - 1 > qcol0) || (k0 + Cfg::BN > p.Sk);
      const int hidden = key >= p.Sk ? W : (diag ? key - qcol0 : 0);              // columns [0, hidden) do not see this key
      const float* st_l = sStat + par * 2 * Cfg::BM + part * W;
      const float* st_d = st_l + Cfg::BM;
      if (!mbar_wait(&bars.st_full[par], (it >> 1) & 1, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 18); ok = false; break; }
      if (!mbar_wait(&bars.s_full, par, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 7); ok = false; break; }
      tcgen05_fence_after();
      const long long pt1 = prof_clock(prof_on);
      uint32_t s[W];
#pragma unroll
      for (int h = 0; h < W / 32; ++h) tmem_ld_32x32b_x32_at(t_lane + Cfg::S_COL + part * W + h * 32, s, h * 32);
      tmem_ld_wait();
      if (!Cfg::SHARE) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.s_read);
      }
      uint32_t pk[W / 2];                     // P^T of this thread's queries, bf16 pairs
      // The masked and the plain form are separate code: a test of need_mask inside the loop costs a branch per element group,
      // which took the scheduler's freedom away (d = 64, 32768 keys: 26.7 ms with it, 17.2 without).
      auto exponentials = [&](auto masked) {
#pragma unroll
        for (int e = 0; e < W; e += 4) {
          const float4 lv = *reinterpret_cast<const float4*>(st_l + e);
          const uint64_t x0 = fma2(pair_of(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sl2_2, pair_of(lv.x, lv.y));
          const uint64_t x1 = fma2(pair_of(__uint_as_float(s[e + 2]), __uint_as_float(s[e + 3])), sl2_2, pair_of(lv.z, lv.w));
          float pv[4] = {fast_exp2(lo_of(x0)), fast_exp2(hi_of(x0)), fast_exp2(lo_of(x1)), fast_exp2(hi_of(x1))};
          if constexpr (decltype(masked)::value) {
#pragma unroll
            for (int i = 0; i < 4; ++i) pv[i] = e + i < hidden ? 0.f : pv[i];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) s[e + i] = __float_as_uint(pv[i]);
          pk[e >> 1] = pack_bf16(pv[0], pv[1]);
          pk[(e >> 1) + 1] = pack_bf16(pv[2], pv[3]);
        }
      };
      if (need_mask) exponentials(std::true_type{});
      else exponentials(std::false_type{});
      if (!Cfg::SHARE && it > 0) {                                  // the dV MMA of the previous step has read its P
        if (!mbar_wait(&bars.p_free, par ^ 1, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 19); ok = false; break; }
        tcgen05_fence_after();
      }
      if constexpr (W == 64) tmem_st_32x32b_x32(t_lane + Cfg::P_COL + part * P_PART, pk);
      else tmem_st_32x32b_x16(t_lane + Cfg::P_COL + part * P_PART, pk);
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.p_ready);
      const long long pt4 = prof_clock(prof_on);
      if (!mbar_wait(&bars.dp_full, par, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 8); ok = false; break; }
      tcgen05_fence_after();
      const long long pt5 = prof_clock(prof_on);
      uint32_t dp[W];
#pragma unroll
      for (int h = 0; h < W / 32; ++h) tmem_ld_32x32b_x32_at(t_lane + Cfg::DP_COL + part * W + h * 32, dp, h * 32);
      tmem_ld_wait();
      if (!Cfg::SHARE) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.dp_read);
      }
#pragma unroll
      for (int e = 0; e < W; e += 4) {
        const float4 dv = *reinterpret_cast<const float4*>(st_d + e);
        const uint64_t d0 = mul2(pair_of(__uint_as_float(s[e]), __uint_as_float(s[e + 1])),
                                 fma2(pair_of(__uint_as_float(dp[e]), __uint_as_float(dp[e + 1])), scale_2, pair_of(dv.x, dv.y)));
        const uint64_t d1 = mul2(pair_of(__uint_as_float(s[e + 2]), __uint_as_float(s[e + 3])),
                                 fma2(pair_of(__uint_as_float(dp[e + 2]), __uint_as_float(dp[e + 3])), scale_2, pair_of(dv.z, dv.w)));
        pk[e >> 1] = pack_bf16(lo_of(d0), hi_of(d0));
        pk[(e >> 1) + 1] = pack_bf16(lo_of(d1), hi_of(d1));
      }
      // the dQ and dK MMAs of the previous step have read its dS
      if (it > 0 && !mbar_wait(&bars.ds_free, par ^ 1, abort_flag)) { if (lane == 0) report_error(status, KID_BWD, 20); ok = false; break; }
#pragma unroll
      for (int u = 0; u < W / 8; ++u)
        *reinterpret_cast<uint4*>(sdS + (ds_off ^ (uint32_t)(u << 4))) =
            make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
      tcgen05_fence_before();                 // (also orders the reads of dP before the dQ MMA that may reuse its columns)
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bars.ds_ready);
        mbar_arrive(&bars.st_empty[par]);
      }
      if (prof_on) {
        const long long pt6 = clock64();
        pacc[0] += (pt1 - pt0) + (pt5 - pt4);
        pacc[1] += (pt4 - pt1) + (pt6 - pt5);
      }
    }
    if (prof_on) {
      for (int i = 0; i < 2; ++i) atomicAdd(&p.prof[i], (unsigned long long)pacc[i]);
      atomicAdd(&p.prof[4], (unsigned long long)total_steps);
      atomicAdd(&p.prof[5], (unsigned long long)(clock64() - pstart));
      atomicAdd(&p.prof[6], work.part == 0 ? 1ull : 0ull);
    }
    {  // names of its own: what the end needs is read anew
      if constexpr (SPLIT) {
        // The other CTAs' sums come to the first one's shared memory, in the place of the operand rings and dS, when everybody's MMAs are done.
        if (ok && !mbar_wait(&bars.acc_full, 0, abort_flag)) {
          if (lane == 0) report_error(status, KID_BWD, 10);
          ok = false;
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        tcgen05_fence_after();
        if (ok && cluster_ctarank() > 0) bwd_send_sums<D, PARTS>(tmem_base, mapa_u32(smem_u32(sQ), 0) + (cluster_ctarank() - 1) * BWD_SUM_BYTES<D>);
        __syncwarp();
        cluster_arrive();
        cluster_wait();
      }
      // dK, dV of this key block (thread t <-> key k0 + t); fp32 when they are partials of a multi-rank reduction
      // (The block and thread are read anew: what is kept from before the loop over the steps takes registers there, and with the stores below
      // its compute warps executed 8 % more instructions, 14.0 -> 14.6 ms at 32,768 tokens.)
      unsigned cta, thread;
      asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
      asm volatile("mov.u32 %0, %%tid.x;" : "=r"(thread));
      const BwdWork work = bwd_work<SPLIT>(p, Cfg::BM, Cfg::BN, cta);
      const int kv_head = work.kv_head, b = work.b, k0 = work.k0, seg = work.seg, total_steps = work.steps;
      constexpr int SUBS = PARTS / 2;
      const int lane = thread & 31, quarter = (thread >> 5) & 3, part = thread >> 7, which = part / SUBS, sub = part % SUBS, key = k0 + (int)(thread & 127);
      const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
      const bool tm_out = !OUT_F32 && p.tma_out;
      const long long seg_off = (long long)seg * p.seg_stride;
      if (SPLIT && work.part > 0) {            // (its sums are with the first)
      } else if (total_steps == 0) {
        if (key < p.Sk && sub == 0) {
          {
            const long long rs_ = which == 0 ? p.dv_row : p.dk_row;
            const long long off = seg_off + ((long long)b * p.Sk + key) * rs_ + (long long)kv_head * D;
            if (OUT_F32) {
              float* orow = reinterpret_cast<float*>(which == 0 ? dV_ : dK_) + off;
              for (int u = 0; u < D / 4; ++u) reinterpret_cast<float4*>(orow)[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
              bf16* orow = reinterpret_cast<bf16*>(which == 0 ? dV_ : dK_) + off;
              for (int u = 0; u < D / 8; ++u) reinterpret_cast<uint4*>(orow)[u] = make_uint4(0, 0, 0, 0);
            }
          }
        }
      } else if (ok && (SPLIT || (which == 0 ? mbar_wait(&bars.p_free, (total_steps - 1) & 1, abort_flag) : mbar_wait(&bars.acc_full, 0, abort_flag)))) {
        // dV is complete with its last MMA, half a step before dK. Rows of 16 columns (32 bytes) of each warp's 32 keys go to TMA through the
        // place of V, which the last dP was the last to read, and of K: stored by every thread for itself they were 16-byte pieces of 32 rows an
        // instruction, and the end of a CTA took 3,600 (d = 64) and 7,600 cycles (d = 128) of the 20,900 and 34,000 that one of 4 x 1024,
        // 32 heads lives.
        tcgen05_fence_after();
        const long long rs_ = which == 0 ? p.dv_row : p.dk_row;
        const long long off = seg_off + ((long long)b * p.Sk + (key < p.Sk ? key : 0)) * rs_ + (long long)kv_head * D;
        uint8_t* const stg = (which == 0 ? sV : sK) + (sub * 4 + quarter) * (D / SUBS * 64);
        int pieces = 0;
        // 4 x N columns of this row from `col` on, of the other CTAs, in their order
        auto add_parts = [&](int col, uint32_t* r, int quads) {
          for (int o = 1; SPLIT && o < p.parts; ++o) {
            const float4* const q = reinterpret_cast<const float4*>(sQ + (o - 1) * BWD_SUM_BYTES<D>) + (which * (D / 4) + col / 4) * 128 + (thread & 127);
  #pragma unroll
            for (int u = 0; u < 8; ++u)
              if (u < quads) {
                const float4 v = q[u * 128];
                r[4 * u] = __float_as_uint(__uint_as_float(r[4 * u]) + v.x);
                r[4 * u + 1] = __float_as_uint(__uint_as_float(r[4 * u + 1]) + v.y);
                r[4 * u + 2] = __float_as_uint(__uint_as_float(r[4 * u + 2]) + v.z);
                r[4 * u + 3] = __float_as_uint(__uint_as_float(r[4 * u + 3]) + v.w);
              }
          }
        };
        auto put16 = [&](int col, const uint32_t* r) {        // 16 columns of this thread's row from `col` on
          const uint4 lo = make_uint4(pack_bf16(__uint_as_float(r[0]), __uint_as_float(r[1])), pack_bf16(__uint_as_float(r[2]), __uint_as_float(r[3])),
                                      pack_bf16(__uint_as_float(r[4]), __uint_as_float(r[5])), pack_bf16(__uint_as_float(r[6]), __uint_as_float(r[7])));
          const uint4 hi = make_uint4(pack_bf16(__uint_as_float(r[8]), __uint_as_float(r[9])), pack_bf16(__uint_as_float(r[10]), __uint_as_float(r[11])),
                                      pack_bf16(__uint_as_float(r[12]), __uint_as_float(r[13])), pack_bf16(__uint_as_float(r[14]), __uint_as_float(r[15])));
          if (tm_out) {
            uint4* const q = reinterpret_cast<uint4*>(stg + pieces * 1024 + lane * 32);
            q[0] = lo;
            q[1] = hi;
            fence_proxy_async_smem();
            __syncwarp();
            if (elect_one()) {
              const int row0 = k0 + quarter * 32;
              if (row0 < p.Sk) tma_store_4d(which == 0 ? &tm_dv : &tm_dk, stg + pieces * 1024, col, kv_head, row0, b);
              tma_store_commit();
            }
            ++pieces;
          } else if (key < p.Sk) {
            uint4* const q = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(which == 0 ? dV_ : dK_) + off + col);
            q[0] = lo;
            q[1] = hi;
          }
        };
        if (!OUT_F32 && which == 1 && p.cosT != nullptr) {
          // dK with the inverse rotation: pairs j <-> j + D/2, 16 columns of each half of the row at a time
          const int pos = (key < p.Sk ? key : 0) % p.rope_seq;
          const float* cos_row = p.cosT + (long long)pos * (D / 2);
          const float* sin_row = p.sinT + (long long)pos * (D / 2);
  #pragma unroll 1
          for (int c = sub; c < D / 32; c += SUBS) {
            uint32_t lo[16], hi[16];
            tmem_ld_32x32b_x16(t_lane + Cfg::DK_COL + c * 16, lo);
            tmem_ld_32x32b_x16(t_lane + Cfg::DK_COL + D / 2 + c * 16, hi);
            tmem_ld_wait();
            add_parts(c * 16, lo, 4);
            add_parts(D / 2 + c * 16, hi, 4);
  #pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 cs = __ldg(reinterpret_cast<const float4*>(cos_row + c * 16 + j));
              const float4 sn = __ldg(reinterpret_cast<const float4*>(sin_row + c * 16 + j));
              const float csv[4] = {cs.x, cs.y, cs.z, cs.w}, snv[4] = {sn.x, sn.y, sn.z, sn.w};
  #pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float a = __uint_as_float(lo[j + i]), b_ = __uint_as_float(hi[j + i]);
                lo[j + i] = __float_as_uint(a * csv[i] + b_ * snv[i]);
                hi[j + i] = __float_as_uint(b_ * csv[i] - a * snv[i]);
              }
            }
            put16(c * 16, lo);
            put16(D / 2 + c * 16, hi);
          }
        } else {
          const int col_base = which == 0 ? Cfg::DV_COL : Cfg::DK_COL;
  #pragma unroll 1
          for (int c = sub; c < D / 32; c += SUBS) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_lane + col_base + c * 32, r);
            tmem_ld_wait();
            add_parts(c * 32, r, 8);
            if (OUT_F32) {
              if (key < p.Sk) {
                float* orow = reinterpret_cast<float*>(which == 0 ? dV_ : dK_) + off + c * 32;
  #pragma unroll
                for (int u = 0; u < 8; ++u)
                  reinterpret_cast<float4*>(orow)[u] = make_float4(__uint_as_float(r[4 * u]), __uint_as_float(r[4 * u + 1]),
                                                                   __uint_as_float(r[4 * u + 2]), __uint_as_float(r[4 * u + 3]));
              }
            } else {
              put16(c * 32, r);
              put16(c * 32 + 16, r + 16);
            }
          }
        }
        if (tm_out && elect_one()) tma_store_wait<0>();
      } else if (ok && lane == 0) {
        report_error(status, KID_BWD, 10);
      }
    }
  }
  if constexpr (SPLIT) {
    if (warp >= CW) {                  // (the compute warps' two)
      for (int i = 0; i < 2; ++i) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == CW + 5) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

#define PT_BWD_PARAMS                                                                                                           \
  const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ KVSegs segs, const __grid_constant__ CUtensorMap tm_do,      \
      const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk,                                     \
      const __grid_constant__ CUtensorMap tm_dv, const float* __restrict__ LSE, const float* __restrict__ DELTA,                 \
      void* __restrict__ dK_, void* __restrict__ dV_, const __grid_constant__ BwdParams p, KernelStatus* status
// (two kernels, because the build checks their register counts by name)
template <int D, bool OUT_F32, bool PROF, bool SPLIT>
__global__ void __launch_bounds__(BwdWarps<2>::THREADS, 1) attn_bwd_kernel(PT_BWD_PARAMS) {
  attn_bwd_body<D, OUT_F32, PROF, SPLIT, 2>(tm_q, segs, tm_do, tm_dq, tm_dk, tm_dv, LSE, DELTA, dK_, dV_, p, status);
}
template <int D, bool OUT_F32, bool PROF, bool SPLIT>
__global__ void __launch_bounds__(BwdWarps<4>::THREADS, 1) attn_bwd_parts4_kernel(PT_BWD_PARAMS) {
  attn_bwd_body<D, OUT_F32, PROF, SPLIT, 4>(tm_q, segs, tm_do, tm_dq, tm_dk, tm_dv, LSE, DELTA, dK_, dV_, p, status);
}
#undef PT_BWD_PARAMS

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
// tensor map over x[B, S, h, d] with token stride `row` (elements): dims {d, h, S, B}, box {64, 1, rows, 1}
static int make_attn_map(CUtensorMap* m, const void* base, int B, int S, int h, int d, long long row, int box_rows) {
  uint64_t dims[4] = {(uint64_t)d, (uint64_t)h, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)d, (uint64_t)row, (uint64_t)row * (uint64_t)S};
  uint32_t box[4] = {64, 1, (uint32_t)box_rows, 1};
  return make_bf16_map(m, base, 4, dims, strides, box);
}

template <int D, int BN, bool PROF = false>
static int launch_fwd(const CUtensorMap& mq, const KVSegs& segs, const CUtensorMap& mo, float* lse, const AttnParams& p,
                      KernelStatus* st, cudaStream_t stream) {
  if (!PROF && p.prof != nullptr) return launch_fwd<D, BN, true>(mq, segs, mo, lse, p, st, stream);
  auto kern = attn_fwd_kernel<D, BN, PROF>;
  static PerDevice configured;
  const int rc = configured.get(current_device(), [&] {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg<D, BN>::SMEM) != cudaSuccess) return -3;
    // two CTAs per SM need the largest shared-memory carve-out
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return 1;
  });
  if (rc <= 0) return rc;
  const int num_qb = (p.Sq + 127) / 128;
  const long long grid = (long long)num_qb * p.hq * p.B;
  launch_pdl(kern, dim3((unsigned)grid), dim3(192), FwdCfg<D, BN>::SMEM, stream, mq, segs, mo, lse, p, st);
  pt_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

static long long key_blocks(const BwdParams& p) { return (long long)((p.Sk + 127) / 128) * p.n_segs * p.hkv * p.B; }

// Steps until the last key block is done, `slots` of them at a time in the order of bwd_work (never longer than those before) with `parts` CTAs
// each; a CTA that has to wait for another costs the six steps of its start and end, too. -1: three waves.
static long long bwd_span(const BwdParams& p, int parts, long long slots) {
  const long long bps = (p.Sk + 127) / 128, num_qb = (p.Sq + 127) / 128, heads = (long long)p.hkv * p.B, n = key_blocks(p);
  auto steps = [&](long long i) {
    const long long of_last = i / heads - (p.n_segs - 1) * bps;          // (causal: number in the last segment, whose blocks get shorter)
    return (p.causal && of_last > 0 ? std::max(num_qb - of_last, 0LL) : num_qb) * (p.hq / p.hkv / parts);
  };
  if (n > 2 * slots) return -1;
  long long span = steps(0);
  for (long long j = 0; j + slots < n; ++j) span = std::max(span, steps(slots - 1 - j) + 6 + steps(slots + j));
  return span;
}

// CTAs of a cluster that share the query heads of a key block, as far as their sums fit beside each other (3 for d = 64, 2 for d = 128) and all parts
// could have an SM each: those that save the most steps beyond what sharing costs, four, or five for three CTAs from a third of the SMs on.
// clusters(n): how many clusters of n CTAs the device holds at a time. Of three CTAs that is 45 here, but from 41 on some came late in every
// few launches (16 steps: 40 clusters 77 us, 42 87, 44 112, 48 117), so a ninth less is counted on; pairs are as many as said (74: 89 us, 75: 117).
// Of 678 shapes (9 head layouts, 64 to 2,048 tokens, causal or not, at most 160 CTAs) none is more than 2 % slower than with whole blocks, and the sum
// is 0.3 % above that of the fastest: 3 x 601, 9 / 3 heads 34.5 us, in three parts 28.7; 8 x 256 (48 blocks, two waves) stays at 21.0, in three
// 29.1; 4 x 256 (24 blocks of 6 steps) at 18.7, in three 19.9; 8 x 384, 12 / 2 heads 40.4, in two 32.3, in three 34.6. Without room for all parts:
// 8 x 1024, 9 / 3 heads 57 us, in three 98.
template <class Clusters>
static int bwd_head_parts(const BwdParams& p, int d, int sms, int largest, Clusters clusters) {
  const long long group = p.hq / p.hkv, ctas = key_blocks(p), whole = bwd_span(p, 1, sms);
  long long most = -1;
  int best = 1;
  for (int parts = std::min(d == 64 ? 3 : 2, largest); parts > 1; --parts) {
    const long long cost = parts == 3 && 3 * 3 * ctas > sms ? 5 : 4;
    if (group % parts || ctas * parts > sms || whole - bwd_span(p, parts, ctas) - cost <= most) continue;       // (not even if all are there at once)
    const int at_once = clusters(parts), slots = parts == 3 ? at_once - at_once / 9 : at_once;
    const long long span = slots > 0 ? bwd_span(p, parts, slots) : -1;
    if (span < 0 || whole - span - cost <= most) continue;
    most = whole - span - cost;
    best = parts;
  }
  return best;
}
static thread_local int g_largest_cluster = 3;       // (the thread's switch, for tests and measurements)

template <int D, bool OUT_F32, bool PROF, bool SPLIT>
static auto bwd_kernel() {
  if constexpr (bwd_parts<D>() == 4) return attn_bwd_parts4_kernel<D, OUT_F32, PROF, SPLIT>;
  else return attn_bwd_kernel<D, OUT_F32, PROF, SPLIT>;
}
// Sets the kernel up for the device; SMs, or with SPLIT the clusters of `size` CTAs that it holds at a time (an SM partition may have none), or an error
// code below zero.
template <int D, bool OUT_F32, bool PROF, bool SPLIT>
static int bwd_slots(int size) {
  using Warps = BwdWarps<bwd_parts<D>()>;
  static PerDevice slots[2];                         // (one more, so that none is a number, too)
  const int n = slots[size > 2].get(current_device(), [&] {
    auto kern = bwd_kernel<D, OUT_F32, PROF, SPLIT>();
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdCfg<D>::SMEM) != cudaSuccess) return -3;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    // the warpgroups share out Warps::REGS registers per thread; with fewer at launch setmaxnreg.inc would wait forever (the build
    // fails for another count, build.py: FIXED_REGISTERS)
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess || fa.numRegs != Warps::REGS) return -6;
    int n = 0;
    if (!SPLIT) {
      int dev = 0;
      if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -3;
      return n + 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3(Warps::THREADS);
    cfg.dynamicSmemBytes = BwdCfg<D>::SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    return n + 1;
  });
  return n > 0 ? n - 1 : n;
}

template <int D, bool OUT_F32, bool PROF = false, bool SPLIT = false>
static int launch_bwd(const CUtensorMap& mq, const KVSegs& segs, const CUtensorMap& mdo, const CUtensorMap& mdq, const CUtensorMap& mdk,
                      const CUtensorMap& mdv, const float* lse, const float* delta, void* dk, void* dv, BwdParams p, KernelStatus* st,
                      cudaStream_t stream) {
  if (!PROF && p.prof != nullptr)
    return launch_bwd<D, OUT_F32, true>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, st, stream);
  if constexpr (!SPLIT) {
    const int sms = bwd_slots<D, OUT_F32, PROF, false>(1);
    if (sms <= 0) return sms;
    p.parts = bwd_head_parts(p, D, sms, g_largest_cluster, bwd_slots<D, OUT_F32, PROF, true>);
    if (p.parts > 1) return launch_bwd<D, OUT_F32, PROF, true>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, st, stream);
  }
  static_assert((D == 64 ? 2 : 1) * BWD_SUM_BYTES<D> <= (BwdCfg<D>::QSTAGES + BwdCfg<D>::OSTAGES) * BwdCfg<D>::TILE_BYTES + BwdCfg<D>::DS_BYTES,
                "the parts' sums take the place of the rings and dS");
  const cudaError_t err = launch_pdl_cluster(bwd_kernel<D, OUT_F32, PROF, SPLIT>(), dim3((unsigned)(key_blocks(p) * p.parts)),
                                             dim3(BwdWarps<bwd_parts<D>()>::THREADS), BwdCfg<D>::SMEM, stream, p.parts, mq, segs, mdo, mdq, mdk, mdv,
                                             lse, delta, dk, dv, p, st);
  pt_count_launches(1);
  return err == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace attn
}  // namespace pt

// Largest cluster of CTAs that share a key block's query heads in the backward: 3 by default, 1: none (for the calling thread).
extern "C" void pt_attention_set_clusters(int largest) { pt::attn::g_largest_cluster = largest; }
// What the rule says for a device with `sms` SMs that holds two / three CTAs a cluster pairs / triples times.
extern "C" int pt_attention_bwd_parts(int B, int Sq, int Sk, int hq, int hkv, int d, int causal, int n_segs, int sms, int pairs, int triples) {
  pt::attn::BwdParams p{};
  p.B = B, p.Sq = Sq, p.Sk = Sk, p.hq = hq, p.hkv = hkv, p.causal = causal, p.n_segs = n_segs;
  return pt::attn::bwd_head_parts(p, d, sms, 3, [&](int size) { return size == 3 ? triples : pairs; });
}

// q [B,Sq,hq,d] bf16 with token stride q_row; K/V in `n_segs` segments: k_ptrs[i]/v_ptrs[i] are [B,Sk,hkv,d] bf16 with
// token strides k_row/v_row (elements, multiples of 8) and may be peer-mapped pointers into other GPUs' memory.
// `causal` masks inside the last segment only. o [B,Sq,hq,d] bf16 contiguous; lse [B,hq,Sq] fp32 (natural log).
extern "C" int pt_attention_fwd_segs(const void* q, const void* const* k_ptrs, const void* const* v_ptrs, int n_segs,
                                     void* o, float* lse, int B, int Sq, int Sk, int hq, int hkv, int d, long long q_row,
                                     long long k_row, long long v_row, int causal, float scale, cudaStream_t st) {
  using namespace pt;
  using namespace pt::attn;
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if ((d != 64 && d != 128) || hq % hkv || (q_row % 8) || (k_row % 8) || (v_row % 8) || n_segs < 1 || n_segs > MAX_SEGS)
    return -10;
  CUtensorMap mq, mo;
  KVSegs segs;
  const int bn = d == 64 ? 128 : 64;
  int rc;
  if ((rc = make_attn_map(&mq, q, B, Sq, hq, d, q_row, 128))) return rc;
  if ((rc = make_attn_map(&mo, o, B, Sq, hq, d, (long long)hq * d, 32))) return rc;
  for (int i = 0; i < n_segs; ++i) {
    if ((rc = make_attn_map(&segs.k[i], k_ptrs[i], B, Sk, hkv, d, k_row, bn))) return rc;
    if ((rc = make_attn_map(&segs.v[i], v_ptrs[i], B, Sk, hkv, d, v_row, bn))) return rc;
  }
  for (int i = n_segs; i < MAX_SEGS; ++i) { segs.k[i] = segs.k[0]; segs.v[i] = segs.v[0]; }
  AttnParams p{B, Sq, Sk, hq, hkv, causal, scale, n_segs, g_attn_prof};
  if (d == 64) return launch_fwd<64, 128>(mq, segs, mo, lse, p, status_word_attn(), st);
  return launch_fwd<128, 64>(mq, segs, mo, lse, p, status_word_attn(), st);
}

extern "C" int pt_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq, int Sk,
                                int hq, int hkv, int d, long long q_row, long long k_row, long long v_row, int causal,
                                float scale, cudaStream_t st) {
  return pt_attention_fwd_segs(q, &k, &v, 1, o, lse, B, Sq, Sk, hq, hkv, d, q_row, k_row, v_row, causal, scale, st);
}

// Backward over `n_segs` K/V segments (see pt_attention_fwd_segs). dout, o [B,Sq,hq,d] bf16 contiguous; lse [B,hq,Sq];
// delta_in optional (else computed into delta_ws [B,hq,Sq]); dq_ws fp32 [B,Sq,hq,d] scratch, cleared together with the computation of
// delta and therefore to be handed in zeroed where delta_in is given; dq bf16 with
// token stride dq_row. dk/dv: outputs of segment i start i*seg_stride elements after dk/dv, token strides dk_row/dv_row,
// bf16 or (out_f32) fp32 -- fp32 is used when they are partial sums that another rank reduces.
static int attention_bwd_impl(const void* dout, const void* q, const void* const* k_ptrs, const void* const* v_ptrs,
                                     int n_segs, const void* o, const float* lse, const float* delta_in, float* delta_ws,
                                     float* dq_ws, void* dq, void* dk, void* dv, int out_f32, long long seg_stride, int B,
                                     int Sq, int Sk, int hq, int hkv, int d, long long q_row, long long k_row,
                                     long long v_row, long long dq_row, long long dk_row, long long dv_row, int causal,
                                     float scale, cudaStream_t st, const float* cosT, const float* sinT, int rope_seq) {
  using namespace pt;
  using namespace pt::attn;
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if ((d != 64 && d != 128) || hq % hkv || (q_row % 8) || (k_row % 8) || (v_row % 8) || (dq_row % 4) || (dk_row % 8) ||
      (dv_row % 8) || n_segs < 1 || n_segs > MAX_SEGS)
    return -10;
  const float* delta = delta_in;
  if (delta == nullptr) {
    const long long threads = (long long)B * Sq * hq * (d / 8);
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    if (d == 64) launch_pdl(delta_kernel<64>, dim3(blocks), dim3(256), 0, st, (const bf16*)dout, (const bf16*)o, delta_ws, dq_ws, B, Sq, hq);
    else launch_pdl(delta_kernel<128>, dim3(blocks), dim3(256), 0, st, (const bf16*)dout, (const bf16*)o, delta_ws, dq_ws, B, Sq, hq);
    pt_count_launches(1);
    delta = delta_ws;
  }
  CUtensorMap mq, mdo, mdq;
  KVSegs segs;
  int rc;
  if ((rc = make_attn_map(&mq, q, B, Sq, hq, d, q_row, 128))) return rc;
  if ((rc = make_attn_map(&mdo, dout, B, Sq, hq, d, (long long)hq * d, 128))) return rc;
  {
    // fp32 dQ workspace [B, Sq, hq, d]: 32-column x 32-row boxes for the TMA reduce-adds
    uint64_t dims[4] = {(uint64_t)d, (uint64_t)hq, (uint64_t)Sq, (uint64_t)B};
    uint64_t strides[3] = {(uint64_t)d, (uint64_t)hq * d, (uint64_t)hq * d * (uint64_t)Sq};
    uint32_t box[4] = {32, 1, 32, 1};
    if ((rc = make_f32_map(&mdq, dq_ws, 4, dims, strides, box))) return rc;
  }
  for (int i = 0; i < n_segs; ++i) {
    if ((rc = make_attn_map(&segs.k[i], k_ptrs[i], B, Sk, hkv, d, k_row, 128))) return rc;
    if ((rc = make_attn_map(&segs.v[i], v_ptrs[i], B, Sk, hkv, d, v_row, 128))) return rc;
  }
  for (int i = n_segs; i < MAX_SEGS; ++i) { segs.k[i] = segs.k[0]; segs.v[i] = segs.v[0]; }
  if (cosT != nullptr && (n_segs != 1 || out_f32 || sinT == nullptr || rope_seq <= 0 || (reinterpret_cast<uintptr_t>(cosT) & 15) ||
                          (reinterpret_cast<uintptr_t>(sinT) & 15)))
    return -12;
  // dk, dv through TMA: pieces of 16 columns and 32 keys
  CUtensorMap mdk = mq, mdv = mq;
  int tma_out = 0;
  if (!out_f32 && n_segs == 1) {
    auto piece_map = [&](CUtensorMap* m, const void* base, long long row) {
      uint64_t dims[4] = {(uint64_t)d, (uint64_t)hkv, (uint64_t)Sk, (uint64_t)B};
      uint64_t strides[3] = {(uint64_t)d, (uint64_t)row, (uint64_t)row * (uint64_t)Sk};
      uint32_t box[4] = {16, 1, 32, 1};
      return make_bf16_map(m, base, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE) == 0;
    };
    tma_out = piece_map(&mdk, dk, dk_row) && piece_map(&mdv, dv, dv_row);
  }
  BwdParams p{B, Sq, Sk, hq, hkv, causal, scale, dk_row, dv_row, n_segs, seg_stride, cosT, sinT, rope_seq, tma_out, 1, g_attn_prof};
  KernelStatus* sw = status_word_attn();
  if (d == 64) rc = out_f32 ? launch_bwd<64, true>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, sw, st)
                            : launch_bwd<64, false>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, sw, st);
  else rc = out_f32 ? launch_bwd<128, true>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, sw, st)
                    : launch_bwd<128, false>(mq, segs, mdo, mdq, mdk, mdv, lse, delta, dk, dv, p, sw, st);
  if (rc) return rc;
  if (dq != nullptr) {
    const long long n = (long long)B * Sq * hq * d;
    if (cosT != nullptr)
      launch_pdl(convert_dq_rope_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, st, dq_ws, (bf16*)dq, (long long)B * Sq,
                 hq, d, dq_row, cosT, sinT, rope_seq);
    else
      launch_pdl(convert_dq_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, st, dq_ws, (bf16*)dq, (long long)B * Sq,
                 hq * d, dq_row);
    pt_count_launches(1);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int pt_attention_bwd_segs(const void* dout, const void* q, const void* const* k_ptrs, const void* const* v_ptrs,
                                     int n_segs, const void* o, const float* lse, const float* delta_in, float* delta_ws,
                                     float* dq_ws, void* dq, void* dk, void* dv, int out_f32, long long seg_stride, int B, int Sq,
                                     int Sk, int hq, int hkv, int d, long long q_row, long long k_row, long long v_row,
                                     long long dq_row, long long dk_row, long long dv_row, int causal, float scale,
                                     cudaStream_t st) {
  return attention_bwd_impl(dout, q, k_ptrs, v_ptrs, n_segs, o, lse, delta_in, delta_ws, dq_ws, dq, dk, dv, out_f32, seg_stride, B,
                            Sq, Sk, hq, hkv, d, q_row, k_row, v_row, dq_row, dk_row, dv_row, causal, scale, st, nullptr, nullptr, 0);
}

// pt_attention_bwd that also undoes RoPE on its dq and dk outputs (the backward of rotating q and k before attention):
// cosT/sinT fp32 [rope_seq, d/2], 16-byte aligned; query / key i sits at position i % rope_seq.
extern "C" int pt_attention_bwd_rope(const void* dout, const void* q, const void* k, const void* v, const void* o,
                                     const float* lse, const float* delta_in, float* delta_ws, float* dq_ws, void* dq,
                                     void* dk, void* dv, int B, int Sq, int Sk, int hq, int hkv, int d, long long q_row,
                                     long long k_row, long long v_row, long long dq_row, long long dk_row, long long dv_row,
                                     int causal, float scale, const float* cosT, const float* sinT, int rope_seq,
                                     cudaStream_t st) {
  return attention_bwd_impl(dout, q, &k, &v, 1, o, lse, delta_in, delta_ws, dq_ws, dq, dk, dv, 0, 0, B, Sq, Sk, hq, hkv, d, q_row,
                            k_row, v_row, dq_row, dk_row, dv_row, causal, scale, st, cosT, sinT, rope_seq);
}

extern "C" int pt_attention_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o,
                                const float* lse, const float* delta_in, float* delta_ws, float* dq_ws, void* dq,
                                void* dk, void* dv, int B, int Sq, int Sk, int hq, int hkv, int d, long long q_row,
                                long long k_row, long long v_row, long long dq_row, long long dk_row, long long dv_row,
                                int causal, float scale, cudaStream_t st) {
  return pt_attention_bwd_segs(dout, q, &k, &v, 1, o, lse, delta_in, delta_ws, dq_ws, dq, dk, dv, 0, 0, B, Sq, Sk, hq, hkv,
                               d, q_row, k_row, v_row, dq_row, dk_row, dv_row, causal, scale, st);
}

// Phase profiling of the attention kernels: `counters` is a device buffer of 16 uint64 that subsequent forward / backward
// launches add their phase cycle counts to (layout next to AttnParams); nullptr switches it off again.
extern "C" void pt_attention_set_profile(unsigned long long* counters) { pt::attn::g_attn_prof = counters; }
