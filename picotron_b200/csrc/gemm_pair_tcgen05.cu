// bf16 GEMM for sm_100a on CTA pairs (tcgen05 cta_group::2): D[M,N] = op(A) * op(B), fp32 accumulate in TMEM.
//
// Same contract and operand layouts as gemm_tcgen05.cu, but two CTAs (a cluster of 2 on neighbouring SMs)
// cooperate on one output tile of 256 rows and 256, 192 or 128 columns (see gain_asked for which): each CTA loads
// its own 128 rows of A and its own half of the columns of B -- with plain, non-multicast TMA loads -- and one
// thread of the leader CTA issues a 256-row MMA that
// reads both CTAs' shared memory and writes both CTAs' tensor memory. Per output element this moves a
// third less operand data from L2 into shared memory than the single-CTA 128x256 tile (each B half is
// fetched once per pair instead of once per CTA), which is what the single-CTA kernel is limited by.
//
// Synchronisation between the two CTAs:
//   full[s]       lives in the leader; the leader's producer arms it with the bytes of BOTH CTAs, the
//                 peer's TMA loads credit their bytes to it (cta_group::2 form of the load).
//   empty[s]      one per CTA; the leader's MMA thread commits to both after the MMAs that read stage s.
//   tmem_full[a]  one per CTA; committed to both after the last k-block of a tile.
//   tmem_empty[a] lives in the leader; the four epilogue warps of each CTA arrive on it (the peer remotely).
// Every wait is bounded; a cluster barrier at start (barriers initialised) and at the end (nobody may
// exit while its partner can still touch its shared memory) brackets the kernel.
//
// Epilogue. Each of the four epilogue warps drains its 32 accumulator rows in chunks of 128 bytes per row
// (64 bf16 or 32 fp32 columns), writes a chunk into a 128B-swizzled 4 KiB staging buffer of its own (two per
// warp) and one lane hands it to TMA: a tiled store for bf16 / fp32 outputs, a tiled reduce-add for the
// "accumulate into an fp32 destination" mode, so the weight-gradient GEMMs never read their destination into
// the SM. TMA clips rows and columns beyond M and N. The older epilogue (each thread storing its own row with
// 16-byte stores, read-modify-write for the accumulate mode) is kept as a template variant. GEMMs of few tiles split K
// over several CTA pairs, which write slices of a workspace that a small kernel sums (pt_gemm_bf16_split).
//
// Fused epilogues (forward GEMMs X W^T with bf16 output only):
//   SwiGLU  W is the packed [gate; up] weight [2I, K]. The leader CTA loads 128 (64) gate rows, its partner the up rows of
//           the same indices, so accumulator columns 0..127 / 128..255 of a tile are gate / up pre-activations of the
//           same 128 hidden units. The epilogue stores both (the backward needs them) and silu(gate) * up to a second
//           output, which replaces the separate activation kernel and its pass over the [T, 2I] tensor.
//   RoPE    the output is the packed q|k|v activation; columns of the rotated heads (a prefix) are rotated in fp32 with
//           the cos/sin of the row's position before the single rounding to bf16 (NeoX pairing j <-> j + d/2, which
//           lies inside one 64-column chunk for d = 64 and inside one pair of chunks for d = 128).
// Epilogues that READ a second operand (the epilogue warps fetch its tile with TMA into their staging buffers while the
// accumulator is still being computed, combine it in place and hand the same buffers to the TMA store):
//   ADD         forward layout: D = A B^T + R with R a bf16 [M, N] tensor (the residual stream): the separate add kernel
//               and its pass over three [T, H] tensors disappear.
//   SWIGLU_BWD  dgrad layout (dY W): the accumulator is da = dL/d(silu(gate) * up) for 64 hidden units at a time; the
//               epilogue loads the matching gate and up pre-activations from the packed [M, 2I] tensor and stores
//               dgate = da * up * silu'(gate) and dup = da * silu(gate) into a packed [M, 2I] gradient. da itself is
//               never written, and the SwiGLU-backward kernel with its five passes over [T, I] is gone. This variant
//               runs with five operand stages because each epilogue warp needs four staging buffers.
#include "common.cuh"
#include "tensormap.cuh"

#include <algorithm>
#include <type_traits>

extern "C" void pt_count_launches(int n);
extern "C" int pt_chain_early();

namespace pt {
namespace gemm_pair {

constexpr int BM = 128;        // rows of A per CTA (256 per pair)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int MAX_STAGES = 8;
constexpr int A_BYTES = BM * BK * 2;        // 16 KiB
constexpr int NUM_THREADS = 192;
constexpr int TMEM_COLS = 512;
constexpr unsigned KERNEL_ID = 2;

enum OutMode { OUT_BF16 = 0, OUT_F32_ACC = 1, OUT_F32 = 2 };
enum Epilogue { EPI_NONE = 0, EPI_SWIGLU = 1, EPI_ROPE64 = 2, EPI_ROPE128 = 3, EPI_ADD = 4, EPI_SWIGLU_BWD = 5, EPI_CE = 6 };
// operand stages and staging buffers per epilogue warp of each variant (see the smem budget in launch())
// (128-column tiles: as many as fit. They are what GEMMs of few rows run with, whose k-blocks take the latency of a load from HBM divided by the
// stages. With that and B's prefetch to L2 below the forward pass of the 135M shape on 256 tokens went from 1,368 to 1,298 us. One stage less with fp32
// results: behind most of them comes the kernel that sums the parts of K, whose CTAs find no shared memory beside eight stages and so cannot
// wait next to the GEMM's: 512 x 1024 x 2048 in four parts 10.9 us with eight, 10.2 with seven; the pass takes 1,278 us with seven for all.)
__host__ __device__ constexpr int stages_of(int epi, int bn, bool f32 = false) {
  return bn != 128 ? 6 - (epi == EPI_SWIGLU_BWD) : epi == EPI_SWIGLU_BWD ? 6 : f32 ? 7 : 8;
}
__host__ __device__ constexpr int staging_bufs_of(int epi) { return epi == EPI_SWIGLU_BWD ? 4 : 2; }
// a stage holds BM x BK of A and bn / 2 x BK of B; four epilogue warps stage [32 rows][128 B] per buffer
// (MN-major operands come in boxes of 64 columns: 192-column tiles fetch 128 columns per CTA and use 96)
__host__ __device__ constexpr int b_bytes_of(int bn) { return (bn / 2 + 63) / 64 * 64 * BK * 2; }
__host__ __device__ constexpr int smem_bytes_of(int epi, int bn, bool f32 = false) {
  return stages_of(epi, bn, f32) * (A_BYTES + b_bytes_of(bn)) + 4 * staging_bufs_of(epi) * 4096 + 1024;
}

struct EpiArgs {
  int inter;              // SwiGLU: I (the weight has 2 I rows, the second output I columns)
  const float* cosT;      // RoPE: fp32 [S, d/2] tables
  const float* sinT;
  int seq;                // RoPE: row r is at position r % seq
  int rot_cols;           // RoPE: columns [0, rot_cols) are rotated (rotated heads x d)
  int early;              // what was written before this chain of launches: B and, of the SwiGLU backward, the second operand (pt_chain_begin)
  int group_m;            // tile numbering: rows of tiles per group (all epilogues)
  // K split into parts (fp32 outputs without a fused epilogue, pt_gemm_bf16_split): k-blocks per part, rows between the slices of
  // the destination, and which slice a part goes to (part >> slice_shift). Unsplit: one part with all k-blocks.
  int kb_per_part, slice_rows, slice_shift;
  // cross-entropy statistics (EPI_CE): per row and per 256-column tile the maximum and the sum of exp(logit - maximum)
  // of the ROUNDED logits go to ce_part[row * ce_tiles + n_blk]; the logit of the row's target column goes to ce_tgt[row]
  float2* ce_part;
  float* ce_tgt;
  const long long* ce_targets;
  long long ce_vocab_start;
  int ce_tiles;
  int ce_store;           // 0: statistics only, the logits are not written (loss without gradient)
};

struct Barriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t epi_load[4][2];    // per epilogue warp and set of buffers: the TMA loads of the second operand (ADD / SWIGLU_BWD)
  uint32_t tmem_base;
  int abort_flag;
};

// Tiles are numbered in groups of `group_m` rows of tiles, column by column inside a group, so that the CTA pairs that run
// at the same time (consecutive tile numbers) share few A row panels and few B column panels in L2.
__device__ __forceinline__ void tile_coords(int t, int num_m, int num_n, int group_m, int& m_blk, int& n_blk) {
  const int per_group = group_m * num_n;
  const int group = t / per_group;
  const int first_m = group * group_m;
  const int gsize = min(num_m - first_m, group_m);
  const int r = t - group * per_group;
  m_blk = first_m + r % gsize;
  n_blk = r / gsize;
}

__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// ask for a tile to be brought into L2
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y) : "memory");
}
// byte offset of 16-byte unit u of row r in a [rows][128 B] tile stored with the 128-byte swizzle
__device__ __forceinline__ uint32_t sw128_unit(int r, int u) { return (uint32_t)(r * 128 + ((u ^ (r & 7)) << 4)); }

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2E = 1.4426950408889634f;
// 1 / (1 + exp(-x)) of two values (x very negative: 1 / infinity = 0)
__device__ __forceinline__ uint64_t sigmoid2(uint64_t x) {
  const uint64_t y = mul2(x, pair_of(-LOG2E, -LOG2E));
  const uint64_t d = add2(pair_of(ex2_approx(lo_of(y)), ex2_approx(hi_of(y))), pair_of(1.f, 1.f));
  return pair_of(rcp_approx(lo_of(d)), rcp_approx(hi_of(d)));
}

// N is the number of output columns, except for EPI_SWIGLU where it is I (tiles pair BN / 2 gate with BN / 2 up columns).
template <bool A_MN, bool B_MN, int OUT_MODE, bool EPI_TMA, int EPI, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const __grid_constant__ CUtensorMap tma_d, const __grid_constant__ CUtensorMap tma_h,
                 void* __restrict__ Dptr, int M, int N, int K, long long ldd, KernelStatus* status, EpiArgs ea) {
  static_assert(EPI == EPI_NONE || (EPI_TMA && !A_MN && OUT_MODE == OUT_BF16 && B_MN == (EPI == EPI_SWIGLU_BWD)),
                "fused epilogues: bf16 output; forward layout, except the SwiGLU backward which rides on the dgrad layout");
  static_assert(BN == 256 || (BN == 128 && EPI_TMA && EPI != EPI_CE) ||
                    (BN == 192 && EPI_TMA && (EPI == EPI_NONE || EPI == EPI_ADD || EPI == EPI_SWIGLU_BWD)),
                "narrow tiles: the epilogues through TMA, but for the statistics; 192 columns: where 64-column chunks are independent");
  constexpr int BN_HALF = BN / 2;                 // columns of B per CTA
  constexpr int B_BYTES = b_bytes_of(BN), STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int LOAD_BYTES = A_BYTES + (B_MN ? B_BYTES : BN_HALF * BK * 2);      // what the loads of a stage bring
  constexpr int STAGES = stages_of(EPI, BN, OUT_MODE != OUT_BF16);
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  __shared__ Barriers bars;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * A_BYTES;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);      // (known to be the same in all lanes)
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();           // 0 = leader
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;
  const int num_m = (M + 2 * BM - 1) / (2 * BM);
  const int num_n = (EPI == EPI_SWIGLU) ? (N + BN_HALF - 1) / BN_HALF : (N + BN - 1) / BN;
  const int num_kb = (K + BK - 1) / BK;
  // Work units: every output tile, once per part of K (outermost, so that concurrently running units share operand panels as
  // before).
  constexpr bool PARTS = OUT_MODE != OUT_BF16 && EPI_TMA;
  const int tiles = num_m * num_n;
  const int kbs = PARTS ? ea.kb_per_part : num_kb;
  const int num_tiles = PARTS ? tiles * ((num_kb + kbs - 1) / kbs) : tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars.tmem_full[s], 1);
      mbar_init(&bars.tmem_empty[s], 8);    // 4 epilogue warps x 2 CTAs (used in the leader only)
    }
    if (EPI == EPI_ADD || EPI == EPI_SWIGLU_BWD)
      for (int q = 0; q < 8; ++q) mbar_init(&bars.epi_load[q >> 1][q & 1], 1);
    bars.abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    if (EPI_TMA) tma_prefetch_desc(&tma_d);
    if (EPI == EPI_SWIGLU || EPI == EPI_ADD || EPI == EPI_SWIGLU_BWD) tma_prefetch_desc(&tma_h);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars.tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  tcgen05_fence_after();
  const uint32_t tmem_base = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // This CTA's part of B. In a chain the first stages' travel under the predecessor's tail, the rest of the prologue's way: a small GEMM is
      // little more than the latency of its first loads, and weights come from HBM (forward of the 135M shape on 256 tokens, 120 of them: 1,418 us
      // a pass without, 1,368 with).
      auto load_b = [&](int st, int kb, int col0) {
        const uint32_t full_leader = mapa_u32(smem_u32(&bars.full[st]), 0);
        uint8_t* sb = smem_b + st * B_BYTES;
        if (!B_MN) {
          tma_load_2d_pair(sb, &tma_b, full_leader, kb * BK, col0);
        } else {
#pragma unroll
          for (int c = 0; c < B_BYTES / (BK * 128); ++c)
            tma_load_2d_pair(sb + c * (BK * 128), &tma_b, full_leader, col0 + c * 64, kb * BK);
        }
      };
      auto first_col = [&](int n_blk) {              // (SwiGLU: gate rows for the leader, the up rows of the same units for its partner)
        return (EPI == EPI_SWIGLU) ? n_blk * BN_HALF + (int)rank * ea.inter : n_blk * BN + (int)rank * BN_HALF;
      };
      int early = 0;
      if (ea.early && cluster_id < num_tiles) {
        int m_blk, n_blk;
        const int part = PARTS ? cluster_id / tiles : 0;
        tile_coords(cluster_id - part * tiles, num_m, num_n, ea.group_m, m_blk, n_blk);
        const int col0 = first_col(n_blk), kb0 = part * kbs;
        early = min(STAGES, min(num_kb - kb0, kbs));
        for (int i = 0; i < early; ++i) {
          if (rank == 0) mbar_expect_tx(&bars.full[i], 2 * LOAD_BYTES);
          load_b(i, kb0 + i, col0);
        }
        // one tile a pair: the rest of its B (of 2,048 rows at most) at least comes to L2
        if (num_tiles <= num_clusters)
          for (int kb = kb0 + early; kb < min(num_kb, min(kb0 + kbs, kb0 + 32)); ++kb) {
            if (!B_MN) {
              tma_prefetch_2d(&tma_b, kb * BK, col0);
            } else {
#pragma unroll
              for (int c = 0; c < B_BYTES / (BK * 128); ++c) tma_prefetch_2d(&tma_b, col0 + c * 64, kb * BK);
            }
          }
      }
      pdl_wait();                    // what the predecessor wrote is needed from here on
      for (int t = cluster_id; t < num_tiles && ok; t += num_clusters) {
        int m_blk, n_blk;
        const int part = PARTS ? t / tiles : 0;
        tile_coords(t - part * tiles, num_m, num_n, ea.group_m, m_blk, n_blk);
        const int row0 = m_blk * 2 * BM + (int)rank * BM;          // this CTA's rows of A
        const int col0 = first_col(n_blk);
        const int kb_end = min(num_kb, (part + 1) * kbs);
        for (int kb = part * kbs; kb < kb_end; ++kb) {
          if (!mbar_wait(&bars.empty[stage], phase ^ 1, abort_flag)) {
            report_error(status, KERNEL_ID, 1);
            ok = false;
            break;
          }
          // (A before B: with B first, 192-column tiles of an MN-major B took 2 to 4 % longer, 8192 x 576 x 3072 30.7 -> 31.8 us)
          const uint32_t full_leader = mapa_u32(smem_u32(&bars.full[stage]), 0);
          if (rank == 0 && early == 0) mbar_expect_tx(&bars.full[stage], 2 * LOAD_BYTES);
          uint8_t* sa = smem_a + stage * A_BYTES;
          if (!A_MN) {
            tma_load_2d_pair(sa, &tma_a, full_leader, kb * BK, row0);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c)
              tma_load_2d_pair(sa + c * (BK * 128), &tma_a, full_leader, row0 + c * 64, kb * BK);
          }
          if (early > 0) --early;
          else load_b(stage, kb, col0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      const uint64_t a_base = make_smem_desc_sw128(smem_u32(smem_a), A_MN ? BK * 128 : 16, 1024);
      const uint64_t b_base = make_smem_desc_sw128(smem_u32(smem_b), B_MN ? BK * 128 : 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int local = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += num_clusters, ++local) {
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        if (!mbar_wait(&bars.tmem_empty[acc], acc_phase ^ 1, abort_flag)) {
          report_error(status, KERNEL_ID, 2);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        const int part = PARTS ? t / tiles : 0;
        const int num_here = min(num_kb - part * kbs, kbs);
        for (int kb = 0; kb < num_here; ++kb) {
          if (!mbar_wait(&bars.full[stage], phase, abort_flag)) {
            report_error(status, KERNEL_ID, 3);
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint64_t a_st = smem_desc_advance(a_base, stage * A_BYTES), b_st = smem_desc_advance(b_base, stage * B_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(d_tmem, smem_desc_advance(a_st, k * UMMA_K * (A_MN ? 128 : 2)), smem_desc_advance(b_st, k * UMMA_K * (B_MN ? 128 : 2)),
                           idesc, (kb > 0 || k > 0) ? 1u : 0u);
          const uint32_t e = smem_u32(&bars.empty[stage]);
          umma_commit_pair(mapa_u32(e, 0));
          umma_commit_pair(mapa_u32(e, 1));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) {
          const uint32_t f = smem_u32(&bars.tmem_full[acc]);
          umma_commit_pair(mapa_u32(f, 0));
          umma_commit_pair(mapa_u32(f, 1));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5 of both CTAs)
    const int quarter = warp & 3;
    bool ok = true;
    int local = 0;
    if (EPI != EPI_SWIGLU_BWD) pdl_wait();
    if constexpr (EPI == EPI_ADD || EPI == EPI_SWIGLU_BWD) {
      // ---- epilogues with a second operand: chunk c of a tile = 64 accumulator columns of this warp's 32 rows
      constexpr int PER = EPI == EPI_SWIGLU_BWD ? 2 : 1;      // buffers of a chunk: the residual, or (gate, up)
      constexpr int SETS = staging_bufs_of(EPI) / PER;
      constexpr int NCH = BN / 64;
      uint8_t* stg = smem + STAGES * STAGE_BYTES + quarter * (SETS * PER * 4096);
      // The operand of chunk (load_t, load_c), SETS - 1 chunks ahead of the one that is combined, goes to set load_set; load_row and
      // load_col are its place in the output.
      int load_t = cluster_id, load_c = 0, load_set = 0, load_row = 0, load_col = 0;
      auto issue_load = [&]() {
        if (load_t < num_tiles) {
          if (load_c == 0) {
            int m_blk, n_blk;
            tile_coords(load_t, num_m, num_n, ea.group_m, m_blk, n_blk);
            load_row = m_blk * 2 * BM + (int)rank * BM + quarter * 32;
            load_col = n_blk * BN;
          }
          if (elect_one()) {
            tma_store_wait_read<0>();        // the store of the chunk before, which used this set
            uint8_t* b0 = stg + load_set * PER * 4096;
            uint64_t* bar = &bars.epi_load[quarter][load_set];
            if (load_row < M && load_col < N) {
              mbar_expect_tx(bar, PER * 4096);
              tma_load_2d(b0, &tma_h, bar, load_col, load_row);
              if (EPI == EPI_SWIGLU_BWD) tma_load_2d(b0 + 4096, &tma_h, bar, ea.inter + load_col, load_row);
            } else {
              mbar_arrive(bar);                                   // nothing to fetch: complete the phase by hand
            }
          }
        }
        load_set = load_set + 1 == SETS ? 0 : load_set + 1;
        load_col += 64;
        if (++load_c == NCH) {
          load_c = 0;
          load_t += num_clusters;
        }
      };
      if (EPI == EPI_SWIGLU_BWD && !ea.early) pdl_wait();
      for (int i = 0; i + 1 < SETS; ++i) issue_load();
      if (EPI == EPI_SWIGLU_BWD && ea.early) pdl_wait();
      int set = 0;
      uint32_t ld_phase = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += num_clusters, ++local) {
        int m_blk, n_blk;
        tile_coords(t, num_m, num_n, ea.group_m, m_blk, n_blk);
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        if (!mbar_wait(&bars.tmem_full[acc], acc_phase, abort_flag)) {
          if (lane == 0) report_error(status, KERNEL_ID, 4);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const int row0 = m_blk * 2 * BM + (int)rank * BM + quarter * 32;
        const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
#pragma unroll 1
        for (int c = 0; c < NCH; ++c) {
          uint32_t v[64];
          tmem_ld_32x32b_x32_at(t_row + c * 64, v, 0);
          tmem_ld_32x32b_x32_at(t_row + c * 64 + 32, v, 32);
          if (!mbar_wait(&bars.epi_load[quarter][set], ld_phase, abort_flag)) {
            if (lane == 0) report_error(status, KERNEL_ID, 5);
            ok = false;
            break;
          }
          uint8_t* b0 = stg + set * PER * 4096;
          if (++set == SETS) {
            set = 0;
            ld_phase ^= 1;
          }
          const int col0 = n_blk * BN + c * 64;
          // All of the chunk's reads come first: the compiler may not move a read of shared memory before a write to it, so that eight
          // rounds of read, combine, write were a chain of eight latencies. With that, packed arithmetic and a reciprocal instead of a
          // quotient, a SwiGLU-backward chunk takes 1,490 cycles to combine instead of 2,450 (its exponentials and reciprocals alone
          // 1,024): 8192 x 1536 x 576: 36 -> 32 us, 4096 x 2560 x 960: 38 -> 34.
          uint4 q0[8], q1[PER == 2 ? 8 : 1];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            q0[u] = *reinterpret_cast<const uint4*>(b0 + sw128_unit(lane, u));
            if constexpr (PER == 2) q1[u] = *reinterpret_cast<const uint4*>(b0 + 4096 + sw128_unit(lane, u));
          }
          issue_load();
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            uint32_t* w0 = reinterpret_cast<uint32_t*>(&q0[u]);
            if constexpr (EPI == EPI_ADD) {
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[e]));
                w0[e] = pack_bf16(__uint_as_float(v[8 * u + 2 * e]) + r.x, __uint_as_float(v[8 * u + 2 * e + 1]) + r.y);
              }
            } else {
              uint32_t* w1 = reinterpret_cast<uint32_t*>(&q1[PER == 2 ? u : 0]);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[e]));
                const float2 up = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w1[e]));
                const uint64_t g2 = pair_of(g.x, g.y), one = pair_of(1.f, 1.f), sg = sigmoid2(g2);
                const uint64_t da = pair_of(__uint_as_float(v[8 * u + 2 * e]), __uint_as_float(v[8 * u + 2 * e + 1]));
                const uint64_t slope = fma2(g2, fma2(sg, pair_of(-1.f, -1.f), one), one);              // 1 + g (1 - s)
                // (da s in common would save a product, 0 to 1.5 %, 4096 x 2560 x 960 40.7 -> 40.0 us, but where s is next to the smallest
                // normal number it flushes to zero what `up` or the gate would have brought back)
                const uint64_t dg = mul2(mul2(da, pair_of(up.x, up.y)), mul2(sg, slope)), du = mul2(mul2(da, g2), sg);
                w0[e] = pack_bf16(lo_of(dg), hi_of(dg));
                w1[e] = pack_bf16(lo_of(du), hi_of(du));
              }
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            *reinterpret_cast<uint4*>(b0 + sw128_unit(lane, u)) = q0[u];
            if constexpr (PER == 2) *reinterpret_cast<uint4*>(b0 + 4096 + sw128_unit(lane, u)) = q1[u];
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (row0 < M && col0 < N) {
              tma_store_2d(&tma_d, b0, col0, row0);
              if (EPI == EPI_SWIGLU_BWD) tma_store_2d(&tma_d, b0 + 4096, ea.inter + col0, row0);
            }
            tma_store_commit();
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bars.tmem_empty[acc]), 0));
      }
      if (elect_one()) tma_store_wait<0>();
    } else if constexpr (EPI != EPI_NONE) {
      uint8_t* stg = smem + STAGES * STAGE_BYTES + quarter * (2 * 4096);
      int buf = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += num_clusters, ++local) {
        int m_blk, n_blk;
        tile_coords(t, num_m, num_n, ea.group_m, m_blk, n_blk);
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        if (EPI == EPI_SWIGLU || EPI == EPI_CE) {              // (RoPE loads its tables first)
          if (!mbar_wait(&bars.tmem_full[acc], acc_phase, abort_flag)) {
            if (lane == 0) report_error(status, KERNEL_ID, 4);
            ok = false;
            break;
          }
          tcgen05_fence_after();
        }
        const int row0 = m_blk * 2 * BM + (int)rank * BM + quarter * 32;      // first of this warp's 32 rows
        const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
        // 64 bf16 of this lane's row (packed in q[32]) -> swizzled staging buffer -> TMA store at (col0, row0)
        auto stage_store = [&](const uint32_t (&q)[32], const CUtensorMap* map, int col0) {
          if (elect_one()) tma_store_wait_read<1>();        // the store issued two chunks ago has finished reading this buffer
          __syncwarp();
          uint8_t* dst = stg + buf * 4096;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<uint4*>(dst + sw128_unit(lane, u)) = make_uint4(q[4 * u], q[4 * u + 1], q[4 * u + 2], q[4 * u + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (row0 < M) tma_store_2d(map, dst, col0, row0);
            tma_store_commit();
          }
          buf ^= 1;
        };
        if constexpr (EPI == EPI_SWIGLU) {
#pragma unroll 1
          for (int c = 0; c < BN_HALF / 64; ++c) {
            uint32_t g[64], u[64];
            tmem_ld_32x32b_x32_at(t_row + c * 64, g, 0);
            tmem_ld_32x32b_x32_at(t_row + c * 64 + 32, g, 32);
            tmem_ld_32x32b_x32_at(t_row + BN_HALF + c * 64, u, 0);
            tmem_ld_32x32b_x32_at(t_row + BN_HALF + c * 64 + 32, u, 32);
            tmem_ld_wait();
            uint32_t qg[32], qu[32], qh[32];
#pragma unroll
            for (int e = 0; e < 64; e += 2) {
              qg[e >> 1] = pack_bf16(__uint_as_float(g[e]), __uint_as_float(g[e + 1]));
              qu[e >> 1] = pack_bf16(__uint_as_float(u[e]), __uint_as_float(u[e + 1]));
              // the activation is computed from the ROUNDED pre-activations, which is what the backward will read
              const float2 gr = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qg[e >> 1]));
              const float2 ur = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qu[e >> 1]));
              const uint64_t g2 = pair_of(gr.x, gr.y), h = mul2(mul2(g2, sigmoid2(g2)), pair_of(ur.x, ur.y));
              qh[e >> 1] = pack_bf16(lo_of(h), hi_of(h));
            }
            const int unit0 = n_blk * BN_HALF + c * 64;
            stage_store(qg, &tma_d, unit0);
            stage_store(qu, &tma_d, ea.inter + unit0);
            stage_store(qh, &tma_h, unit0);
          }
        } else if constexpr (EPI == EPI_CE) {
          // LM-head logits tile: store it, and keep per row the running maximum and the sum of exponentials over the
          // tile's 256 columns (online, chunk by chunk) of the values as stored (bf16), plus the target's logit
          const int row = row0 + lane;
          const long long tcol = (row < M ? ea.ce_targets[row] : -1) - ea.ce_vocab_start;     // column of the target in this shard
          float m_run = -INFINITY, s_run = 0.f;
#pragma unroll 1
          for (int c = 0; c < BN / 64; ++c) {
            uint32_t v[64];
            tmem_ld_32x32b_x32_at(t_row + c * 64, v, 0);
            tmem_ld_32x32b_x32_at(t_row + c * 64 + 32, v, 32);
            tmem_ld_wait();
            const int col0 = n_blk * BN + c * 64;
            uint32_t q[32];
            float cm[2] = {-INFINITY, -INFINITY};
            // (Columns are tested against N only in the last, partial chunk: a test per column is as much work as its exponential. With
            // two running maxima and packed sums: 2048 x 49152 x 576: 124 -> 116 us, x 960: 143 -> 136; from K = 2048 on the MMAs hide it.)
            const bool whole = col0 + 64 <= N;
#pragma unroll
            for (int e = 0; e < 64; e += 2) {
              q[e >> 1] = pack_bf16(__uint_as_float(v[e]), __uint_as_float(v[e + 1]));
              const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q[e >> 1]));
              v[e] = __float_as_uint(r.x);
              v[e + 1] = __float_as_uint(r.y);
            }
            if (!whole) {
#pragma unroll
              for (int e = 0; e < 64; ++e) v[e] = col0 + e < N ? v[e] : __float_as_uint(-INFINITY);
            }
#pragma unroll
            for (int e = 0; e < 64; ++e) cm[e & 1] = fmaxf(cm[e & 1], __uint_as_float(v[e]));
            if (col0 < N) {
              const float nm = fmaxf(m_run, fmaxf(cm[0], cm[1]));
              uint64_t sums[2] = {0, 0};
              const uint64_t neg_m = pair_of(-nm, -nm), log2e = pair_of(LOG2E, LOG2E);
#pragma unroll
              for (int e = 0; e < 64; e += 2) {
                const uint64_t d = mul2(add2(pair_of(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), neg_m), log2e);
                sums[(e >> 1) & 1] = add2(sums[(e >> 1) & 1], pair_of(ex2_approx(lo_of(d)), ex2_approx(hi_of(d))));
              }
              const float acc = (lo_of(sums[0]) + hi_of(sums[0])) + (lo_of(sums[1]) + hi_of(sums[1]));
              s_run = s_run * ex2_approx((m_run - nm) * LOG2E) + acc;
              m_run = nm;
              if (tcol >= col0 && tcol < col0 + 64 && tcol < N && row < M) {     // (a target beyond N belongs to another shard)
                float tv = 0.f;
#pragma unroll
                for (int e = 0; e < 64; ++e) tv = ((long long)(col0 + e) == tcol) ? __uint_as_float(v[e]) : tv;
                ea.ce_tgt[row] = tv;
              }
              if (ea.ce_store) stage_store(q, &tma_d, col0);
            }
          }
          if (row < M) ea.ce_part[(long long)row * ea.ce_tiles + n_blk] = make_float2(m_run, s_run);
        } else {
          constexpr int HD = (EPI == EPI_ROPE64) ? 64 : 128;          // head dim = columns handled per iteration
          const int row = row0 + lane;
          const int pos = (row < M ? row : 0) % ea.seq;
          const float* cos_row = ea.cosT + (long long)pos * (HD / 2);
          const float* sin_row = ea.sinT + (long long)pos * (HD / 2);
          // Head dim 64: a row's tables (32 cosines, 32 sines) are the same for all heads of the tile, so a lane reads them once per tile,
          // before it waits for the accumulator. Every lane reads another row of the table, 32 cache lines per load: read again for each
          // head that was 4.3 us a tile (8192 x 9472 x 576: 126 us, now 82; 8192 x 960 x 576: 21 -> 14.5; 4096 x 1600 x 960: 21 -> 16.5).
          // Head dim 128 has no registers for its 128 values, and its models' reductions are long enough to hide the loads.
          float cs64[EPI == EPI_ROPE64 ? 32 : 1], sn64[EPI == EPI_ROPE64 ? 32 : 1];
          if constexpr (EPI == EPI_ROPE64) {
            if (n_blk * BN < ea.rot_cols) {
#pragma unroll
              for (int jj = 0; jj < 32; jj += 4) {
                const float4 cs = __ldg(reinterpret_cast<const float4*>(cos_row + jj));
                const float4 sn = __ldg(reinterpret_cast<const float4*>(sin_row + jj));
                cs64[jj] = cs.x; cs64[jj + 1] = cs.y; cs64[jj + 2] = cs.z; cs64[jj + 3] = cs.w;
                sn64[jj] = sn.x; sn64[jj + 1] = sn.y; sn64[jj + 2] = sn.z; sn64[jj + 3] = sn.w;
              }
            }
          }
          if (!mbar_wait(&bars.tmem_full[acc], acc_phase, abort_flag)) {
            if (lane == 0) report_error(status, KERNEL_ID, 4);
            ok = false;
            break;
          }
          tcgen05_fence_after();
#pragma unroll 1
          for (int c = 0; c < BN / HD; ++c) {
            uint32_t v[HD];
#pragma unroll
            for (int h = 0; h < HD / 32; ++h) tmem_ld_32x32b_x32_at(t_row + c * HD + h * 32, v, h * 32);
            tmem_ld_wait();
            const int col0 = n_blk * BN + c * HD;
            if (col0 < ea.rot_cols) {
#pragma unroll
              for (int jj = 0; jj < HD / 2; jj += 4) {
                float csv[4], snv[4];
                if constexpr (EPI == EPI_ROPE64) {
#pragma unroll
                  for (int i = 0; i < 4; ++i) { csv[i] = cs64[jj + i]; snv[i] = sn64[jj + i]; }
                } else {
                  const float4 cs = __ldg(reinterpret_cast<const float4*>(cos_row + jj));
                  const float4 sn = __ldg(reinterpret_cast<const float4*>(sin_row + jj));
                  csv[0] = cs.x; csv[1] = cs.y; csv[2] = cs.z; csv[3] = cs.w;
                  snv[0] = sn.x; snv[1] = sn.y; snv[2] = sn.z; snv[3] = sn.w;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const float a = __uint_as_float(v[jj + i]), b = __uint_as_float(v[jj + i + HD / 2]);
                  v[jj + i] = __float_as_uint(a * csv[i] - b * snv[i]);
                  v[jj + i + HD / 2] = __float_as_uint(b * csv[i] + a * snv[i]);
                }
              }
            }
#pragma unroll
            for (int part = 0; part < HD / 64; ++part) {
              uint32_t q[32];
#pragma unroll
              for (int e = 0; e < 64; e += 2)
                q[e >> 1] = pack_bf16(__uint_as_float(v[part * 64 + e]), __uint_as_float(v[part * 64 + e + 1]));
              if (col0 + part * 64 < N) stage_store(q, &tma_d, col0 + part * 64);
            }
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bars.tmem_empty[acc]), 0));
      }
      if (elect_one()) tma_store_wait<0>();
    } else if constexpr (EPI_TMA) {
      constexpr int CH_COLS = (OUT_MODE == OUT_BF16) ? 64 : 32;      // columns per 128-byte chunk row

      constexpr int NCH = BN / CH_COLS;
      constexpr int CH_REGS = (OUT_MODE == OUT_BF16) ? 64 : 32;      // accumulator registers per chunk
      uint8_t* stg = smem + STAGES * STAGE_BYTES + quarter * (2 * 4096);
      int buf = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += num_clusters, ++local) {
        int m_blk, n_blk;
        const int part = PARTS ? t / tiles : 0;
        tile_coords(t - part * tiles, num_m, num_n, ea.group_m, m_blk, n_blk);
        const int slice_row0 = PARTS ? (part >> ea.slice_shift) * ea.slice_rows : 0;
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        if (!mbar_wait(&bars.tmem_full[acc], acc_phase, abort_flag)) {
          if (lane == 0) report_error(status, KERNEL_ID, 4);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const int row0 = m_blk * 2 * BM + (int)rank * BM + quarter * 32;      // first of this warp's 32 rows
        const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
        uint32_t r[2][CH_REGS];
        auto load_chunk = [&](int c, uint32_t (&dst)[CH_REGS]) {
#pragma unroll
          for (int h = 0; h < CH_REGS / 32; ++h) tmem_ld_32x32b_x32_at(t_row + c * CH_COLS + h * 32, dst, h * 32);
        };
        load_chunk(0, r[0]);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          tmem_ld_wait();
          if (c + 1 < NCH) load_chunk(c + 1, r[(c + 1) & 1]);
          const uint32_t (&v)[CH_REGS] = r[c & 1];
          if (elect_one()) tma_store_wait_read<1>();        // the store issued two chunks ago has finished reading this buffer
          __syncwarp();
          uint8_t* dst = stg + buf * 4096;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            uint4 q;
            if (OUT_MODE == OUT_BF16) {
              q.x = pack_bf16(__uint_as_float(v[8 * u + 0]), __uint_as_float(v[8 * u + 1]));
              q.y = pack_bf16(__uint_as_float(v[8 * u + 2]), __uint_as_float(v[8 * u + 3]));
              q.z = pack_bf16(__uint_as_float(v[8 * u + 4]), __uint_as_float(v[8 * u + 5]));
              q.w = pack_bf16(__uint_as_float(v[8 * u + 6]), __uint_as_float(v[8 * u + 7]));
            } else {
              q = make_uint4(v[(4 * u + 0) % CH_REGS], v[(4 * u + 1) % CH_REGS], v[(4 * u + 2) % CH_REGS], v[(4 * u + 3) % CH_REGS]);
            }
            *reinterpret_cast<uint4*>(dst + sw128_unit(lane, u)) = q;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            const int col0 = n_blk * BN + c * CH_COLS;
            if (row0 < M && col0 < N) {
              if (OUT_MODE == OUT_F32_ACC) tma_reduce_add_2d(&tma_d, dst, col0, slice_row0 + row0);
              else tma_store_2d(&tma_d, dst, col0, slice_row0 + row0);
            }
            tma_store_commit();
          }
          buf ^= 1;
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bars.tmem_empty[acc]), 0));
      }
      if (elect_one()) tma_store_wait<0>();
    } else {
    for (int t = cluster_id; t < num_tiles && ok; t += num_clusters, ++local) {
      int m_blk, n_blk;
      tile_coords(t, num_m, num_n, ea.group_m, m_blk, n_blk);
      const int acc = local & 1;
      const uint32_t acc_phase = (local >> 1) & 1;
      if (!mbar_wait(&bars.tmem_full[acc], acc_phase, abort_flag)) {
        if (lane == 0) report_error(status, KERNEL_ID, 4);
        ok = false;
        break;
      }
      tcgen05_fence_after();
      const int row = m_blk * 2 * BM + (int)rank * BM + quarter * 32 + lane;
      const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
      // Software-pipelined drain of the accumulator: the TMEM load of chunk c+1 is in flight while chunk c is stored.
      auto store_chunk = [&](const uint32_t (&r)[32], int c) {
        const int col0 = n_blk * BN + c * 32;
        if (row < M && col0 < N) {
          if (OUT_MODE == OUT_BF16) {
            __nv_bfloat16* drow = reinterpret_cast<__nv_bfloat16*>(Dptr) + (long long)row * ldd + col0;
            if (col0 + 32 <= N) {
              uint4* d4 = reinterpret_cast<uint4*>(drow);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint4 v;
                v.x = pack_bf16(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1]));
                v.y = pack_bf16(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
                v.z = pack_bf16(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
                v.w = pack_bf16(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
                d4[j] = v;
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < N; ++j) drow[j] = __float2bfloat16(__uint_as_float(r[j]));
            }
          } else {
            float* drow = reinterpret_cast<float*>(Dptr) + (long long)row * ldd + col0;
            if (col0 + 32 <= N) {
              float4* d4 = reinterpret_cast<float4*>(drow);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float4 v = make_float4(__uint_as_float(r[4 * j + 0]), __uint_as_float(r[4 * j + 1]),
                                       __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                if (OUT_MODE == OUT_F32_ACC) {
                  const float4 o = d4[j];
                  v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
                }
                d4[j] = v;
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < N; ++j) {
                float v = __uint_as_float(r[j]);
                if (OUT_MODE == OUT_F32_ACC) v += drow[j];
                drow[j] = v;
              }
            }
          }
        }
            };
      {
        uint32_t ra[32], rb[32];
        tmem_ld_32x32b_x32(t_row, ra);
#pragma unroll
        for (int c = 0; c < BN / 32; c += 2) {
          tmem_ld_wait();
          tmem_ld_32x32b_x32(t_row + (c + 1) * 32, rb);
          store_chunk(ra, c);
          tmem_ld_wait();
          if (c + 2 < BN / 32) tmem_ld_32x32b_x32(t_row + (c + 2) * 32, ra);
          store_chunk(rb, c + 1);
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bars.tmem_empty[acc]), 0));
    }
    }
  }

  // ------------------------------------------------------------------ teardown
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// GEMM whose K is shared by the two CTA pairs of one cluster: each sums its half of K for a 256 x 128 tile in tensor memory, sends the 64 columns
// that are the other's through distributed shared memory (fp32, in the place of the operand stages), adds what it is sent to its own 64 and
// stores these (with the residual). One tile per cluster.
// What it is for: few output tiles, where a tile's k-blocks, one after the other, are all that the time consists of. The same split through an
// fp32 workspace costs two launches more (clearing, summing) and two passes over the slices. Measured whole or through a workspace / this way (us,
// operands not in L2): with residual 256 x 960 x 2560: 17.4 / 14.4; 512 x 2048 x 8192: 29.7 / 26.7; input gradient 256 x 2048 x 3072: 19.5 / 16.4;
// 384 x 2048 x 6144: 27.7 / 22.4. Clusters of four pairs and tiles of 256 columns were slower at all but one of 240 shapes (512 x 2048 x 8192: 45.1, 34.7).
struct ClusterArgs {
  int kb_per_part, num_m, early;
};
struct ClusterBarriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t tmem_full;
  uint64_t epi_load[4];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int CLUSTER_BN = 128, CLUSTER_PARTS = 2;

template <bool B_MN, bool ADD>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ CUtensorMap tma_d,
                    const __grid_constant__ CUtensorMap tma_h, int M, int N, int K, KernelStatus* status, ClusterArgs ca) {
  constexpr int BN = CLUSTER_BN, BN_HALF = BN / 2, B_BYTES = b_bytes_of(BN), STAGE_BYTES = A_BYTES + B_BYTES, STAGES = stages_of(EPI_NONE, BN);
  constexpr int LOAD_BYTES = A_BYTES + (B_MN ? B_BYTES : BN_HALF * BK * 2);
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  __shared__ ClusterBarriers bars;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + STAGES * A_BYTES;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), pair = crank >> 1, rank = crank & 1, leader = crank & ~1u;
  const int tile = (int)(blockIdx.x / (2 * CLUSTER_PARTS)), m_blk = tile % ca.num_m, n_blk = tile / ca.num_m;
  const int num_kb = (K + BK - 1) / BK, kb0 = (int)pair * ca.kb_per_part, kbs = min(num_kb - kb0, ca.kb_per_part);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    mbar_init(&bars.tmem_full, 1);
    for (int q = 0; q < 4; ++q) mbar_init(&bars.epi_load[q], 1);
    bars.abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    tma_prefetch_desc(&tma_d);
    if (ADD) tma_prefetch_desc(&tma_h);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars.tmem_base, BN);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  tcgen05_fence_after();
  const uint32_t tmem_base = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;
  const int quarter = warp & 3;
  const int row0 = m_blk * 2 * BM + (int)rank * BM + quarter * 32;
  const uint32_t t_row = tmem_base + (uint32_t(quarter * 32) << 16);
  uint8_t* const stg = smem + STAGES * STAGE_BYTES + quarter * 4096;
  const int own0 = n_blk * BN + (int)pair * 64, other0 = n_blk * BN + (int)(pair ^ 1) * 64;      // columns this pair stores; those it sends
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (B ahead of the predecessor as in gemm_pair_kernel)
    if (elect_one()) {
      const int arow0 = m_blk * 2 * BM + (int)rank * BM, col0 = n_blk * BN + (int)rank * BN_HALF;
      auto load_b = [&](int st, int kb) {
        const uint32_t full_leader = mapa_u32(smem_u32(&bars.full[st]), leader);
        if (rank == 0) mbar_expect_tx(&bars.full[st], 2 * LOAD_BYTES);
        uint8_t* sb = smem_b + st * B_BYTES;
        if (!B_MN) {
          tma_load_2d_pair(sb, &tma_b, full_leader, kb * BK, col0);
        } else {
#pragma unroll
          for (int c = 0; c < B_BYTES / (BK * 128); ++c)
            tma_load_2d_pair(sb + c * (BK * 128), &tma_b, full_leader, col0 + c * 64, kb * BK);
        }
      };
      const int early = ca.early ? min(STAGES, kbs) : 0;
      for (int i = 0; i < early; ++i) load_b(i, kb0 + i);
      pdl_wait();
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < kbs; ++i) {
        if (!mbar_wait(&bars.empty[stage], phase ^ 1, abort_flag)) {
          report_error(status, KERNEL_ID, 11);
          break;
        }
        if (i >= early) load_b(stage, kb0 + i);
        tma_load_2d_pair(smem_a + stage * A_BYTES, &tma_a, mapa_u32(smem_u32(&bars.full[stage]), leader), (kb0 + i) * BK, arow0);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA of each pair)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, false, B_MN);
      const uint64_t a_base = make_smem_desc_sw128(smem_u32(smem_a), 16, 1024);
      const uint64_t b_base = make_smem_desc_sw128(smem_u32(smem_b), B_MN ? BK * 128 : 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      bool fine = true;
      for (int i = 0; i < kbs; ++i) {
        if (!mbar_wait(&bars.full[stage], phase, abort_flag)) {
          report_error(status, KERNEL_ID, 13);
          fine = false;
          break;
        }
        tcgen05_fence_after();
        const uint64_t a_st = smem_desc_advance(a_base, stage * A_BYTES), b_st = smem_desc_advance(b_base, stage * B_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_bf16_pair(tmem_base, smem_desc_advance(a_st, k * UMMA_K * 2), smem_desc_advance(b_st, k * UMMA_K * (B_MN ? 128 : 2)), idesc,
                         (i > 0 || k > 0) ? 1u : 0u);
        const uint32_t e = smem_u32(&bars.empty[stage]);
        umma_commit_pair(mapa_u32(e, leader));
        umma_commit_pair(mapa_u32(e, leader + 1));
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (fine) {
        const uint32_t f = smem_u32(&bars.tmem_full);
        umma_commit_pair(mapa_u32(f, leader));
        umma_commit_pair(mapa_u32(f, leader + 1));
      }
    }
  } else {
    pdl_wait();
    if (ADD && own0 < N && row0 < M && elect_one()) {
      mbar_expect_tx(&bars.epi_load[quarter], 4096);
      tma_load_2d(stg, &tma_h, &bars.epi_load[quarter], own0, row0);
    }
    if (!mbar_wait(&bars.tmem_full, 0, abort_flag)) {
      if (lane == 0) report_error(status, KERNEL_ID, 14);
      ok = false;
    }
    tcgen05_fence_after();
  }
  // All MMAs of the cluster are done: the stages may take the sums.
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (warp >= 2 && ok && other0 < N) {
    uint32_t v[64];
    tmem_ld_32x32b_x32_at(t_row + (pair ^ 1) * 64, v, 0);
    tmem_ld_32x32b_x32_at(t_row + (pair ^ 1) * 64 + 32, v, 32);
    tmem_ld_wait();
    // [16 quads of columns][128 rows][4 floats]
    const uint32_t to = mapa_u32(smem_u32(smem), (pair ^ 1) * 2 + rank) + (quarter * 32 + lane) * 16;
#pragma unroll
    for (int u = 0; u < 16; ++u)
      asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + u * 2048), "r"(v[4 * u]), "r"(v[4 * u + 1]), "r"(v[4 * u + 2]),
                   "r"(v[4 * u + 3])
                   : "memory");
  }
  uint32_t v[64];
  if (warp >= 2 && ok) {                       // its own columns, while the others' are on the way
    tmem_ld_32x32b_x32_at(t_row + pair * 64, v, 0);
    tmem_ld_32x32b_x32_at(t_row + pair * 64 + 32, v, 32);
    tmem_ld_wait();
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (ADD && warp >= 2 && ok && own0 < N && row0 < M && !mbar_wait(&bars.epi_load[quarter], 0, abort_flag)) {
    if (lane == 0) report_error(status, KERNEL_ID, 15);
    ok = false;
  }
  if (warp >= 2 && ok && own0 < N && row0 < M) {
    const float4* sent = reinterpret_cast<const float4*>(smem) + quarter * 32 + lane;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      uint4* const at = reinterpret_cast<uint4*>(stg + sw128_unit(lane, u));
      const uint4 r = ADD ? *at : make_uint4(0, 0, 0, 0);
      const uint32_t res[4] = {r.x, r.y, r.z, r.w};
      const float4 lo = sent[2 * u * 128], hi = sent[(2 * u + 1) * 128];
      const float add[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float a = __uint_as_float(v[8 * u + 2 * e]) + add[2 * e], b = __uint_as_float(v[8 * u + 2 * e + 1]) + add[2 * e + 1];
        if (ADD) {
          const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&res[e]));
          a += h.x;
          b += h.y;
        }
        w[e] = pack_bf16(a, b);
      }
      *at = make_uint4(w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (elect_one()) {
      tma_store_2d(&tma_d, stg, own0, row0);
      tma_store_commit();
      tma_store_wait<0>();
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, BN);
  }
}

static int g_group_m = 8;   // rows of 256-row tiles per group; measured on the model's shapes: 8 and 16 beat 4 by ~1 %, 1 is worst

// K-split GEMMs keep their parts in slices of an fp32 workspace: cleared before where two parts add to a slice, summed after in the
// order of the slices.
__global__ void __launch_bounds__(256) clear_f32_kernel(float4* __restrict__ x, long long n4) {
  pdl_enter();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < n4) x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// out[r, c] = sum over the slices (+ res[r, c]) (bf16), or out[r, c] += that sum (fp32, one atomic per element as the unsplit
// epilogue's reduce-add). Bound by the workspace's bytes, which lie in L2; four columns per thread.
template <bool TO_BF16, bool ADD>
__global__ void __launch_bounds__(256) sum_slices_kernel(const float* __restrict__ ws, int slices, long long slice_elems, void* __restrict__ out,
                                                         int rows, int cols, int ws_cols, long long ldd,
                                                         const __nv_bfloat16* __restrict__ res, long long ldr) {
  pdl_enter();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const int quads = ws_cols / 4;
  const long long r = i / quads;
  const int c = (int)(i - r * quads) * 4;
  if (r >= rows) return;
  const float* src = ws + r * ws_cols + c;
  float4 v = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
  for (int k = 1; k < slices; ++k) {
    const float4 u = *reinterpret_cast<const float4*>(src + k * slice_elems);
    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
  }
  if (ADD) {
    const uint2 q = *reinterpret_cast<const uint2*>(res + r * ldr + c);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.y));
    v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
  }
  if (TO_BF16) {
    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + r * ldd + c) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  } else {
    float* dst = reinterpret_cast<float*>(out) + r * ldd + c;
    if (c + 4 <= cols) {
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
      for (int j = 0; j < 4 && c + j < cols; ++j) atomicAdd(dst + j, e[j]);
    }
  }
}

static int num_pairs() {
  static int pairs = 0;
  if (pairs == 0) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    pairs = sms / 2 > 0 ? sms / 2 : 1;
  }
  return pairs;
}

// Switches for tests and measurements, of the calling thread only: other threads' launches keep the rules.
static thread_local int g_split_k = 1;   // 0: never, 1: by split_parts' rule, n > 1: always n parts
static thread_local int g_tile_n = 0;    // 0: by the rule below, 128 / 192 / 256: as given (tests, measurements)

// Microseconds of a GEMM as far as they depend on the width of its tiles and on the parts K is split into: waves of units over the
// CTA pairs, each its k-blocks and what of its epilogue shows, and for a split the summing kernel and its slices' traffic.
// A 64-deep k-block of a 256 x 256 tile takes the MMA's 512 cycles; one of a 256 x 128 tile half of that, until the pairs share
// L2's bandwidth (three quarters of the operand bytes for half of the products). Constants fitted to 211 shapes (weight and input
// gradients, forward with and without residual; widths of 20M to 1.7B models, 256 to 8,192 tokens; both widths, 1 to 32 parts): 7 %
// off, and the choice it makes 0.5 % slower than the best measured one; those of 192 columns to 66 shapes. Measured 256 / 128 columns /
// 128 split (us): forward 256 x 576 x 576: 7.1 / 5.3; 1024 x 2048 x 2048: 14.9 / 10.2; 8192 x 2048 x 2048: 47.0 / 50.4; weight gradient 576 x 576, 512 tokens: 8.6 / 6.2;
// 2048 x 576 x 3072: 18.0 / 11.3; with residual 256 x 2048 x 8192: 43.0 / 24.5 / 12.8; input gradient 512 x 2048 x 16384: 78 / 54 /
// 35.5 (31.5 with 256 columns).
// (asked: the parts K is to be split into; that gives `parts` of at most kb_part k-blocks.)
struct GemmShape {
  int M, n_cols, K, kb;
  GemmShape(int M_, int n_cols_, int K_) : M(M_), n_cols(n_cols_), K(K_), kb((K_ + BK - 1) / BK) {}
  long long tiles(int bn) const { return (long long)((M + 2 * BM - 1) / (2 * BM)) * ((n_cols + bn - 1) / bn); }
  double mbytes32() const { return (double)M * n_cols * 4e-6; }
};
static double gemm_us(const GemmShape& g, int bn, int asked, int parts, int kb_part, bool f32) {
  const int pairs = num_pairs();
  const long long units = g.tiles(bn) * parts;
  const double load = units < pairs ? (double)units / pairs : 1.0, waves = units <= pairs ? 1.0 : (double)((units + pairs - 1) / pairs);
  const bool slices = asked > 1;
  const double unit = bn == 256   ? kb_part * (0.29 + 0.026 * load) + 1.6 + (f32 || slices ? 0.8 : 0)
                      : bn == 192 ? kb_part * (0.21 + 0.02 * load) + 1.25 + (f32 || slices ? 1.5 : 0)
                                  : kb_part * (0.149 + 0.04 * load) + 0.85 + (f32 || slices ? 0.55 : 0);
  return waves * unit + (slices ? 1.0 + 0.147 * asked * g.mbytes32() : 0.0);
}

// The gain that tiles of bn columns have to promise over wider ones. Narrower tiles fetch more operand bytes per product (192 columns as
// many bytes of an MN-major B as 256), and where these come from HBM or L2's bandwidth is short, that takes what gemm_us sees them give. So 192
// columns need a gain of 6 %, of 12 % for an MN-major B from K = 2048 on; 128 columns in more than one wave 7 %, from K = 4096 on 12 %, and
// 20 % beyond K = 8192 whatever the waves; and among parts, those of 128 columns 5 %. Fitted to 864 shapes (widths of a 20M to an 8B model, 64 to
// 8,192 tokens, operands not in L2; every layout and epilogue with 128 and 256 columns, RoPE and SwiGLU forward without, the others with 192): 3 of
// them are more than 3 % slower than with 256 columns wherever 128 give several waves (22 without these gains, by up to 17 %), and the choice is
// 0.5 % off the best one on average (RoPE 0.15, SwiGLU 0.0, its backward 0.1, forward 1.0, with residual 2.1, input gradients 0.4, weight gradients 0.4 %).
// Measured 256 / 128 columns (us): SwiGLU backward 1024 x 11008 x 4096: 86.1 / 101.0; 768 x 14336 x 4096: 88.1 / 102.4; SwiGLU 512 x 22016 x 4096:
// 81.9 / 92.6; RoPE 512 x 12288 x 4096: 55.3 / 59.5; input gradient 1024 x 2048 x 16384: 60.4 in two parts / 65.8; weight gradient 2048 x 512 over
// 8,192 tokens: 27.6 in four parts / 29.6 in two. 256 / 192: SwiGLU backward 2048 x 8192 x 2048: 69.7 / 73.7.
// Where narrow ones win, 256 / 128 / 192: input gradient 4096 x 576 x 3072: 20.7 / 19.8 / 17.2; 2048 x 576 x 49152, in parts: 101 / 120 / 91; weight
// gradient 960 x 2560 over 4,096 tokens: 26.0 / 27.3 / 22.5; 49152 x 576 over 2,048: 110 / 118 / 102; 5120 x 960 over 8,192: 76.8 / 81.2 / 69.3.
static double gain_asked(const GemmShape& g, int bn, int parts, bool b_mn) {
  if (bn == 192) return b_mn && parts == 1 && g.K >= 2048 ? 0.88 : 0.94;
  if (bn == 256) return 1.0;
  if (parts > 1) return 0.95;
  if (g.K > 8192) return 0.8;
  return g.tiles(128) <= num_pairs() ? 1.0 : g.K < 4096 ? 0.93 : 0.88;
}
static double whole_us(const GemmShape& g, int bn, bool f32, bool b_mn) { return gemm_us(g, bn, 1, 1, g.kb, f32) / gain_asked(g, bn, 1, b_mn); }

// Columns of an output tile; 192 where the epilogue works on independent 64-column chunks.
static int tile_columns(int M, int n_cols, int K, bool f32, bool b_mn, bool has_192) {
  if (g_tile_n) return g_tile_n == 192 && !has_192 ? 256 : g_tile_n;
  const GemmShape g(M, n_cols, K);
  int best = 256;
  double best_us = whole_us(g, 256, f32, b_mn);
  for (const int bn : {192, 128}) {
    if (bn == 192 && !has_192) continue;
    const double us = whole_us(g, bn, f32, b_mn);
    if (us < best_us) {
      best = bn;
      best_us = us;
    }
  }
  return best;
}

template <bool A_MN, bool B_MN, int OUT_MODE, bool EPI_TMA, int EPI = EPI_NONE, int BN = 256>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& md, void* D, int M, int N, int K,
                  long long ldd, KernelStatus* status, cudaStream_t stream, const CUtensorMap* mh = nullptr,
                  EpiArgs ea = EpiArgs{}) {
  auto kern = gemm_pair_kernel<A_MN, B_MN, OUT_MODE, EPI_TMA, EPI, BN>;
  static PerDevice clusters_that_fit;
  const int max_clusters = clusters_that_fit.get(current_device(), [&] {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes_of(EPI, BN, OUT_MODE != OUT_BF16)) != cudaSuccess) return -3;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes_of(EPI, BN, OUT_MODE != OUT_BF16);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return -5;
    }
    return n;
  });
  if (max_clusters <= 0) return max_clusters;
  const int n_tiles = (EPI == EPI_SWIGLU) ? (N + BN / 2 - 1) / (BN / 2) : (N + BN - 1) / BN;
  const int tiles = ((M + 2 * BM - 1) / (2 * BM)) * n_tiles;
  const int num_kb = (K + BK - 1) / BK;
  ea.group_m = g_group_m;
  ea.early = pt_chain_early();
  if (ea.kb_per_part <= 0) ea.kb_per_part = num_kb;
  const int units = tiles * ((num_kb + ea.kb_per_part - 1) / ea.kb_per_part);
  const int clusters = units < max_clusters ? units : max_clusters;
  const cudaError_t err = launch_pdl(kern, dim3(2 * clusters), dim3(NUM_THREADS), smem_bytes_of(EPI, BN, OUT_MODE != OUT_BF16), stream, ma, mb, md,
                                     mh ? *mh : md, D, M, N, K, ldd, status, ea);
  pt_count_launches(1);
  return (err == cudaSuccess && cudaGetLastError() == cudaSuccess) ? 0 : -4;
}

}  // namespace gemm_pair
}  // namespace pt

extern "C" void pt_gemm_set_group_m(int g) { pt::gemm_pair::g_group_m = g < 1 ? 1 : g; }
extern "C" int pt_gemm_get_group_m() { return pt::gemm_pair::g_group_m; }
extern "C" void pt_gemm_set_tile_n(int n) { pt::gemm_pair::g_tile_n = n == 128 || n == 192 || n == 256 ? n : 0; }

// 1 (default): epilogue through shared memory and TMA store / reduce-add; 0: per-thread 16-byte stores.
static int g_tma_epilogue = 1;
extern "C" void pt_gemm_set_tma_epilogue(int on) { g_tma_epilogue = on; }
extern "C" int pt_gemm_get_tma_epilogue() { return g_tma_epilogue; }

extern "C" void pt_gemm_set_split_k(int on) { pt::gemm_pair::g_split_k = on; }

namespace pt {
namespace gemm_pair {
// GEMMs that may be split: dY W, dY^T X into an fp32 destination, X W^T
enum SplitKind { SPLIT_DGRAD = 0, SPLIT_WGRAD = 1, SPLIT_FWD = 2 };
struct SplitPlan {
  int parts, kb_per_part, slices, shift, slice_rows, ws_cols, bn;
};
// Two parts add to a slice of an input gradient's workspace (a sum of two is the same in either order); the parts of a weight
// gradient, whose result has to be read and written anyway, and those of a forward GEMM each store a slice of their own.
static SplitPlan split_plan(int M, int N, int K, int kind, int parts, int bn) {
  SplitPlan s;
  const int kb = (K + BK - 1) / BK;
  s.kb_per_part = (kb + parts - 1) / parts;
  s.parts = (kb + s.kb_per_part - 1) / s.kb_per_part;
  s.shift = kind == SPLIT_DGRAD ? 1 : 0;
  s.slices = (s.parts + s.shift) >> s.shift;
  s.slice_rows = (M + 31) / 32 * 32;        // the epilogue writes 32 rows at a time
  s.ws_cols = (N + 3) / 4 * 4;
  s.bn = bn;
  return s;
}
static int run_pair(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd, int a_mn,
                    int b_mn, int out_mode, const SplitPlan* split, void* status, cudaStream_t stream);
}  // namespace gemm_pair
}  // namespace pt

// Columns of the tiles of an unsplit GEMM with n_cols output columns (fp32 or bf16 results; B MN-major or not; 192 columns allowed or not).
extern "C" int pt_gemm_tile_columns(int M, int n_cols, int K, int f32, int b_mn, int has_192) {
  return pt::gemm_pair::tile_columns(M, n_cols, K, f32 != 0, b_mn != 0, has_192 != 0);
}

// Thread's switch for K shared within clusters: 0 by the rule, 1 never, 2 wherever it can be.
static thread_local int g_cluster = 0;
extern "C" void pt_gemm_set_cluster(int n) { g_cluster = n == 1 || n == 2 ? n : 0; }

namespace pt {
namespace gemm_pair {
template <bool B_MN, bool ADD>
static int clusters_that_fit() {
  static PerDevice fit;
  return fit.get(current_device(), [] {
    auto kern = gemm_cluster_kernel<B_MN, ADD>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes_of(EPI_NONE, CLUSTER_BN)) != cudaSuccess) return -3;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * CLUSTER_PARTS, 1, 1);
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes_of(EPI_NONE, CLUSTER_BN);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2 * CLUSTER_PARTS;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return -5;
    }
    return n;
  });
}
template <typename F>
static int with_cluster_kernel(bool b_mn, bool add, F f) {
  return b_mn ? f(std::true_type{}, std::false_type{}) : add ? f(std::false_type{}, std::true_type{}) : f(std::false_type{}, std::false_type{});
}
}  // namespace gemm_pair
}  // namespace pt

// Whether K is shared within clusters: where one wave of them holds all tiles and gemm_us, with 0.8 us for the exchange, promises 5 % less than
// `others_us`, what the GEMM takes whole or through a workspace, from K = 1536 on, with a residual (which comes in while the tensor cores work) from
// 896. Below, the exchange costs what half of K takes: input gradient 1024 x 576 x 960: 12.3 us whole and this way; with residual 256 x 576 x 576 12.4
// and 12.4, 256 x 960 x 960 14.3 and 12.3. Input gradients with K above 8192 stay with the workspace, whose parts can be many: 64 x 576 x 49152
// has 5 tiles for 74 pairs, here 10 of them would work; what clusters gain is 4 to 7 % by then (512 x 2048 x 16384: 44.0 / 41.0). Of 240 shapes
// (32 to 4,096 tokens; output projections and input gradients of the widths of a 20M to a 7B model) 108 go this way, 11 % faster.
static bool shares_k_in_clusters(int M, int N, int K, bool b_mn, bool add, double others_us) {
  using namespace pt::gemm_pair;
  if (g_cluster == 1 || (g_tile_n && g_cluster != 2)) return false;
  const GemmShape g(M, N, K);
  const int kb_part = (g.kb + CLUSTER_PARTS - 1) / CLUSTER_PARTS;
  if (g.kb < CLUSTER_PARTS) return false;
  if (g_cluster != 2 && (K < (add ? 896 : 1536) || (b_mn && K > 8192))) return false;
  if (g_cluster != 2 && gemm_us(g, CLUSTER_BN, 1, CLUSTER_PARTS, kb_part, false) + 0.8 >= 0.95 * others_us) return false;
  const int fit = with_cluster_kernel(b_mn, add, [](auto b, auto a) { return clusters_that_fit<b(), a()>(); });
  return fit > 0 && (g.tiles(CLUSTER_BN) <= fit || g_cluster == 2);
}

// D = A B (b_mn) or A B^T (+ res, bf16 [M, N], row stride ldr % 8 == 0, or nullptr) with K shared by the pairs of a cluster; N % 8 == 0, K > 64.
extern "C" int pt_gemm_bf16_cluster(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd, int b_mn,
                                    const void* res, long long ldr, void* status, cudaStream_t stream) {
  using namespace pt;
  using namespace pt::gemm_pair;
  CUtensorMap ma, mb, md, mh;
  int rc;
  if ((rc = make_bf16_map_2d(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, BM))) return rc * 10 - 1;
  if ((rc = b_mn ? make_bf16_map_2d(&mb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, BK)
                 : make_bf16_map_2d(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, CLUSTER_BN / 2)))
    return rc * 10 - 2;
  if ((rc = make_bf16_map_2d(&md, D, (uint64_t)N, (uint64_t)M, (uint64_t)ldd, 64, 32))) return rc * 10 - 3;
  mh = md;
  if (res != nullptr && (rc = make_bf16_map_2d(&mh, res, (uint64_t)N, (uint64_t)M, (uint64_t)ldr, 64, 32))) return rc * 10 - 4;
  ClusterArgs ca;
  ca.kb_per_part = ((K + BK - 1) / BK + CLUSTER_PARTS - 1) / CLUSTER_PARTS;
  ca.num_m = (M + 2 * BM - 1) / (2 * BM);
  ca.early = pt_chain_early();
  const int grid = ca.num_m * ((N + CLUSTER_BN - 1) / CLUSTER_BN) * 2 * CLUSTER_PARTS;
  return with_cluster_kernel(b_mn != 0, res != nullptr, [&](auto b, auto a) {
    if (clusters_that_fit<b(), a()>() <= 0) return -5;
    const cudaError_t err = launch_pdl_cluster(gemm_cluster_kernel<b(), a()>, dim3(grid), dim3(NUM_THREADS), smem_bytes_of(EPI_NONE, CLUSTER_BN), stream,
                                               2 * CLUSTER_PARTS, ma, mb, md, mh, M, N, K, reinterpret_cast<KernelStatus*>(status), ca);
    pt_count_launches(1);
    return err == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -4;
  });
}

// How many parts K is split into (1: not at all) and the columns of a tile then, by gemm_us and gain_asked; adding the weight gradient to what is
// there costs 0.08 us a megabyte more in the GEMM's epilogue than in the summing kernel; an input gradient clears its slices first. A
// split has to give 3 %, or 15 % (2048 x 2048 x 128256 on 64 whole tiles: 724 us, in parts 760), and a forward GEMM 2 us more: its second
// launch costs the host 3.5, and passes of small forward GEMMs are bound by the host (256 x 576 x 1536 is 8.7 us whole and 7.6 in five
// parts; the forward pass of the 135M shape on 256 tokens, with 30 of them, took 1,590 us with whole ones and 1,740 with parts; these share K
// within clusters by now, pt_gemm_parts).
// (`us`: what the choice is expected to take, the host's extra included)
static int split_parts(int M, int N, int K, int kind, int* tile_n, double* us) {
  using namespace pt::gemm_pair;
  *tile_n = g_tile_n ? g_tile_n : 256;
  *us = 0;
  const bool wgrad = kind == SPLIT_WGRAD, b_mn = kind != SPLIT_FWD;
  if (M <= 0 || N <= 0 || K <= 0 || !g_split_k || (!wgrad && N % 8)) return 1;
  const GemmShape g(M, N, K);
  if (g_split_k > 1) return g_split_k < g.kb ? g_split_k : g.kb;
  if (g_tile_n) return 1;                  // (a width given for a measurement: of whole tiles)
  // (where whole tiles fill more than half of the pairs, what is left to gain is less than what parts at different K cost in L2 reuse)
  const bool few = 2 * g.tiles(256) <= num_pairs();
  const double whole = whole_us(g, tile_columns(M, N, K, wgrad, b_mn, true), wgrad, b_mn) + (wgrad ? 0.08 * g.mbytes32() : 0.0);
  *us = whole;
  double best = 1e30, best_us = 0;
  int best_parts = 1, best_bn = 256;
  for (const int asked : {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32}) {
    if (g.kb < 2 * asked) break;
    const int kb_part = (g.kb + asked - 1) / asked, parts = (g.kb + kb_part - 1) / kb_part;
    for (const int bn : {128, 192, 256}) {
      const double us = gemm_us(g, bn, asked, parts, kb_part, true), t = us / gain_asked(g, bn, asked, b_mn);
      if (t < best) {
        best = t;
        best_us = us;
        best_parts = asked;
        best_bn = bn;
      }
    }
  }
  if (best_parts == 1) return 1;
  const double split = best_us + (kind == SPLIT_DGRAD ? 2.0 : 0.0);
  if (split >= (few ? 0.97 : 0.85) * whole - (kind == SPLIT_FWD ? 2.0 : 0.0)) return 1;
  *tile_n = best_bn;
  *us = split + (kind == SPLIT_FWD ? 2.0 : 0.0);
  return best_parts;
}
// The choice, or -1: K shared within clusters (pt_gemm_bf16_cluster).
extern "C" int pt_gemm_parts(int M, int N, int K, int kind, int add, int* tile_n) {
  using namespace pt::gemm_pair;
  double us;
  const int parts = split_parts(M, N, K, kind, tile_n, &us);
  if (kind == SPLIT_WGRAD || M <= 0 || N <= 0 || K <= 0 || N % 8 || !g_split_k || g_split_k > 1) return parts;
  return shares_k_in_clusters(M, N, K, kind == SPLIT_DGRAD, add != 0, us) ? -1 : parts;
}

// Floats of workspace for pt_gemm_bf16_split with `parts` parts.
extern "C" long long pt_gemm_split_elems(int M, int N, int K, int kind, int parts) {
  const pt::gemm_pair::SplitPlan p = pt::gemm_pair::split_plan(M, N, K, kind, parts, 256);
  return (long long)p.slices * p.slice_rows * p.ws_cols;
}

// GEMM with K in `parts` parts, each computed by CTA pairs of its own, through the fp32 workspace ws (pt_gemm_split_elems floats,
// 16-byte aligned). Kind 0: D = A B, 2: D = A B^T (+ res, a bf16 [M, N] tensor with row stride ldr % 4 == 0, or nullptr), both rounded
// once (N % 8 == 0, ldd % 8 == 0); 1: D += A^T B in fp32 with one addition per element (ldd % 4 == 0). The result does not depend on
// the order in which the parts finish.
extern "C" int pt_gemm_bf16_split(const void* A, const void* B, void* D, float* ws, int M, int N, int K, long long lda, long long ldb,
                                  long long ldd, int kind, int parts, int tile_n, const void* res, long long ldr, void* status,
                                  cudaStream_t stream) {
  using namespace pt;
  using namespace pt::gemm_pair;
  const SplitPlan p = split_plan(M, N, K, kind, parts, tile_n);
  const long long slice_elems = (long long)p.slice_rows * p.ws_cols, n4 = p.slices * slice_elems / 4;
  if (p.shift > 0) {
    launch_pdl(clear_f32_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, reinterpret_cast<float4*>(ws), n4);
    pt_count_launches(1);
  }
  const int rc = run_pair(A, B, ws, M, N, K, lda, ldb, p.ws_cols, kind == SPLIT_WGRAD, kind != SPLIT_FWD, p.shift > 0 ? OUT_F32_ACC : OUT_F32,
                          &p, status, stream);
  if (rc) return rc;
  const dim3 grid((unsigned)(((long long)M * (p.ws_cols / 4) + 255) / 256));
  auto sum = [&](auto kern) {
    launch_pdl(kern, grid, dim3(256), 0, stream, (const float*)ws, p.slices, slice_elems, D, M, N, p.ws_cols, ldd,
               (const __nv_bfloat16*)res, ldr);
  };
  if (kind == SPLIT_WGRAD) sum(sum_slices_kernel<false, false>);
  else if (res == nullptr) sum(sum_slices_kernel<true, false>);
  else sum(sum_slices_kernel<true, true>);
  pt_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Same contract as pt_gemm_bf16 (gemm_tcgen05.cu). Returns -5 when CTA pairs cannot be scheduled.
extern "C" int pt_gemm_bf16_pair(const void* A, const void* B, void* D, int M, int N, int K, long long lda,
                                 long long ldb, long long ldd, int a_mn, int b_mn, int out_mode, void* status,
                                 cudaStream_t stream) {
  return pt::gemm_pair::run_pair(A, B, D, M, N, K, lda, ldb, ldd, a_mn, b_mn, out_mode, nullptr, status, stream);
}

static int pt::gemm_pair::run_pair(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
                                   long long ldd, int a_mn, int b_mn, int out_mode, const SplitPlan* split, void* status,
                                   cudaStream_t stream) {
  using namespace pt;
  using namespace pt::gemm_pair;
  const bool epi_tma = g_tma_epilogue != 0;
  // narrow tiles exist for the layouts of the model: X W^T, dY W, and dY^T X into fp32
  const bool has_narrow = epi_tma && (out_mode == OUT_BF16 ? !a_mn : (b_mn || (!a_mn && out_mode == OUT_F32)));
  const int bn = !has_narrow ? 256 : split ? split->bn : tile_columns(M, N, K, out_mode != OUT_BF16, b_mn != 0, true);
  CUtensorMap ma, mb;
  int rc;
  rc = a_mn ? make_bf16_map_2d(&ma, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, BK)
            : make_bf16_map_2d(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, BM);
  if (rc) return rc * 10 - 1;    // -21: tensor map of A could not be encoded
  rc = b_mn ? make_bf16_map_2d(&mb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, BK)
            : make_bf16_map_2d(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, bn / 2);
  if (rc) return rc * 10 - 2;    // -22: tensor map of B could not be encoded
  CUtensorMap md = ma;           // unused by the per-thread epilogue
  if (epi_tma) {
    uint64_t dims[2] = {(uint64_t)N, split ? (uint64_t)split->slices * split->slice_rows : (uint64_t)M};
    uint64_t strides[1] = {(uint64_t)ldd};
    uint32_t box_bf16[2] = {64, 32}, box_f32[2] = {32, 32};
    rc = out_mode == OUT_BF16 ? make_bf16_map(&md, D, 2, dims, strides, box_bf16) : make_f32_map(&md, D, 2, dims, strides, box_f32);
    if (rc) return rc * 10 - 3;  // -23: tensor map of D could not be encoded
  }
  EpiArgs ea{};
  if (split) {
    ea.kb_per_part = split->kb_per_part;
    ea.slice_rows = split->slice_rows;
    ea.slice_shift = split->shift;
  }
  KernelStatus* st = reinterpret_cast<KernelStatus*>(status);
#define PT_GEMM_NARROW(AM, BMN, OM)                                                                           \
  if (bn != 256 && a_mn == AM && b_mn == BMN && out_mode == OM)                                               \
    return bn == 128 ? launch<AM, BMN, OM, true, EPI_NONE, 128>(ma, mb, md, D, M, N, K, ldd, st, stream, nullptr, ea) \
                     : launch<AM, BMN, OM, true, EPI_NONE, 192>(ma, mb, md, D, M, N, K, ldd, st, stream, nullptr, ea);
  PT_GEMM_NARROW(0, 0, 0) PT_GEMM_NARROW(0, 1, 0) PT_GEMM_NARROW(0, 0, 2) PT_GEMM_NARROW(0, 1, 1) PT_GEMM_NARROW(0, 1, 2) PT_GEMM_NARROW(1, 1, 1)
  PT_GEMM_NARROW(1, 1, 2)
#undef PT_GEMM_NARROW
#define PT_GEMM_CASE(AM, BMN, OM)                                                                             \
  if (a_mn == AM && b_mn == BMN && out_mode == OM)                                                            \
    return epi_tma ? launch<AM, BMN, OM, true>(ma, mb, md, D, M, N, K, ldd, st, stream, nullptr, ea)          \
                   : launch<AM, BMN, OM, false>(ma, mb, md, D, M, N, K, ldd, st, stream);
  PT_GEMM_CASE(0, 0, 0) PT_GEMM_CASE(0, 0, 1) PT_GEMM_CASE(0, 0, 2)
  PT_GEMM_CASE(0, 1, 0) PT_GEMM_CASE(0, 1, 1) PT_GEMM_CASE(0, 1, 2)
  PT_GEMM_CASE(1, 1, 0) PT_GEMM_CASE(1, 1, 1) PT_GEMM_CASE(1, 1, 2)
  PT_GEMM_CASE(1, 0, 0) PT_GEMM_CASE(1, 0, 1) PT_GEMM_CASE(1, 0, 2)
#undef PT_GEMM_CASE
  return -11;
}

// Forward GEMM D[M, N] = A[M, K] B[N, K]^T (bf16) with a fused epilogue; requirements as pt_gemm_bf16 plus:
//   epi 1 (SwiGLU): B is [2 I, K] (gate rows, then up rows), D is [M, 2 I] (ldd), H is [M, I] bf16 (ldh, 16-byte aligned,
//                   ldh % 8 == 0), I % 128 == 0; N is ignored.
//   epi 2 (RoPE):   D is the packed q|k|v activation [M, N]; head_dim 64 or 128; columns [0, rot_heads * head_dim) are
//                   rotated with cosT/sinT (fp32 [seq, head_dim / 2], 16-byte aligned) at position row % seq.
//   epi 4 (ADD):    D = A B^T + H with H a bf16 [M, N] tensor (ldh); N % 8 == 0.
//   epi 5 (SwiGLU backward, dgrad layout): A is dY [M, K], B is the down-projection weight stored [K, I] (ldb), so the
//                   accumulator is da [M, I]; H is the packed pre-activation [M, 2 I] (ldh), D the packed gradient [M, 2 I]
//                   (ldd): D[:, :I] = da * up * silu'(gate), D[:, I:] = da * silu(gate). inter = I, I % 64 == 0; N is ignored.
// Returns 1 (nothing launched) when the shape is not covered, so that the caller can run the unfused kernels.
extern "C" int pt_gemm_bf16_fused(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
                                  long long ldd, int epi, void* H, long long ldh, int inter, const float* cosT,
                                  const float* sinT, int seq, int rot_heads, int head_dim, void* status,
                                  cudaStream_t stream) {
  using namespace pt;
  using namespace pt::gemm_pair;
  if (!g_tma_epilogue) return 1;
  if ((lda % 8) || (ldb % 8) || (ldd % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(D) & 15))
    return -10;
  EpiArgs ea{};
  int n_out = N;
  if (epi == EPI_SWIGLU) {
    if (inter <= 0 || inter % 128 || H == nullptr || (ldh % 8) || (reinterpret_cast<uintptr_t>(H) & 15)) return 1;
    ea.inter = inter;
    n_out = 2 * inter;
  } else if (epi == EPI_ADD) {
    if (H == nullptr || (ldh % 8) || (reinterpret_cast<uintptr_t>(H) & 15) || (N % 8)) return 1;
  } else if (epi == EPI_SWIGLU_BWD) {
    if (inter <= 0 || inter % 64 || H == nullptr || (ldh % 8) || (reinterpret_cast<uintptr_t>(H) & 15)) return 1;
    ea.inter = inter;
    n_out = 2 * inter;
  } else if (epi == 2) {
    if ((head_dim != 64 && head_dim != 128) || seq <= 0 || cosT == nullptr || sinT == nullptr ||
        (reinterpret_cast<uintptr_t>(cosT) & 15) || (reinterpret_cast<uintptr_t>(sinT) & 15) || rot_heads < 0 ||
        (long long)rot_heads * head_dim > N)
      return 1;
    ea.cosT = cosT;
    ea.sinT = sinT;
    ea.seq = seq;
    ea.rot_cols = rot_heads * head_dim;
  } else {
    return -11;
  }
  if (M <= 0 || n_out <= 0 || K <= 0) return 0;
  const int bn = tile_columns(M, epi == EPI_SWIGLU_BWD ? inter : n_out, K, false, epi == EPI_SWIGLU_BWD, epi == EPI_ADD || epi == EPI_SWIGLU_BWD);
  CUtensorMap ma, mb, md, mh;
  int rc;
  if ((rc = make_bf16_map_2d(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, BM))) return rc * 10 - 1;
  if (epi == EPI_SWIGLU_BWD) {
    // B is stored [K, I] (MN-major operand): 64-column x BK-row boxes, as in the plain dgrad GEMM
    if ((rc = make_bf16_map_2d(&mb, B, (uint64_t)inter, (uint64_t)K, (uint64_t)ldb, 64, BK))) return rc * 10 - 2;
  } else {
    if ((rc = make_bf16_map_2d(&mb, B, (uint64_t)K, (uint64_t)n_out, (uint64_t)ldb, BK, bn / 2))) return rc * 10 - 2;
  }
  if ((rc = make_bf16_map_2d(&md, D, (uint64_t)n_out, (uint64_t)M, (uint64_t)ldd, 64, 32))) return rc * 10 - 3;
  mh = md;
  if ((epi == EPI_ADD || epi == EPI_SWIGLU_BWD) &&
      (rc = make_bf16_map_2d(&mh, H, (uint64_t)n_out, (uint64_t)M, (uint64_t)ldh, 64, 32)))
    return rc * 10 - 4;
  if (epi == EPI_SWIGLU && (rc = make_bf16_map_2d(&mh, H, (uint64_t)inter, (uint64_t)M, (uint64_t)ldh, 64, 32))) return rc * 10 - 4;
  KernelStatus* st = reinterpret_cast<KernelStatus*>(status);
  auto run = [&](auto width) -> int {
    constexpr int W = decltype(width)::value;
    if (epi == EPI_ADD) return launch<false, false, OUT_BF16, true, EPI_ADD, W>(ma, mb, md, D, M, N, K, ldd, st, stream, &mh, ea);
    if (epi == EPI_SWIGLU_BWD) return launch<false, true, OUT_BF16, true, EPI_SWIGLU_BWD, W>(ma, mb, md, D, M, inter, K, ldd, st, stream, &mh, ea);
    if constexpr (W != 192) {                           // (tile_columns does not give 192 to the others)
      if (epi == EPI_SWIGLU) return launch<false, false, OUT_BF16, true, EPI_SWIGLU, W>(ma, mb, md, D, M, inter, K, ldd, st, stream, &mh, ea);
      if (head_dim == 64) return launch<false, false, OUT_BF16, true, EPI_ROPE64, W>(ma, mb, md, D, M, N, K, ldd, st, stream, &mh, ea);
      return launch<false, false, OUT_BF16, true, EPI_ROPE128, W>(ma, mb, md, D, M, N, K, ldd, st, stream, &mh, ea);
    }
    return -11;
  };
  if (bn == 192) return run(std::integral_constant<int, 192>{});
  return bn == 128 ? run(std::integral_constant<int, 128>{}) : run(std::integral_constant<int, 256>{});
}

// LM-head GEMM with the cross-entropy row statistics in its epilogue: D[M, N] = A[M, K] B[N, K]^T (bf16, stored because the
// gradient pass rewrites it in place) and, per row and per 256-column tile, (max, sum exp(logit - max)) of the stored
// values -> part[M, tiles] (tiles = ceil(N / 256)), plus tgt[M] = logit of column targets[row] - vocab_start where that
// column lies in [0, N) (rows whose target lies elsewhere are not written). Replaces the separate statistics pass over the logits.
// D == nullptr: the statistics alone (the loss without a gradient never reads the logits again). Returns 1 when the kernel does not
// cover the case.
extern "C" int pt_gemm_bf16_ce(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
                               long long ldd, const long long* targets, long long vocab_start, void* part, float* tgt,
                               void* status, cudaStream_t stream) {
  using namespace pt;
  using namespace pt::gemm_pair;
  if (!g_tma_epilogue) return 1;
  if ((lda % 8) || (ldb % 8) || (ldd % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(D) & 15) || (reinterpret_cast<uintptr_t>(part) & 7) || (N % 8))
    return -10;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  EpiArgs ea{};
  ea.ce_part = reinterpret_cast<float2*>(part);
  ea.ce_tgt = tgt;
  ea.ce_targets = targets;
  ea.ce_vocab_start = vocab_start;
  ea.ce_tiles = (N + 255) / 256;
  ea.ce_store = D != nullptr;
  CUtensorMap ma, mb, md;
  int rc;
  if ((rc = make_bf16_map_2d(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, BM))) return rc * 10 - 1;
  if ((rc = make_bf16_map_2d(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, 128))) return rc * 10 - 2;
  md = ma;                       // (not used without D)
  if (D != nullptr && (rc = make_bf16_map_2d(&md, D, (uint64_t)N, (uint64_t)M, (uint64_t)ldd, 64, 32))) return rc * 10 - 3;
  return launch<false, false, OUT_BF16, true, EPI_CE>(ma, mb, md, D, M, N, K, ldd, reinterpret_cast<KernelStatus*>(status), stream,
                                                      &md, ea);
}
