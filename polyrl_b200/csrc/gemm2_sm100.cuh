// polyrl_b200 — CTA-pair (cta_group::2) persistent tcgen05 GEMM family for sm_100a.
//
//   D[M,N] = sum_k A(m,k) * B(n,k)
//
// One mainloop serves the three layouts a Linear layer needs (reference: the cuBLAS calls behind
// nn.Linear forward/backward in 3rdparty/verl/verl/workers/actor/dp_actor.py:86-273 and the CE
// backward GEMMs of verl/utils/kernel/kernels.py:1571-1581):
//   NT  forward   y  = x  · W^T     A = x  [M,K]  K-major      B = W  [N,K]  K-major
//   NN  dgrad     dx = dy · W       A = dy [M,Kr] K-major      B = W  [Kr,N] MN-major
//   TN  wgrad     dW = dy^T · x     A = dy [Kr,M] MN-major     B = x  [Kr,N] MN-major
// (Kr = reduction length).  MN-major operands are staged by {64 x 64} SWIZZLE_128B TMA boxes and
// consumed through MN-major UMMA descriptors, so no operand is ever transposed in memory.
//
// A cluster of two CTAs (one SM pair) owns a 256 x BN output tile: each CTA stages its own 128
// rows of A and HALF of the B tile (BN/2 rows), the leader CTA's single elected thread issues
// `tcgen05.mma.cta_group::2` (M = 256) which reads both CTAs' shared memory, and each CTA's TMEM
// receives its 128 accumulator rows.  Halving the per-SM B traffic is what lifts the kernel off
// the shared-memory bandwidth limit of the 1-CTA 128x256 tile (gemm_sm100.cuh).
//
// Warp roles per CTA (192 threads with one epilogue group): warp 0 TMA producer (both CTAs, completion bytes counted on the
// LEADER's full barrier), warp 1 TMEM allocator + (leader only) MMA issuer, warps 2..5 (2..9) epilogue.
// Barriers: full[s] leader-only (count 1, expect 2 x stage bytes); empty[s] and tmem_full[a] per
// CTA, signalled by multicast `tcgen05.commit`; tmem_empty[a] on the leader, one remote arrival per epilogue warp
// (an elected lane per epilogue warp of both CTAs).
//
// Epilogues: (a) functor mode — same `Epi` interface as gemm_sm100.cuh (SwiGLU, linear-CE, ...);
// (b) TMA-store mode — accumulators -> bf16 -> 128B-swizzled shared staging -> `cp.async.bulk.tensor`
// store, optional fused residual add; each epilogue warp double-buffers its own 32 x 64
// box so no cross-warp barrier is needed.
#pragma once
#include "gemm_sm100.cuh"

namespace prl {

constexpr int kSmemMax = 232448;   // 227 KB opt-in limit per CTA

// EPI_GROUPS: warpgroups that share a tile's columns in the epilogue.  One is enough where the epilogue converts and stores; an epilogue
// that takes an exponential per element gets two, because a warp per scheduler cannot hide its latencies and short reductions
// (K of about a thousand) leave it no time: the figures are beside its users.
template <int BN, bool A_MN_, bool B_MN_, bool TMA_STORE_, int EPI_GROUPS_ = 1>
struct Gemm2Cfg {
  static constexpr int EPI_GROUPS = EPI_GROUPS_, EPI_WARPS = 4 * EPI_GROUPS, THREADS = 64 + 32 * EPI_WARPS;
  static constexpr int GROUP_N = BN / EPI_GROUPS;     // columns of a group
  static constexpr bool A_MN = A_MN_, B_MN = B_MN_, TMA_STORE = TMA_STORE_;
  static constexpr int BLOCK_M = 256;                 // per CTA pair
  static constexpr int CTA_M = 128;
  static constexpr int BLOCK_N = BN;
  static constexpr int CTA_N = BN / 2;                // rows of B staged by each CTA
  static constexpr int BLOCK_K = 64;
  static constexpr int A_BYTES = CTA_M * 128;
  static constexpr int B_BYTES = CTA_N * 128;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_BYTES = TMA_STORE ? EPI_WARPS * 2 * 4096 : 0;
  static constexpr int STAGES_RAW = (kSmemMax - 1024 - 512 - EPI_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_RAW > 8 ? 8 : STAGES_RAW;
  static constexpr int TMEM_COLS = 2 * BN;            // 256 or 512
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 + 512;
  static_assert(BN == 128 || BN == 256, "CTA-pair tile is 256 x {128,256}");
  static_assert(STAGES >= 3, "pipeline too shallow");
};

// TMA-store epilogue tag (handled inside the kernel, not a per-row functor).
struct TmaStoreParams {
  const __nv_bfloat16* R;              // optional residual, pitch as D
  int64_t ldd;
  __nv_bfloat16* D = nullptr;          // the matrix that the TMA stores write, for tiles that are finished from their slots
};
struct EpiTmaStore {
  using Params = TmaStoreParams;
  static constexpr bool kFinish = true;
  // columns [n0 + c, n0 + c + 4) of one row; sum(c) gives the fp32 sums (N is a multiple of 8)
  template <class Sum>
  __device__ __forceinline__ static void finish(const Params& p, const Sum& sum, int row, int n0, int c, int N) {
    const int col = n0 + c;
    if (col >= N) return;
    float4 t = sum(c);
    if (p.R != nullptr) {
      const uint2 q = *reinterpret_cast<const uint2*>(p.R + static_cast<int64_t>(row) * p.ldd + col);
      const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y);
      t.x += a.x; t.y += a.y; t.z += b.x; t.w += b.y;
    }
    *reinterpret_cast<uint2*>(p.D + static_cast<int64_t>(row) * p.ldd + col) = make_uint2(pack_bf16(t.x, t.y), pack_bf16(t.z, t.w));
  }
  static constexpr bool kRow = false;   // true: a functor with per-row state, begin(params, row, M) and apply(params, r[64], column)
  static constexpr int kAct = 0;
};
// same with gelu (tanh form) on the accumulators, in the exactly equivalent shape z * sigmoid(2 u)
struct EpiTmaStoreGelu {
  using Params = TmaStoreParams;
  static constexpr bool kFinish = false;
  static constexpr bool kRow = false;
  static constexpr int kAct = 1;
};
struct EpiTmaStoreSilu {
  using Params = TmaStoreParams;
  static constexpr bool kFinish = false;
  static constexpr bool kRow = false;
  static constexpr int kAct = 2;
};
__device__ __forceinline__ float gelu_fast(float z) {
  return __fdividef(z, 1.0f + __expf(fminf(-1.5957691216057308f * (z + 0.044715f * z * z * z), 80.f)));
}
__device__ __forceinline__ float silu_fast(float z) { return __fdividef(z, 1.0f + __expf(fminf(-z, 80.f))); }

// The last round of tiles, cut along the reduction (as in "stream-K" decompositions).  `full` tiles go to the pairs whole; the k-blocks of the remaining `tiles` are dealt
// out evenly, in order, to `workers` pairs, each of which takes a run of k-blocks of one tile or of the end of one and the start of the
// next, and leaves its fp32 sums in a slot of `ws`.  split_finish_kernel adds a tile's slots in order and applies the epilogue.
struct KSplit {
  int full, tiles, workers;
  float* ws;                 // [2 * workers slots][256 rows][256 columns]
};
struct KRun {
  int tile, kb0, kb1, slot;
};
// run `i` (0 or 1) of worker w; false: there is none.  tiles <= workers, so a worker's run is no longer than a tile.
__host__ __device__ __forceinline__ bool k_run(const KSplit& ks, int num_kb, int w, int i, KRun& r) {
  const int64_t all = static_cast<int64_t>(ks.tiles) * num_kb;
  int64_t a = all * w / ks.workers;
  const int64_t b = all * (w + 1) / ks.workers, edge = (a / num_kb + 1) * num_kb;
  if (i == 1) {
    if (b <= edge) return false;
    a = edge;
  }
  const int64_t e = b < edge || i == 1 ? b : edge;
  r.tile = static_cast<int>(a / num_kb);
  r.kb0 = static_cast<int>(a - static_cast<int64_t>(r.tile) * num_kb);
  r.kb1 = r.kb0 + static_cast<int>(e - a);
  r.slot = 2 * w + i;
  return e > a;
}

template <class Cfg, class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg::THREADS, 1)
gemm2_sm100_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmD, typename Epi::Params ep, int M, int N, int K,
                   int num_m_blocks, int num_n_blocks, int n_splits, int nb_per_split, Sched sc, KSplit ks) {
  constexpr int BN = Cfg::BLOCK_N;
  constexpr int kStages = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kStages * Cfg::A_BYTES;
  uint8_t* smem_epi = smem + kStages * Cfg::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_epi + Cfg::EPI_BYTES);
  uint64_t* full_bar = bars;                       // [kStages]  TMA (both CTAs) -> leader MMA
  uint64_t* empty_bar = bars + kStages;            // [kStages]  MMA -> TMA, one copy per CTA
  uint64_t* tmem_full = bars + 2 * kStages;        // [2]        MMA -> epilogue, one copy per CTA
  uint64_t* tmem_empty = bars + 2 * kStages + 2;   // [2]        epilogue (both CTAs) -> leader MMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;
  const int total_work = ks.tiles ? ks.full : num_m_blocks * n_splits;
  const int num_kb = (K + Cfg::BLOCK_K - 1) / Cfg::BLOCK_K;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if constexpr (Cfg::TMA_STORE) tma_prefetch_desc(&tmD);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * Cfg::EPI_WARPS);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_2sm(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_2sm();
  }
  tc_fence_before();
  cluster_sync_all();            // barrier inits + TMEM allocation visible across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ================================ TMA producer (both CTAs) ================================
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      auto load = [&](int m_blk, int nb, int kb0, int kb1) {
        const int m0 = m_blk * Cfg::BLOCK_M + static_cast<int>(rank) * Cfg::CTA_M;
        const int n0 = rot_n(nb, num_n_blocks, sc) * BN + static_cast<int>(rank) * Cfg::CTA_N;
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(&empty_bar[stage], phase ^ 1);
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * Cfg::STAGE_BYTES);
          uint8_t* sa = smem_a + stage * Cfg::A_BYTES;
          uint8_t* sb = smem_b + stage * Cfg::B_BYTES;
          const int k0 = kb * Cfg::BLOCK_K;
          if constexpr (!Cfg::A_MN) {
            tma_load_2d_2sm(&tmA, &full_bar[stage], sa, k0, m0, kEvictNormal);
          } else {
#pragma unroll
            for (int c = 0; c < Cfg::CTA_M / 64; ++c)
              tma_load_2d_2sm(&tmA, &full_bar[stage], sa + c * 8192, m0 + c * 64, k0, kEvictNormal);
          }
          if constexpr (!Cfg::B_MN) {
            tma_load_2d_2sm(&tmB, &full_bar[stage], sb, k0, n0, kEvictNormal);
          } else {
#pragma unroll
            for (int c = 0; c < Cfg::CTA_N / 64; ++c)
              tma_load_2d_2sm(&tmB, &full_bar[stage], sb + c * 8192, n0 + c * 64, k0, kEvictNormal);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      };
      for (int w = cluster_id; w < total_work; w += num_clusters) {
        const WorkInfo wi = decode_work(w, num_m_blocks, num_n_blocks, n_splits, nb_per_split, sc);
        for (int nbs = wi.n_begin; nbs < wi.n_end; ++nbs) load(wi.m_blk, nbs, 0, num_kb);
      }
      if (cluster_id < ks.workers) {
        KRun kr;
        for (int i = 0; i < 2 && k_run(ks, num_kb, cluster_id, i, kr); ++i) {
          const WorkInfo wi = decode_work(ks.full + kr.tile, num_m_blocks, num_n_blocks, n_splits, nb_per_split, sc);
          load(wi.m_blk, wi.n_begin, kr.kb0, kr.kb1);
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer (leader CTA only) ============================
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = umma_idesc_major(Cfg::BLOCK_M, BN, 1, 1, Cfg::A_MN ? 1 : 0, Cfg::B_MN ? 1 : 0);
      constexpr uint32_t a_step = Cfg::A_MN ? (16 * 128) >> 4 : 32 >> 4;   // descriptor units (16 B) per UMMA_K
      constexpr uint32_t b_step = Cfg::B_MN ? (16 * 128) >> 4 : 32 >> 4;
      int stage = 0;
      uint32_t phase = 0;
      uint32_t tile_iter = 0;
      auto multiply = [&](int kb0, int kb1) {
        const uint32_t as = tile_iter & 1;
        const uint32_t aphase = (tile_iter >> 1) & 1;
        mbar_wait(&tmem_empty[as], aphase ^ 1);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + as * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint8_t* sa = smem_a + stage * Cfg::A_BYTES;
          const uint8_t* sb = smem_b + stage * Cfg::B_BYTES;
          const uint64_t da = Cfg::A_MN ? umma_desc_sw128_mnmajor(sa, 8192) : umma_desc_sw128_kmajor(sa);
          const uint64_t db = Cfg::B_MN ? umma_desc_sw128_mnmajor(sb, 8192) : umma_desc_sw128_kmajor(sb);
#pragma unroll
          for (int k = 0; k < Cfg::BLOCK_K / 16; ++k)
            umma_bf16_ss_2sm(tmem_d, da + k * a_step, db + k * b_step, idesc, kb != kb0 || k != 0);
          umma_commit_2sm(&empty_bar[stage], 3);          // both CTAs' producers may refill this slot
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        umma_commit_2sm(&tmem_full[as], 3);               // both CTAs' epilogues may drain their half
        ++tile_iter;
      };
      for (int w = cluster_id; w < total_work; w += num_clusters) {
        const WorkInfo wi = decode_work(w, num_m_blocks, num_n_blocks, n_splits, nb_per_split, sc);
        for (int nb = wi.n_begin; nb < wi.n_end; ++nb) multiply(0, num_kb);
      }
      if (cluster_id < ks.workers) {
        KRun kr;
        for (int i = 0; i < 2 && k_run(ks, num_kb, cluster_id, i, kr); ++i) multiply(kr.kb0, kr.kb1);
      }
    }
  } else {
    // ================================ epilogue (both CTAs) ====================================
    const int quad = warp & 3;                       // TMEM lane quadrant this warp may read
    const int group = (warp - 2) >> 2;               // which columns of the tile are its own
    const int row_in_tile = static_cast<int>(rank) * Cfg::CTA_M + quad * 32 + lane;
    uint32_t tile_iter = 0;
    if constexpr (Cfg::TMA_STORE) {
      uint8_t* ebuf = smem_epi + (warp - 2) * 8192;
      [[maybe_unused]] Epi epi;
      uint32_t chunk_ctr = 0;
      for (int w = cluster_id; w < total_work; w += num_clusters) {
        const WorkInfo wi = decode_work(w, num_m_blocks, num_n_blocks, n_splits, nb_per_split, sc);
        const int row = wi.m_blk * Cfg::BLOCK_M + row_in_tile;
        const int row0 = row - lane;
        if constexpr (Epi::kRow) epi.begin(ep, row, M);
        for (int nb = wi.n_begin; nb < wi.n_end; ++nb, ++tile_iter) {
          const uint32_t as = tile_iter & 1;
          const uint32_t aphase = (tile_iter >> 1) & 1;
          const int n0 = rot_n(nb, num_n_blocks, sc) * BN + group * Cfg::GROUP_N;
          mbar_wait(&tmem_full[as], aphase);
          tc_fence_after();
          const uint32_t taddr = tmem_base + as * BN + group * Cfg::GROUP_N + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
          for (int c = 0; c < Cfg::GROUP_N / 64; ++c, ++chunk_ctr) {
            uint8_t* buf = ebuf + (chunk_ctr & 1) * 4096;
            if (lane == 0) tma_store_wait_read<1>();   // the store that last read `buf` has drained it
            __syncwarp();
            uint32_t r[64];
            tmem_ld_32x32(taddr + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
            tmem_ld_32x32(taddr + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
            tmem_ld_wait();
            if (c == Cfg::GROUP_N / 64 - 1) {                     // accumulator fully read: hand TMEM back early
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(&tmem_empty[as], 0);
            }
            const int col0 = n0 + c * 64;
            if constexpr (Epi::kRow) {
              epi.apply(ep, r, col0);
            } else {
            if (ep.R != nullptr && row < M) {
              const __nv_bfloat16* rp = ep.R + static_cast<int64_t>(row) * ep.ldd + col0;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if (col0 + 8 * j < N) {
                  const int4 q = ld_nc_v4(rp + 8 * j);
                  const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), cc = unpack_bf16(q.z), d = unpack_bf16(q.w);
                  r[8 * j + 0] = __float_as_uint(__uint_as_float(r[8 * j + 0]) + a.x);
                  r[8 * j + 1] = __float_as_uint(__uint_as_float(r[8 * j + 1]) + a.y);
                  r[8 * j + 2] = __float_as_uint(__uint_as_float(r[8 * j + 2]) + b.x);
                  r[8 * j + 3] = __float_as_uint(__uint_as_float(r[8 * j + 3]) + b.y);
                  r[8 * j + 4] = __float_as_uint(__uint_as_float(r[8 * j + 4]) + cc.x);
                  r[8 * j + 5] = __float_as_uint(__uint_as_float(r[8 * j + 5]) + cc.y);
                  r[8 * j + 6] = __float_as_uint(__uint_as_float(r[8 * j + 6]) + d.x);
                  r[8 * j + 7] = __float_as_uint(__uint_as_float(r[8 * j + 7]) + d.y);
                }
              }
            }
            if constexpr (Epi::kAct != 0) {
#pragma unroll
              for (int j = 0; j < 64; ++j)
                r[j] = __float_as_uint(Epi::kAct == 1 ? gelu_fast(__uint_as_float(r[j])) : silu_fast(__uint_as_float(r[j])));
            }
            }
            // row `lane` of the 32 x 64 box: 8 x 16 B chunks, chunk j lands at (j ^ (lane & 7)) (128B swizzle)
            const uint32_t row_base = smem_u32(buf) + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t p0 = pack_bf16(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1]));
              const uint32_t p1 = pack_bf16(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
              const uint32_t p2 = pack_bf16(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
              const uint32_t p3 = pack_bf16(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_base + ((j ^ (lane & 7)) << 4)),
                           "r"(p0), "r"(p1), "r"(p2), "r"(p3)
                           : "memory");
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              if (row0 < M && col0 < N) tma_store_2d(&tmD, buf, col0, row0);   // TMA clips partial boxes
              tma_store_commit();
            }
          }
        }
      }
      if (lane == 0) tma_store_wait<0>();
    } else {
      Epi epi;
      for (int w = cluster_id; w < total_work; w += num_clusters) {
        WorkInfo wi = decode_work(w, num_m_blocks, num_n_blocks, n_splits, nb_per_split, sc);
        const int row = wi.m_blk * Cfg::BLOCK_M + row_in_tile;
        wi.split = wi.split * Cfg::EPI_GROUPS + group;       // each group carries running state of its own
        epi.begin(ep, row, M, wi);
        for (int nb = wi.n_begin; nb < wi.n_end; ++nb, ++tile_iter) {
          const uint32_t as = tile_iter & 1;
          const uint32_t aphase = (tile_iter >> 1) & 1;
          mbar_wait(&tmem_full[as], aphase);
          tc_fence_after();
          AccReader acc{tmem_base + as * BN + group * Cfg::GROUP_N + (static_cast<uint32_t>(quad * 32) << 16)};
          epi.template tile<Cfg::GROUP_N>(ep, acc, row, M, rot_n(nb, num_n_blocks, sc) * BN + group * Cfg::GROUP_N, N);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(&tmem_empty[as], 0);
        }
        epi.end(ep, row, M, wi);
      }
    }
    if (cluster_id < ks.workers) {                    // runs of k-blocks: the sums as they are
      KRun kr;
      for (int i = 0; i < 2 && k_run(ks, num_kb, cluster_id, i, kr); ++i, ++tile_iter) {
        const uint32_t as = tile_iter & 1;
        mbar_wait(&tmem_full[as], (tile_iter >> 1) & 1);
        tc_fence_after();
        AccReader acc{tmem_base + as * BN + group * Cfg::GROUP_N + (static_cast<uint32_t>(quad * 32) << 16)};
        float* dst = ks.ws + (static_cast<int64_t>(kr.slot) * Cfg::BLOCK_M + row_in_tile) * BN + group * Cfg::GROUP_N;
#pragma unroll 1
        for (int c = 0; c < Cfg::GROUP_N; c += 32) {
          float v[32];
          acc.load(c, v);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(dst + c + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(&tmem_empty[as], 0);
      }
    }
  }

  tc_fence_before();
  cluster_sync_all();            // nobody leaves while the peer may still read its smem / signal its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, Cfg::TMEM_COLS);
  }
}

// Sum of a tile's slots at columns [c, c + 4) of one row, in the order of the k-blocks.
struct SlotSum {
  const float* ws;
  int first, count, skip, row;         // worker that holds the tile's first run, workers, whether that is its second run, row in the tile
  __device__ __forceinline__ float4 operator()(int c) const {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4* p = reinterpret_cast<const float4*>(ws + (static_cast<int64_t>(2 * first) * 256 + row) * 256 + c);
    constexpr int kStep = 2 * 256 * 256 / 4;             // from one worker's first slot to the next one's
    for (int i = 0; i < count; i += 8) {                 // eight loads in flight
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = i + j < count ? p[static_cast<int64_t>(i + j) * kStep + (i + j == 0 && skip ? kStep / 2 : 0)] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) { t.x += v[j].x; t.y += v[j].y; t.z += v[j].z; t.w += v[j].w; }
    }
    return t;
  }
};
constexpr int kFinishRows = 4;
// grid (tiles, 256 / kFinishRows), 256 threads: 64 threads a row, four columns each, so that a few tiles still fill the chip
template <class Epi>
__global__ void __launch_bounds__(256) split_finish_kernel(typename Epi::Params ep, KSplit ks, int num_kb, int M, int N, int num_m_blocks,
                                                           int num_n_blocks, Sched sc) {
  const WorkInfo wi = decode_work(ks.full + blockIdx.x, num_m_blocks, num_n_blocks, num_n_blocks, 1, sc);
  const int64_t all = static_cast<int64_t>(ks.tiles) * num_kb, lo = static_cast<int64_t>(blockIdx.x) * num_kb, hi = lo + num_kb;
  int first = static_cast<int>(lo * ks.workers / all);
  while (all * (first + 1) / ks.workers <= lo) ++first;
  while (first > 0 && all * first / ks.workers > lo) --first;
  int last = first;
  while (last + 1 < ks.workers && all * (last + 1) / ks.workers < hi) ++last;
  const int n0 = rot_n(wi.n_begin, num_n_blocks, sc) * 256, c = (threadIdx.x & 63) * 4;
  const int in_tile = blockIdx.y * kFinishRows + (threadIdx.x >> 6), row = wi.m_blk * 256 + in_tile;
  if (row >= M) return;
  const SlotSum sum{ks.ws, first, last - first + 1, all * first / ks.workers < lo ? 1 : 0, in_tile};
  Epi::finish(ep, sum, row, n0, c, N);
}

// Cut of the last round for tiles of 256 x 256 over `pairs` SM pairs; tiles = 0 when it is not worth it.  In microseconds, a k-block takes a
// pair 0.3, and a slot (256 KB) is written and read back in 0.25 when all pairs do it together, behind 3 for the second kernel.  It has to
// save a twentieth of the product: long ones run at the power limit, where an idle pair's share goes to the others.
// 2781 x 3584 with K 3584 (kept whole) and 18944 (6 tiles of 154 cut into runs), and qkv, twice: 939 -> 814 us, the second kernel
// included; 2781 tokens through two 7B blocks 2444 -> 2329 us.
inline KSplit plan_k_split(int64_t total, int num_kb, int pairs) {
  KSplit none{0, 0, 0, nullptr};
  const int rest = static_cast<int>(total % pairs);
  if (rest == 0 || 2 * rest > pairs * 3 / 2) return none;
  const double tile = 0.3 * num_kb, rounds = static_cast<double>(total / pairs + 1);
  int best = 0;
  double best_cost = tile - 0.05 * tile * rounds;
  for (int w = rest + 1; w <= pairs && static_cast<int64_t>(rest) * num_kb >= 4ll * w; ++w) {
    const double cost = tile * rest / w + 3.0 + 0.25 * (w + rest);
    if (cost < best_cost) { best_cost = cost; best = w; }
  }
  if (!best) return none;
  return KSplit{static_cast<int>(total - rest), rest, best, nullptr};
}
inline KSplit plan_k_split(int M, int N, int K) {
  return plan_k_split(static_cast<int64_t>((M + 255) / 256) * ((N + 255) / 256), (K + 63) / 64, sm_count() / 2);
}

// ------------------------------------------------------------------------------------------
// host launcher.  Pitches in BYTES.  For an MN-major operand the pointer addresses the
// [reduction, M-or-N] row-major matrix (i.e. the tensor as it lies in memory).
// ------------------------------------------------------------------------------------------
template <class Cfg, class Epi>
int launch_gemm2(const void* A, const void* B, void* D, int M, int N, int K, int64_t lda_bytes, int64_t ldb_bytes,
                 int64_t ldd_bytes, const typename Epi::Params& ep, int n_splits, cudaStream_t stream,
                 Sched sc = Sched{0, 1, 0}, float* ws = nullptr) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  CUtensorMap tmA, tmB, tmD;
  if (Cfg::A_MN ? make_tmap_kmajor(&tmA, A, K, M, lda_bytes, 64, 2) : make_tmap_kmajor(&tmA, A, M, K, lda_bytes, Cfg::CTA_M, 2))
    return -2;
  if (Cfg::B_MN ? make_tmap_kmajor(&tmB, B, K, N, ldb_bytes, 64, 2) : make_tmap_kmajor(&tmB, B, N, K, ldb_bytes, Cfg::CTA_N, 2))
    return -3;
  if (Cfg::TMA_STORE) {
    if (make_tmap_kmajor(&tmD, D, M, N, ldd_bytes, 32, 2)) return -4;
  } else {
    tmD = tmA;
  }
  const int num_m_blocks = (M + Cfg::BLOCK_M - 1) / Cfg::BLOCK_M;
  const int num_n_blocks = (N + Cfg::BLOCK_N - 1) / Cfg::BLOCK_N;
  if (n_splits <= 0 || n_splits > num_n_blocks) n_splits = num_n_blocks;
  const int nb_per_split = (num_n_blocks + n_splits - 1) / n_splits;
  n_splits = (num_n_blocks + nb_per_split - 1) / nb_per_split;
  auto kern = gemm2_sm100_kernel<Cfg, Epi>;
  static bool attr_set = false;
  if (!attr_set) {
    PRL_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    attr_set = true;
  }
  int clusters = sm_count() / 2;
  const int total = num_m_blocks * n_splits;
  KSplit ks{0, 0, 0, nullptr};
  if constexpr (Epi::kFinish) {        // ws: room for the slots of plan_k_split(M, N, K); without it every tile is computed whole
    if (ws != nullptr && Cfg::BLOCK_N == 256 && n_splits == num_n_blocks) ks = plan_k_split(M, N, K);
    ks.ws = ws;
  }
  if (!ks.tiles && total < clusters) clusters = total;
  kern<<<2 * clusters, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(tmA, tmB, tmD, ep, M, N, K, num_m_blocks, num_n_blocks,
                                                               n_splits, nb_per_split, sc, ks);
  PRL_CUDA_CHECK(cudaGetLastError());
  if constexpr (Epi::kFinish) {
    if (ks.tiles) {
      split_finish_kernel<Epi><<<dim3(ks.tiles, 256 / kFinishRows), 256, 0, stream>>>(ep, ks, (K + Cfg::BLOCK_K - 1) / Cfg::BLOCK_K, M, N, num_m_blocks,
                                                                                     num_n_blocks, sc);
      PRL_CUDA_CHECK(cudaGetLastError());
    }
  }
  return 0;
}

}  // namespace prl
