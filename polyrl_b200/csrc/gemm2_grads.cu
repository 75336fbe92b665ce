// polyrl_b200 — both gradients of a linear layer in one launch of CTA pairs:
//
//   dX[T, K] = dY[T, N] · W[N, K]          dW[N, K] = dY[T, N]^T · X[T, K]
//
// (the input and weight gradients behind nn.Linear's backward, 3rdparty/verl/verl/workers/actor/dp_actor.py:86-273, and of the fused
// LM head, verl/utils/kernel/kernels.py:1571-1581; the mainloop is that of gemm2_sm100.cuh).
//
// As two launches each ends with a round of tiles that does not fill the chip: the head's dX [2503, 896] has 40 tiles for 74 SM pairs.
// Here one persistent grid works through both products.  The one with the longer reduction is dealt out first, round robin; the tiles of
// the other are dealt so that all pairs finish together (grad_schedule), which is a closed formula of the pair's number, so nothing is
// read or counted at run time.  Every tile is still summed by one pair, in the order that the separate products have.
// The head's [2503, 896] x 151936 in ten slices: 1470 -> 1296 us.  Two 0.5B blocks, 387 tokens: 200 -> 156 us.
#include "gemm2_sm100.cuh"

namespace prl {

// Pair c of C takes the long tiles c, c + C, ...; then `hi` short tiles if c < cut (it has one long tile more than the others), else `lo`.
struct GradSchedule {
  int pairs, n_long, n_short, cut, hi, lo;
};
__host__ __device__ __forceinline__ bool grad_item(const GradSchedule& g, int c, int k, bool& is_long, int& tile) {
  const int longs = c < g.n_long ? (g.n_long - 1 - c) / g.pairs + 1 : 0;
  is_long = k < longs;
  if (is_long) {
    tile = c + k * g.pairs;
    return true;
  }
  const int s = k - longs, others = g.pairs - g.cut;
  if (c < g.cut) {
    tile = g.lo * others + s * g.cut + c;
    return s < g.hi && tile < g.n_short;
  }
  tile = s * others + c - g.cut;
  return s < g.lo && tile < g.n_short;
}

struct GradProblem {
  int m_blocks, num_kb;
};
struct GradParams {
  GradProblem p[2];          // 0: dX, 1: dW
  int n_blocks, long_one;    // column blocks of both; which of the two is dealt out first
  int T, N, K;
  GradSchedule sched;
  float* dx32;               // fp32 dX: beta * dx32 + product; else the bf16 map is stored to
  int64_t ld32;
  float beta;
};

using GradCfg = Gemm2Cfg<256, false, true, true>;

template <bool ACC32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GradCfg::THREADS, 1)
gemm2_grads_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmD0,
                   const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmD1,
                   GradParams g) {
  using Cfg = GradCfg;
  constexpr int BN = 256, kStages = Cfg::STAGES;
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

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  // k-th tile of this pair: which product, its first row and column
  auto item = [&](int k, int& which, int& row0, int& col0) {
    bool is_long;
    int tile;
    if (!grad_item(g.sched, pair, k, is_long, tile)) return false;
    which = is_long ? g.long_one : g.long_one ^ 1;
    const WorkInfo wi = decode_work(tile, g.p[which].m_blocks, g.n_blocks, g.n_blocks, 1, Sched{0, 1, 0});
    row0 = wi.m_blk * Cfg::BLOCK_M;
    col0 = wi.n_begin * BN;
    return true;
  };

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA0); tma_prefetch_desc(&tmB0); tma_prefetch_desc(&tmA1); tma_prefetch_desc(&tmB1); tma_prefetch_desc(&tmD1);
    if constexpr (!ACC32) tma_prefetch_desc(&tmD0);
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
  int which, row0, col0;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int k = 0; item(k, which, row0, col0); ++k) {
        const int m0 = row0 + static_cast<int>(rank) * Cfg::CTA_M, n0 = col0 + static_cast<int>(rank) * Cfg::CTA_N;
        const CUtensorMap* tb = which ? &tmB1 : &tmB0;
        for (int kb = 0; kb < g.p[which].num_kb; ++kb) {
          mbar_wait(&empty_bar[stage], phase ^ 1);
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * Cfg::STAGE_BYTES);
          uint8_t* sa = smem_a + stage * Cfg::A_BYTES;
          uint8_t* sb = smem_b + stage * Cfg::B_BYTES;
          const int k0 = kb * Cfg::BLOCK_K;
          if (which == 0) {
            tma_load_2d_2sm(&tmA0, &full_bar[stage], sa, k0, m0, kEvictNormal);
          } else {
            tma_load_2d_2sm(&tmA1, &full_bar[stage], sa, m0, k0, kEvictNormal);
            tma_load_2d_2sm(&tmA1, &full_bar[stage], sa + 8192, m0 + 64, k0, kEvictNormal);
          }
          tma_load_2d_2sm(tb, &full_bar[stage], sb, n0, k0, kEvictNormal);
          tma_load_2d_2sm(tb, &full_bar[stage], sb + 8192, n0 + 64, k0, kEvictNormal);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {
      constexpr uint32_t id0 = umma_idesc_major(Cfg::BLOCK_M, BN, 1, 1, 0, 1), id1 = umma_idesc_major(Cfg::BLOCK_M, BN, 1, 1, 1, 1);
      constexpr uint32_t mn_step = (16 * 128) >> 4, k_step = 32 >> 4;      // descriptor units (16 B) per UMMA_K
      int stage = 0;
      uint32_t phase = 0;
      for (int k = 0; item(k, which, row0, col0); ++k) {
        const uint32_t as = k & 1;
        mbar_wait(&tmem_empty[as], ((k >> 1) & 1) ^ 1);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + as * BN;
        for (int kb = 0; kb < g.p[which].num_kb; ++kb) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint8_t* sa = smem_a + stage * Cfg::A_BYTES;
          const uint64_t db = umma_desc_sw128_mnmajor(smem_b + stage * Cfg::B_BYTES, 8192);
          if (which == 0) {
            const uint64_t da = umma_desc_sw128_kmajor(sa);
#pragma unroll
            for (int q = 0; q < Cfg::BLOCK_K / 16; ++q) umma_bf16_ss_2sm(tmem_d, da + q * k_step, db + q * mn_step, id0, (kb | q) != 0);
          } else {
            const uint64_t da = umma_desc_sw128_mnmajor(sa, 8192);
#pragma unroll
            for (int q = 0; q < Cfg::BLOCK_K / 16; ++q) umma_bf16_ss_2sm(tmem_d, da + q * mn_step, db + q * mn_step, id1, (kb | q) != 0);
          }
          umma_commit_2sm(&empty_bar[stage], 3);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        umma_commit_2sm(&tmem_full[as], 3);
      }
    }
  } else {
    const int quad = warp & 3;                       // TMEM lane quadrant this warp may read
    uint8_t* ebuf = smem_epi + (warp - 2) * 8192;
    uint32_t chunk_ctr = 0;
    for (int k = 0; item(k, which, row0, col0); ++k) {
      const uint32_t as = k & 1;
      const int first = row0 + static_cast<int>(rank) * Cfg::CTA_M + quad * 32, rows = which ? g.N : g.T;
      mbar_wait(&tmem_full[as], (k >> 1) & 1);
      tc_fence_after();
      const uint32_t taddr = tmem_base + as * BN + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN; c += 64) {
        uint32_t r[64];
        __syncwarp();
        tmem_ld_32x32(taddr + c, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
        tmem_ld_32x32(taddr + c + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
        tmem_ld_wait();
        if (c == BN - 64) {                          // accumulator fully read: hand TMEM back early
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(&tmem_empty[as], 0);
        }
        const int col = col0 + c;
        if (ACC32 && which == 0) {
          if (first + lane < rows) {
            float* dst = g.dx32 + static_cast<int64_t>(first + lane) * g.ld32 + col;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (col + 4 * j >= g.K) continue;      // (K is a multiple of 8)
              float4 o = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
              if (g.beta != 0.f) {
                const float4 q = *reinterpret_cast<const float4*>(dst + 4 * j);
                o.x += g.beta * q.x; o.y += g.beta * q.y; o.z += g.beta * q.z; o.w += g.beta * q.w;
              }
              *reinterpret_cast<float4*>(dst + 4 * j) = o;
            }
          }
          continue;
        }
        uint8_t* buf = ebuf + (chunk_ctr++ & 1) * 4096;
        if (lane == 0) tma_store_wait_read<1>();     // the store that last read `buf` has drained it
        __syncwarp();
        // row `lane` of the 32 x 64 box: 8 x 16 B chunks, chunk j lands at (j ^ (lane & 7)) (128B swizzle)
        const uint32_t row_base = smem_u32(buf) + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t q[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) q[e] = pack_bf16(__uint_as_float(r[8 * j + 2 * e]), __uint_as_float(r[8 * j + 2 * e + 1]));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_base + ((j ^ (lane & 7)) << 4)), "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3])
                       : "memory");
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (first < rows && col < g.K) tma_store_2d(which ? &tmD1 : &tmD0, buf, col, first);   // TMA clips partial boxes
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  cluster_sync_all();            // nobody leaves while the peer may still read its smem / signal its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, Cfg::TMEM_COLS);
  }
}

// Short tiles for the pairs with and without an extra long one, so that the latest pair is done as early as can be.  A tile counts for its
// k-blocks and four more, the part of its epilogue that the next tile does not hide.
static GradSchedule grad_schedule(int n_long, int kb_long, int n_short, int kb_short, int pairs) {
  GradSchedule g{pairs, n_long, n_short, n_long % pairs, 0, 0};
  const int64_t a = kb_long + 4, b = kb_short + 4, base = n_long / pairs, others = pairs - g.cut;
  int64_t best = INT64_MAX;
  for (int64_t hi = 0; hi == 0 || (g.cut > 0 && (hi - 1) * g.cut < n_short); ++hi) {
    const int64_t left = n_short > hi * g.cut ? n_short - hi * g.cut : 0, lo = (left + others - 1) / others;
    const int64_t t_hi = g.cut > 0 ? (base + 1) * a + hi * b : 0, t_lo = base * a + lo * b, t = t_hi > t_lo ? t_hi : t_lo;
    if (t < best) { best = t; g.hi = static_cast<int>(hi); g.lo = static_cast<int>(lo); }
  }
  return g;
}

// Time of one of the products by itself, in k-blocks: whole rounds, or the cut of plan_k_split (in its terms: a k-block 0.3 us, 3 us and
// 0.25 us a slot for the second kernel).
static double single_cost(const GradProblem& p, int n_blocks, int pairs) {
  const int64_t tiles = static_cast<int64_t>(p.m_blocks) * n_blocks;
  const KSplit ks = plan_k_split(tiles, p.num_kb, pairs);
  if (!ks.tiles) return static_cast<double>((tiles + pairs - 1) / pairs) * (p.num_kb + 4);
  return static_cast<double>(ks.full / pairs) * (p.num_kb + 4) + static_cast<double>(p.num_kb) * ks.tiles / ks.workers +
         (3.0 + 0.25 * (ks.workers + ks.tiles)) / 0.3;
}

}  // namespace prl

using namespace prl;

// Is the joint launch the faster one?  Not where few long tiles hold it up which the separate product would cut along the reduction
// (387 tokens: dX of [387, 9728] x 896 is eight tiles of 152 k-blocks), and not for large products: two working sets share the L2 then, and
// what their rounds would save (4% at 12287 tokens of an 8B block) is lost twice over (7.6 -> 8.4 ms).  It has to promise a tenth; the second
// launch counts for 3 us.
extern "C" int prl_gemm2_grads_joint(int T, int N, int K) {
  const GradProblem p[2] = {{(T + 255) / 256, (N + 63) / 64}, {(N + 255) / 256, (T + 63) / 64}};
  const int nb = (K + 255) / 256, sms = sm_count() / 2, l = p[1].num_kb > p[0].num_kb ? 1 : 0;
  const int64_t tiles = static_cast<int64_t>(p[0].m_blocks + p[1].m_blocks) * nb;
  if (K <= 128 || N <= 128 || tiles > 0x3fffffff) return 0;       // (tiles half as wide then: the separate kernels have them)
  const int pairs = static_cast<int>(tiles < sms ? tiles : sms);
  const GradSchedule g = grad_schedule(p[l].m_blocks * nb, p[l].num_kb, p[l ^ 1].m_blocks * nb, p[l ^ 1].num_kb, pairs);
  const double a = p[l].num_kb + 4, b = p[l ^ 1].num_kb + 4, base = g.n_long / pairs;
  const double hi = g.cut > 0 ? (base + 1) * a + g.hi * b : 0, lo = base * a + g.lo * b;
  return 1.1 * (hi > lo ? hi : lo) <= single_cost(p[0], nb, sms) + single_cost(p[1], nb, sms) + 10;
}

// dY [T, N], W [N, K], X [T, K] bf16, pitches in elements (multiples of 8, 16-byte aligned bases); N and K multiples of 8.
// dX: bf16 at dx (pitch lddx), or fp32 at dx32 = beta * dx32 + product (pitch ld32, a multiple of 4); dW: bf16 (pitch lddw).
extern "C" int prl_gemm2_grads(const void* dy, const void* w, const void* x, void* dx, float* dx32, float beta, void* dw, int T, int N, int K, int64_t lddy,
                               int64_t ldw, int64_t ldx, int64_t lddx, int64_t ld32, int64_t lddw, cudaStream_t stream) {
  if (T <= 0 || N <= 0 || K <= 0) return -30;
  using Cfg = GradCfg;
  CUtensorMap a0, b0, d0, a1, b1, d1;
  if (make_tmap_kmajor(&a0, dy, T, N, lddy * 2, Cfg::CTA_M, 2)) return -31;
  if (make_tmap_kmajor(&b0, w, N, K, ldw * 2, 64, 2)) return -32;
  if (make_tmap_kmajor(&a1, dy, T, N, lddy * 2, 64, 2)) return -33;
  if (make_tmap_kmajor(&b1, x, T, K, ldx * 2, 64, 2)) return -34;
  if (make_tmap_kmajor(&d1, dw, N, K, lddw * 2, 32, 2)) return -35;
  d0 = d1;
  if (dx32 == nullptr && make_tmap_kmajor(&d0, dx, T, K, lddx * 2, 32, 2)) return -36;
  GradParams g{};
  g.p[0] = {(T + 255) / 256, (N + 63) / 64};
  g.p[1] = {(N + 255) / 256, (T + 63) / 64};
  g.n_blocks = (K + 255) / 256;
  g.T = T; g.N = N; g.K = K;
  g.dx32 = dx32; g.ld32 = ld32; g.beta = beta;
  g.long_one = g.p[1].num_kb > g.p[0].num_kb ? 1 : 0;
  const GradProblem lo = g.p[g.long_one], sh = g.p[g.long_one ^ 1];
  const int64_t tiles = static_cast<int64_t>(lo.m_blocks + sh.m_blocks) * g.n_blocks;
  if (tiles > 0x3fffffff) return -37;
  const int pairs = static_cast<int>(tiles < sm_count() / 2 ? tiles : sm_count() / 2);
  g.sched = grad_schedule(lo.m_blocks * g.n_blocks, lo.num_kb, sh.m_blocks * g.n_blocks, sh.num_kb, pairs);
  static bool attr = false;
  if (!attr) {
    PRL_CUDA_CHECK(cudaFuncSetAttribute(gemm2_grads_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    PRL_CUDA_CHECK(cudaFuncSetAttribute(gemm2_grads_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    attr = true;
  }
  if (dx32 != nullptr) gemm2_grads_kernel<true><<<2 * pairs, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(a0, b0, d0, a1, b1, d1, g);
  else gemm2_grads_kernel<false><<<2 * pairs, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(a0, b0, d0, a1, b1, d1, g);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
