// polyrl_b200 — varlen causal flash-attention BACKWARD on tcgen05 / TMEM / TMA (head_dim 64 or 128, GQA).
//
// Replaces flash-attn 2's backward (reference: the autograd of `_flash_attention_forward`,
// 3rdparty/verl/verl/models/transformers/monkey_patch.py:49-117).
//
// Two kernels, each of which owns what it writes, so nothing is added up in memory:
//   keys:     item = (128-key tile of one sequence, one KV head), walks every query head of the GQA group and every query tile that
//             sees these keys.  Scores are computed transposed, lanes = keys:
//                 S^T = K Q^T,  dP^T = V dO^T,  P^T = exp2(S^T c - lse),  dS^T = P^T (dP^T - D) sm_scale
//                 dV += P^T dO    A = P^T in TMEM, over the columns of S^T         B = dO (MN-major)
//                 dK += dS^T Q    A = dS^T in shared memory (K-major)              B = Q  (MN-major)
//   queries:  item = (128-row query tile, one head), walks the key tiles; lanes = queries:
//                 S = Q K^T,  dP = dO V^T,  dS as above,   dQ += dS K              A = dS in TMEM, over the columns of S;  B = K (MN-major)
// S and dP are computed twice (7 products a tile pair instead of 5).  The one-kernel form added dQ with fp32 reductions in global memory,
// 64 KB a tile pair, had one stage of Q and dO and waited for each step in turn.
// Both run one CTA an SM over many items: operands arrive through two stages, the next pair's scores are multiplied while the warps work
// on this one, an item's first loads run under the end of the one before, and results leave through shared memory in whole 64-byte pieces.
// 32 heads of 128 over 8, causal, 19 sequences of 647: as the one-kernel form when it was written, 637 us before and 623 with products that end
// at the sequence's last row; 16 heads over 8, 9 sequences of 455: 132 -> 101 us a call; head width 64 took a library (two 0.5B blocks,
// 387 tokens: 1870 -> 1365 us, most of it on the host).
#include "common.cuh"

namespace prl {

constexpr int kAbThreads = 320;          // warp 0 TMA, warp 1 MMA, warps 2-9: two warpgroups, each half of a tile's score columns

struct AttnBwdParams {
  __nv_bfloat16* dq;           // [Tq, nq*D], row pitch lddq
  __nv_bfloat16* dk;           // [Tk, nkv*D], row pitch lddkv
  __nv_bfloat16* dv;
  int64_t lddq, lddkv;
  const float2* stats;         // [nq, Tq]   (log-sum-exp in base 2, D = rowsum(dO * O))
  const int32_t* cu_q;
  const int32_t* cu_k;
  int B, nq, nkv, Tq;
  float scale_log2, sm_scale;
  int causal;
};

int af_tmap(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld_bytes, uint32_t box_rows);

// a 128-row tile of D columns, as chunks of 64 columns (16 KB each, 128-byte swizzle)
template <int D>
__device__ __forceinline__ void load_tile(const CUtensorMap* m, uint64_t* bar, uint8_t* dst, int col, int row) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) tma_load_2d(m, bar, dst + c * 16384, col + c * 64, row);
}
// acc = A B^T over D columns, both tiles K-major
template <int D>
__device__ __forceinline__ void mma_scores(uint32_t acc, const uint8_t* a, const uint8_t* b) {
  constexpr uint32_t id = umma_idesc(128, 128, 1, 1);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
    umma_bf16_ss(acc, umma_desc_sw128_kmajor(a + (kk >> 2) * 16384) + 2 * (kk & 3), umma_desc_sw128_kmajor(b + (kk >> 2) * 16384) + 2 * (kk & 3), id, kk != 0);
}
// acc (+)= A B over the `left` rows of B, with A [128, 128] as bf16 in TMEM (columns 64 g .. 64 g + 31 hold columns 64 g .. 64 g + 63),
// B [128, D] read MN-major
template <int D>
__device__ __forceinline__ void mma_from_tmem(uint32_t acc, uint32_t a, const uint8_t* b, bool add, int left) {
  constexpr uint32_t id = umma_idesc_major(128, D, 1, 1, 0, 1);
  for_row_steps(left, [&](int kk) {
    umma_bf16_ts(acc, a + (kk >> 2) * 64 + 8 * (kk & 3), umma_desc_sw128_mnmajor(b, 16384) + kk * 128, id, add || kk != 0);
  });
}
// 32 fp32 columns of a warp's 32 TMEM rows -> bf16 rows in memory, through 2 KB of shared memory; row `lane` of the warp is valid if
// lane < rows.  any = false: zeros.
__device__ __forceinline__ void store_acc32(uint32_t taddr, uint32_t stage, __nv_bfloat16* dst, int64_t ld, int rows, bool any) {
  const int lane = threadIdx.x & 31;
  uint32_t a[32];
  __syncwarp();
  if (any) {
    tmem_ld_32x32(taddr, a);
    tmem_ld_wait();
  } else {
#pragma unroll
    for (int e = 0; e < 32; ++e) a[e] = 0;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint32_t q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) q[e] = pack_bf16(__uint_as_float(a[8 * u + 2 * e]), __uint_as_float(a[8 * u + 2 * e + 1]));
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + lane * 64 + ((u ^ (lane >> 1 & 3)) << 4)), "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3])
                 : "memory");
  }
  __syncwarp();
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int row = 8 * g + (lane >> 2);
    int4 q;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                 : "r"(stage + row * 64 + (((lane & 3) ^ (row >> 1 & 3)) << 4)) : "memory");
    if (row < rows) st_v4(dst + row * ld + (lane & 3) * 8, q);
  }
}

template <int D>
struct AbkCfg {
  static constexpr int T = 128 * D * 2;                                // one operand tile
  // K, V, two stages of Q and dO, dS^T, two stages of row statistics, barriers.  At D = 128 this is all of the 227 KB but for 896 bytes,
  // which align the base to 1024 from the 128 that it has at least (nothing else in this kernel lies in shared memory).
  static constexpr int SMEM = 6 * T + 32768 + 2048 + 128 + 896;
};

template <int D>
__global__ void __launch_bounds__(kAbThreads, 1)
attn_bwd_keys_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int T = AbkCfg<D>::T;
  uint8_t* sK = smem;
  uint8_t* sV = smem + T;
  uint8_t* sQ = smem + 2 * T;         // [2]
  uint8_t* sdO = smem + 4 * T;        // [2]
  uint8_t* sdS = smem + 6 * T;        // [128 keys][128 queries], two chunks of 64 queries; a warp's own rows stage its results
  float* stat = reinterpret_cast<float*>(sdS + 32768);                 // [2 stages][lse2 | D][128 queries]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sdS + 32768 + 2048);
  uint64_t* k_full = bars;            // TMA
  uint64_t* v_full = bars + 1;        // TMA
  uint64_t* q_full = bars + 2;        // [2] TMA
  uint64_t* do_full = bars + 4;       // [2] TMA
  uint64_t* s_full = bars + 6;        // commit: S^T (behind an item's last, K may be overwritten)
  uint64_t* dp_full = bars + 7;       // commit: dP^T (and V)
  uint64_t* p_full = bars + 8;        // 256 arrivals: P^T in TMEM
  uint64_t* ds_full = bars + 9;       // 256 arrivals: dS^T in shared memory, dP^T read
  // one per stage: the producer asks for the use of two tiles ago, and the next tile's may be over by then
  uint64_t* dv_done = bars + 10;      // [2] commit: P^T and dO consumed
  uint64_t* dk_done = bars + 12;      // [2] commit: dS^T and Q consumed
  uint64_t* acc_free = bars + 14;     // 256 arrivals: the item's dK and dV have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.nq / p.nkv;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
    for (int i = 0; i < 15; ++i) mbar_init(bars + i, i == 8 || i == 9 || i == 14 ? 256 : 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 384;

  struct Item {
    int hk, k0, qs, lq, ks, lk, off, i0, n_i, iters;
  };
  // item w (all of a warp asks): false behind the last one.  KV heads of a tile are neighbours.
  auto item = [&](int w, Item& t) {
    int k0 = 0;
    const int seq = find_row_tile(p.cu_k, p.B, w / p.nkv, &k0);
    if (seq < 0) return false;
    t.hk = w % p.nkv; t.k0 = k0;
    t.qs = p.cu_q[seq]; t.lq = p.cu_q[seq + 1] - t.qs;
    t.ks = p.cu_k[seq]; t.lk = p.cu_k[seq + 1] - t.ks;
    t.off = t.lk - t.lq;
    t.i0 = p.causal ? max(0, (k0 - t.off) / 128) : 0;                  // first query tile whose LAST row can see key k0:  row + off >= k0
    t.n_i = max(0, (t.lq + 127) / 128 - t.i0);
    t.iters = t.n_i * G;
    return true;
  };
  Item t;
  int n = 0, i = 0;                   // tile pairs and items (with any) so far: the barriers' phases

  if (warp == 0) {
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      if (t.iters == 0) continue;
      if (lane == 0) {
        for (int it = 0; it < t.iters; ++it, ++n) {
          const int h = t.hk * G + it / t.n_i, row = t.qs + (t.i0 + it % t.n_i) * 128, s = n & 1;
          const uint32_t before = ((n - 2) >> 1) & 1;
          // The scores of the last pair are waited for at every pair, not only where K changes: a parity tells the last completion from the
          // one before, so a wait must never be two behind or ahead.  (They are done by the time dK of two pairs ago is.)
          if (n > 0) mbar_wait(s_full, (n - 1) & 1);
          if (it == 0) {
            mbar_expect_tx(k_full, T);
            load_tile<D>(&tmK, k_full, sK, t.hk * D, t.ks + t.k0);
          }
          if (n >= 2) mbar_wait(&dk_done[s], before);
          mbar_expect_tx(&q_full[s], T);
          load_tile<D>(&tmQ, &q_full[s], sQ + s * T, h * D, row);
          if (n > 0) mbar_wait(dp_full, (n - 1) & 1);
          if (it == 0) {
            mbar_expect_tx(v_full, T);
            load_tile<D>(&tmV, v_full, sV, t.hk * D, t.ks + t.k0);
          }
          if (n >= 2) mbar_wait(&dv_done[s], before);
          mbar_expect_tx(&do_full[s], T);
          load_tile<D>(&tmdO, &do_full[s], sdO + s * T, h * D, row);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idKM = umma_idesc_major(128, D, 1, 1, 0, 1);               // A K-major, B MN-major
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      if (t.iters == 0) continue;
      // All lanes wait, for they clear rows, and meet before lane 0 issues anything: a lane that were still asking for a phase when the next
      // one is over would wait for good.
      // rows of the item's it-th query tile that are its sequence's
      auto left = [&](int it) { return min(t.lq - (t.i0 + it % t.n_i) * 128, 128); };
      auto scores = [&](int m, int it) {                  // S^T of pair m: P^T of the one before is consumed
        mbar_wait(&q_full[m & 1], (m >> 1) & 1);
        if (left(it) & 15) clear_rows<D>(sQ + (m & 1) * T, left(it));
        if (m > 0) mbar_wait(&dv_done[(m - 1) & 1], ((m - 1) >> 1) & 1);
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_scores<D>(tS, sK, sQ + (m & 1) * T);
          umma_commit(s_full);
        }
      };
      auto operand = [&](int m, int it) {                 // dO of pair m
        mbar_wait(&do_full[m & 1], (m >> 1) & 1);
        if (left(it) & 15) clear_rows<D>(sdO + (m & 1) * T, left(it));
      };
      auto products = [&](int m) {                        // dP^T of pair m: that of the one before has been read (ds_full)
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_scores<D>(tdP, sV, sdO + (m & 1) * T);
          umma_commit(dp_full);
        }
      };
      mbar_wait(k_full, i & 1);
      scores(n, 0);
      operand(n, 0);
      mbar_wait(v_full, i & 1);
      products(n);
      for (int it = 0; it < t.iters; ++it, ++n) {
        const int s = n & 1;
        mbar_wait(p_full, n & 1);
        if (it == 0 && i > 0) mbar_wait(acc_free, (i - 1) & 1);
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_from_tmem<D>(tdV, tS, sdO + s * T, it != 0, left(it));   // dV += P^T dO
          umma_commit(&dv_done[s]);
        }
        if (it + 1 < t.iters) {
          scores(n + 1, it + 1);
          operand(n + 1, it + 1);
        }
        mbar_wait(ds_full, n & 1);
        tc_fence_after();
        if (it + 1 < t.iters) products(n + 1);
        __syncwarp();
        if (lane == 0) {
          for_row_steps(left(it), [&](int kk) {                                   // dK += dS^T Q  (reduction over the query rows)
            umma_bf16_ss(tdK, umma_desc_sw128_kmajor(sdS + (kk >> 2) * 16384) + 2 * (kk & 3), umma_desc_sw128_mnmajor(sQ + s * T, 16384) + kk * 128, idKM,
                         (it | kk) != 0);
          });
          umma_commit(&dk_done[s]);
        }
        __syncwarp();
      }
      ++i;
    }
  } else {
    const int g = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                       // key row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t sdS_u32 = smem_u32(sdS) + g * 16384 + r * 128, stage = smem_u32(sdS) + g * 16384 + quad * 4096;
    const int tid = threadIdx.x - 64;
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      const int key = t.k0 + r;
      // thread tid brings statistic tid >> 7 of query tid & 127, one tile ahead
      auto fetch = [&](int h, int tile) {
        const int q = tile * 128 + (tid & 127);
        if (q >= t.lq) return 0.f;
        return reinterpret_cast<const float*>(p.stats + static_cast<int64_t>(h) * p.Tq + t.qs + q)[tid >> 7];
      };
      const int tiles_end = t.i0 + t.n_i;
      int tile = t.i0, h_next = t.hk * G, tile_next = t.i0;
      float ahead = t.iters > 0 ? fetch(h_next, tile_next) : 0.f;
      for (int it = 0; it < t.iters; ++it, ++n, tile = tile_next) {
        const int q0 = tile * 128;
        if (++tile_next == tiles_end) { tile_next = t.i0; ++h_next; }
        float* st = stat + (n & 1) * 256;
        st[tid] = ahead;
        asm volatile("bar.sync 1, 256;" ::: "memory");    // (a stage is overwritten two tiles later: everyone has passed the barrier between)
        if (it + 1 < t.iters) ahead = fetch(h_next, tile_next);
        const bool whole = q0 + 127 < t.lq && t.k0 + 127 < t.lk && (!p.causal || t.k0 + 127 <= q0 + t.off);
        // this thread's 64 queries that see its key: [seen_lo, seen_lo + seen_n)
        const int seen_lo = p.causal ? max(0, key - t.off - q0 - g * 64) : 0;
        const unsigned seen_n = key < t.lk ? max(0, min(64, t.lq - q0 - g * 64) - seen_lo) : 0;
        float pv[64];
        mbar_wait(s_full, n & 1);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t v[32], pk[16];
          __syncwarp();
          tmem_ld_32x32(tS + lane_base + g * 64 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 l = *reinterpret_cast<const float4*>(st + g * 64 + c + e);
            pv[c + e] = __uint_as_float(v[e]) * p.scale_log2 - l.x;
            pv[c + e + 1] = __uint_as_float(v[e + 1]) * p.scale_log2 - l.y;
            pv[c + e + 2] = __uint_as_float(v[e + 2]) * p.scale_log2 - l.z;
            pv[c + e + 3] = __uint_as_float(v[e + 3]) * p.scale_log2 - l.w;
          }
          if (!whole) {
#pragma unroll
            for (int e = 0; e < 32; ++e) pv[c + e] = static_cast<unsigned>(c + e - seen_lo) < seen_n ? pv[c + e] : -INFINITY;
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) pv[c + e] = fast_exp2(pv[c + e]);
#pragma unroll
          for (int e = 0; e < 16; ++e) pk[e] = pack_bf16(pv[c + 2 * e], pv[c + 2 * e + 1]);
          tmem_st_32x16(tS + lane_base + g * 64 + (c >> 1), pk);    // (over scores that this thread has read)
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(p_full);
        mbar_wait(dp_full, n & 1);
        tc_fence_after();
        if (n > 0) mbar_wait(&dk_done[(n - 1) & 1], ((n - 1) >> 1) & 1);           // dS^T of the last tile has been read
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(tdP + lane_base + g * 64 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 d = *reinterpret_cast<const float4*>(st + 128 + g * 64 + c + e);
            pv[c + e] *= (__uint_as_float(v[e]) - d.x) * p.sm_scale;
            pv[c + e + 1] *= (__uint_as_float(v[e + 1]) - d.y) * p.sm_scale;
            pv[c + e + 2] *= (__uint_as_float(v[e + 2]) - d.z) * p.sm_scale;
            pv[c + e + 3] *= (__uint_as_float(v[e + 3]) - d.w) * p.sm_scale;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float* f = pv + c + 8 * q;
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sdS_u32 + ((((c >> 3) + q) ^ (r & 7)) << 4)), "r"(pack_bf16(f[0], f[1])),
                         "r"(pack_bf16(f[2], f[3])), "r"(pack_bf16(f[4], f[5])), "r"(pack_bf16(f[6], f[7]))
                         : "memory");
          }
        }
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive(ds_full);
      }
      const bool any = t.iters > 0;
      if (any) {
        mbar_wait(&dk_done[(n - 1) & 1], ((n - 1) >> 1) & 1);        // (the last dV product was issued before the last dK product)
        tc_fence_after();
      }
      const int64_t at = static_cast<int64_t>(t.ks + t.k0 + quad * 32) * p.lddkv + t.hk * D + g * (D / 2);
      const int rows = t.lk - t.k0 - quad * 32;
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        store_acc32(tdK + lane_base + g * (D / 2) + c, stage, p.dk + at + c, p.lddkv, rows, any);
        store_acc32(tdV + lane_base + g * (D / 2) + c, stage, p.dv + at + c, p.lddkv, rows, any);
      }
      if (any) {
        tc_fence_before();
        mbar_arrive(acc_free);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

template <int D>
struct AbqCfg {
  static constexpr int T = 128 * D * 2;
  static constexpr int SMEM = 6 * T + 8 * 2048 + 256 + 1024;        // Q, dO, two stages of K and V, staging of the results
};

template <int D>
__global__ void __launch_bounds__(kAbThreads, 1)
attn_bwd_queries_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int T = AbqCfg<D>::T;
  uint8_t* sQ = smem;
  uint8_t* sdO = smem + T;
  uint8_t* sK = smem + 2 * T;         // [2]
  uint8_t* sV = smem + 4 * T;         // [2]
  uint8_t* sOut = smem + 6 * T;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + 8 * 2048);
  uint64_t* q_full = bars;            // TMA
  uint64_t* do_full = bars + 1;       // TMA
  uint64_t* k_full = bars + 2;        // [2] TMA
  uint64_t* v_full = bars + 4;        // [2] TMA
  uint64_t* s_full = bars + 6;        // [2] commit: S
  uint64_t* dp_full = bars + 8;       // commit: dP
  uint64_t* ds_full = bars + 9;       // 256 arrivals: dS in TMEM, dP read
  // one per stage: the producer asks for the use of two tiles ago, and the next tile's may be over by then
  uint64_t* v_done = bars + 10;       // [2] commit: V (and behind an item's last, Q and dO) consumed
  uint64_t* dq_done = bars + 12;      // [2] commit: dS and K consumed
  uint64_t* acc_free = bars + 14;     // 256 arrivals: the item's dQ has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
    for (int i = 0; i < 15; ++i) mbar_init(bars + i, i == 9 || i == 14 ? 256 : 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tdP = tmem_base + 256, tdQ = tmem_base + 384;      // S: two buffers

  struct Item {
    int h, q0, qs, lq, ks, lk, off, nt;
  };
  auto item = [&](int w, Item& t) {                       // (as in the other kernel; heads of a tile are neighbours)
    int q0 = 0;
    const int seq = find_row_tile(p.cu_q, p.B, w / p.nq, &q0);
    if (seq < 0) return false;
    t.h = w % p.nq; t.q0 = q0;
    t.qs = p.cu_q[seq]; t.lq = p.cu_q[seq + 1] - t.qs;
    t.ks = p.cu_k[seq]; t.lk = p.cu_k[seq + 1] - t.ks;
    t.off = t.lk - t.lq;
    t.nt = max(0, ((p.causal ? min(t.lk, q0 + 128 + t.off) : t.lk) + 127) / 128);
    return true;
  };
  Item t;
  int n = 0, i = 0;                   // key tiles and items (with any) so far: the barriers' phases

  if (warp == 0) {
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      if (t.nt == 0) continue;
      if (lane == 0) {
        const int hk = t.h / (p.nq / p.nkv);
        for (int j = 0; j < t.nt; ++j, ++n) {
          const int s = n & 1, row = t.ks + j * 128;
          const uint32_t before = ((n - 2) >> 1) & 1;
          if (j == 0) {                                   // the last dP was issued behind the last S
            if (n > 0) mbar_wait(&v_done[(n - 1) & 1], ((n - 1) >> 1) & 1);
            mbar_expect_tx(q_full, T);
            load_tile<D>(&tmQ, q_full, sQ, t.h * D, t.qs + t.q0);
          }
          if (n >= 2) mbar_wait(&dq_done[s], before);
          mbar_expect_tx(&k_full[s], T);
          load_tile<D>(&tmK, &k_full[s], sK + s * T, hk * D, row);
          if (j == 0) {
            mbar_expect_tx(do_full, T);
            load_tile<D>(&tmdO, do_full, sdO, t.h * D, t.qs + t.q0);
          }
          if (n >= 2) mbar_wait(&v_done[s], before);
          mbar_expect_tx(&v_full[s], T);
          load_tile<D>(&tmV, &v_full[s], sV + s * T, hk * D, row);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      if (t.nt == 0) continue;
      auto left = [&](int j) { return min(t.lk - j * 128, 128); };                // keys of tile j that are the sequence's
      auto scores = [&](int m, int j) {                   // S of tile m, over dS of tile m - 2
        const int s = m & 1;
        mbar_wait(&k_full[s], (m >> 1) & 1);
        if (left(j) & 15) clear_rows<D>(sK + s * T, left(j));
        if (m >= 2) mbar_wait(&dq_done[s], ((m - 2) >> 1) & 1);
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_scores<D>(tS + s * 128, sQ, sK + s * T);
          umma_commit(&s_full[s]);
        }
      };
      auto operand = [&](int m, int j) {                  // V of tile m
        mbar_wait(&v_full[m & 1], (m >> 1) & 1);
        if (left(j) & 15) clear_rows<D>(sV + (m & 1) * T, left(j));
      };
      auto products = [&](int m) {                        // dP of tile m: that of the one before has been read (ds_full)
        const int s = m & 1;
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_scores<D>(tdP, sdO, sV + s * T);
          umma_commit(dp_full);
          umma_commit(&v_done[s]);
        }
      };
      mbar_wait(q_full, i & 1);
      scores(n, 0);
      operand(n, 0);
      mbar_wait(do_full, i & 1);
      products(n);
      for (int j = 0; j < t.nt; ++j, ++n) {
        const int s = n & 1;
        if (j + 1 < t.nt) {
          scores(n + 1, j + 1);
          operand(n + 1, j + 1);
        }
        mbar_wait(ds_full, n & 1);
        tc_fence_after();
        if (j + 1 < t.nt) products(n + 1);
        if (j == 0 && i > 0) mbar_wait(acc_free, (i - 1) & 1);
        tc_fence_after();
        __syncwarp();
        if (lane == 0) {
          mma_from_tmem<D>(tdQ, tS + s * 128, sK + s * T, j != 0, left(j));      // dQ += dS K
          umma_commit(&dq_done[s]);
        }
        __syncwarp();
      }
      ++i;
    }
  } else {
    const int g = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                       // query row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t stage = smem_u32(sOut) + (warp - 2) * 2048;
    for (int w = blockIdx.x; item(w, t); w += gridDim.x) {
      const int qrow = t.q0 + r;
      const float2 st = qrow < t.lq ? p.stats[static_cast<int64_t>(t.h) * p.Tq + t.qs + qrow] : make_float2(INFINITY, 0.f);
      const int kmax = p.causal ? min(qrow + t.off, t.lk - 1) : t.lk - 1, kmin = p.causal ? min(t.q0 + t.off, t.lk - 1) : t.lk - 1;
      for (int j = 0; j < t.nt; ++j, ++n) {
        const int s = n & 1, base = j * 128 + g * 64;
        float pv[64];
        mbar_wait(&s_full[s], (n >> 1) & 1);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(tS + s * 128 + lane_base + g * 64 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) pv[c + e] = __uint_as_float(v[e]) * p.scale_log2 - st.x;
        }
        if (base + 63 > kmin) {                           // (the same for the whole warpgroup)
          const int in = kmax - base;
#pragma unroll
          for (int e = 0; e < 64; ++e) pv[e] = e <= in ? pv[e] : -INFINITY;
        }
#pragma unroll
        for (int e = 0; e < 64; ++e) pv[e] = fast_exp2(pv[e]);
        mbar_wait(dp_full, n & 1);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t v[32], pk[16];
          __syncwarp();
          tmem_ld_32x32(tdP + lane_base + g * 64 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) pv[c + e] *= (__uint_as_float(v[e]) - st.y) * p.sm_scale;
#pragma unroll
          for (int e = 0; e < 16; ++e) pk[e] = pack_bf16(pv[c + 2 * e], pv[c + 2 * e + 1]);
          tmem_st_32x16(tS + s * 128 + lane_base + g * 64 + (c >> 1), pk);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(ds_full);
      }
      const bool any = t.nt > 0;
      if (any) {
        mbar_wait(&dq_done[(n - 1) & 1], ((n - 1) >> 1) & 1);
        tc_fence_after();
      }
      __nv_bfloat16* dst = p.dq + static_cast<int64_t>(t.qs + t.q0 + quad * 32) * p.lddq + t.h * D + g * (D / 2);
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) store_acc32(tdQ + lane_base + g * (D / 2) + c, stage, dst + c, p.lddq, t.lq - t.q0 - quad * 32, any);
      if (any) {
        tc_fence_before();
        mbar_arrive(acc_free);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// stats[h, t] = (lse in base 2, D = sum_d dO[t, h, d] * O[t, h, d]).  A warp takes 32 tokens of one head, D / 8 threads a row, with 16-byte
// loads; what it writes is 256 contiguous bytes.  Rows that belong to no sequence get a zero gradient here.
template <int D>
__global__ void __launch_bounds__(256)
attn_stats_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, int64_t ldo, int64_t lddo,
                  const float* __restrict__ lse, float2* __restrict__ stats, __nv_bfloat16* __restrict__ dq, int64_t lddq,
                  const int32_t* __restrict__ cu_q, int B, int Tq, int nq) {
  constexpr int L = D / 8, R = 32 / L;
  const int lane = threadIdx.x & 31, l = lane % L, w = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int h = w % nq, t0 = w / nq * 32;
  if (t0 >= Tq) return;
  const int begin = cu_q[0], end = cu_q[B];
  float mine = 0.f;
#pragma unroll 8
  for (int k = 0; k < 32 / R; ++k) {
    const int in = k * R + lane / L, t = t0 + in;
    float s = 0.f;
    if (t < Tq) {
      const int4 a = ld_nc_v4(o + static_cast<int64_t>(t) * ldo + h * D + l * 8);
      const int4 b = ld_nc_v4(d_o + static_cast<int64_t>(t) * lddo + h * D + l * 8);
      const uint32_t* au = reinterpret_cast<const uint32_t*>(&a);
      const uint32_t* bu = reinterpret_cast<const uint32_t*>(&b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = unpack_bf16(au[i]), y = unpack_bf16(bu[i]);
        s += x.x * y.x + x.y * y.y;
      }
      if (t < begin || t >= end) st_v4(dq + static_cast<int64_t>(t) * lddq + h * D + l * 8, make_int4(0, 0, 0, 0));
    }
#pragma unroll
    for (int f = L / 2; f > 0; f >>= 1) s += __shfl_xor_sync(0xffffffffu, s, f);
    const float v = __shfl_sync(0xffffffffu, s, (lane % R) * L);       // row k R + lane % R
    if (lane / R == k) mine = v;
  }
  const int t = t0 + lane;
  if (t < Tq) {
    const int64_t at = static_cast<int64_t>(h) * Tq + t;
    stats[at] = make_float2(lse[at] * 1.4426950408889634f, mine);
  }
}

template <int D>
static int run_attn_bwd(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmdO, const AttnBwdParams& p, int q_tiles,
                        int k_tiles, cudaStream_t stream) {
  static bool attr = false;
  static int sms = 0;
  if (!attr) {
    int dev = 0;
    PRL_CUDA_CHECK(cudaGetDevice(&dev));
    PRL_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PRL_CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_keys_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, AbkCfg<D>::SMEM));
    PRL_CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_queries_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, AbqCfg<D>::SMEM));
    attr = true;
  }
  auto grid = [&](int64_t items) { return static_cast<unsigned>(items < sms ? items : sms); };       // (a CTA without an item returns)
  attn_bwd_keys_kernel<D><<<grid(static_cast<int64_t>(k_tiles) * p.nkv), kAbThreads, AbkCfg<D>::SMEM, stream>>>(tmQ, tmK, tmV, tmdO, p);
  PRL_CUDA_CHECK(cudaGetLastError());
  attn_bwd_queries_kernel<D><<<grid(static_cast<int64_t>(q_tiles) * p.nq), kAbThreads, AbqCfg<D>::SMEM, stream>>>(tmQ, tmK, tmV, tmdO, p);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace prl

using namespace prl;

// dq: bf16 [Tq, nq*d] with row pitch lddq; dk / dv: bf16 [Tk, nkv*d] with row pitch lddkv; all fully overwritten.  d = 64 or 128.
// stats: 2 * nq * Tq floats of scratch.  q_tiles, k_tiles: upper bounds on sum_b ceil(l_b / 128).
extern "C" int prl_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                            float* stats, void* dq, void* dk, void* dv, const int32_t* cu_q, const int32_t* cu_k, int B,
                            int Tq, int Tk, int nq, int nkv, int d, int64_t ldq, int64_t ldk, int64_t ldv, int64_t ldo, int64_t lddo,
                            int64_t lddq, int64_t lddkv, float sm_scale, int causal, int q_tiles, int k_tiles, cudaStream_t stream) {
  if (Tq <= 0) return 0;
  if (nq % nkv != 0 || (d != 64 && d != 128)) return -120;
  if (Tk <= 0 || B <= 0) {                                 // no key is seen
    PRL_CUDA_CHECK(cudaMemset2DAsync(dq, lddq * 2, 0, static_cast<size_t>(nq) * d * 2, Tq, stream));
    return 0;
  }
  const int64_t blocks = (static_cast<int64_t>((Tq + 31) / 32) * nq + 7) / 8;
  const auto* op = static_cast<const __nv_bfloat16*>(o);
  const auto* gp = static_cast<const __nv_bfloat16*>(d_o);
  auto* st = reinterpret_cast<float2*>(stats);
  auto* dqp = static_cast<__nv_bfloat16*>(dq);
  if (d == 64) attn_stats_kernel<64><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(op, gp, ldo, lddo, lse, st, dqp, lddq, cu_q, B, Tq, nq);
  else attn_stats_kernel<128><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(op, gp, ldo, lddo, lse, st, dqp, lddq, cu_q, B, Tq, nq);
  PRL_CUDA_CHECK(cudaGetLastError());
  CUtensorMap tmQ, tmK, tmV, tmdO;
  if (af_tmap(&tmQ, q, Tq, static_cast<uint64_t>(nq) * d, ldq * 2, 128)) return -121;
  if (af_tmap(&tmK, k, Tk, static_cast<uint64_t>(nkv) * d, ldk * 2, 128)) return -122;
  if (af_tmap(&tmV, v, Tk, static_cast<uint64_t>(nkv) * d, ldv * 2, 128)) return -123;
  if (af_tmap(&tmdO, d_o, Tq, static_cast<uint64_t>(nq) * d, lddo * 2, 128)) return -124;
  AttnBwdParams p;
  p.dq = static_cast<__nv_bfloat16*>(dq); p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  p.lddq = lddq; p.lddkv = lddkv;
  p.stats = st; p.cu_q = cu_q; p.cu_k = cu_k;
  p.B = B; p.nq = nq; p.nkv = nkv; p.Tq = Tq;
  p.sm_scale = sm_scale; p.scale_log2 = sm_scale * 1.4426950408889634f; p.causal = causal;
  return d == 64 ? run_attn_bwd<64>(tmQ, tmK, tmV, tmdO, p, q_tiles, k_tiles, stream) : run_attn_bwd<128>(tmQ, tmK, tmV, tmdO, p, q_tiles, k_tiles, stream);
}
