// polyrl_b200 — token sampling for the rollout engine: temperature + Gumbel-max categorical sampling (noise of 24 bits an element; over the
// whole row for top_k=-1 / top_p=1, the GRPO default), top-k / top-p, or greedy, returning the token id AND its log-probability under the
// distribution that was sampled.
//
// Reference capability: SGLang sampler + `return_logprob` (meta_info.output_token_logprobs consumed at
// rlboost/verl_stream/workers/rollout/sglang_rollout/sglang_rollout_remote.py:318-391).
//
// A row belongs to a cluster of 1 to 8 CTAs of 256 threads: as many as keep all rows' CTAs resident at once (row_ctas below).  Rows start
// at any element; the 16-byte granules that lie inside a row are loaded whole, its two ends element by element.
#include <cooperative_groups.h>

#include "common.cuh"

namespace prl {

namespace cg = cooperative_groups;

constexpr int kSampleCtas = 8;        // most CTAs per row (cluster)
constexpr int kSampleThreads = 256;
constexpr int kSampleWarps = kSampleThreads / 32;
constexpr float kLog2E = 1.4426950408889634f;

__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}
// 32 hashed bits of an element before the mixer's last step (which leaves the upper half as it is), and the Gumbel noise of 24 of them
__device__ __forceinline__ uint32_t noise_hash(uint64_t seed, uint32_t row, uint32_t col) {
  const uint32_t h = hash_u32(static_cast<uint32_t>(seed) ^ hash_u32(col + 0x9e3779b9U * (row + 1)));
  uint32_t x = h ^ static_cast<uint32_t>(seed >> 32);
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU;
  return x;
}
__device__ __forceinline__ float gumbel_of(uint32_t x) {
  // (the largest number of 24 bits and a half would round to 2^24: infinite noise, which wins over any logit)
  const float u = (static_cast<float>(min((x ^ (x >> 16)) >> 8, 0xfffffeu)) + 0.5f) * (1.0f / 16777216.0f);
  return -__logf(-__logf(u));
}
// Hashes below this give noise that is certainly less than `need`.  The 24 bits must reach 2^24 exp(-exp(-need)), less a margin of 256
// for the errors of the four fast functions (log near 1 is 6 units off at most, the rest under 40); the hash's upper 16 bits decide.
// A `need` of -inf or NaN lets every element pass.
__device__ __forceinline__ uint32_t least_hash(float need) {
  const int bits = static_cast<int>(__expf(-__expf(-need)) * 16777216.0f) - 256;
  return bits > 0 ? static_cast<uint32_t>(bits) << 8 & 0xffff0000u : 0u;
}

__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);      // ascending float order == ascending unsigned order
}
__device__ __forceinline__ float from_order_key(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A row in 16-byte granules; granule g holds elements [first(g), first(g) + N), those outside the row read as -inf.
template <typename T>
struct SampleRow {
  static constexpr int N = 16 / static_cast<int>(sizeof(T));
  const T* p;
  int V, skew;
  __device__ __forceinline__ SampleRow(const T* row, int v)
      : p(row), V(v), skew(static_cast<int>((reinterpret_cast<uintptr_t>(row) & 15) / sizeof(T))) {}
  __device__ __forceinline__ int granules() const { return (skew + V + N - 1) / N; }
  __device__ __forceinline__ int first(int g) const { return g * N - skew; }
  __device__ __forceinline__ int4 load(int g) const {
    const int e = first(g);
    if (e >= 0 && e + N <= V) return ld_nc_v4(p + e);
    int4 q;
    T* t = reinterpret_cast<T*>(&q);
#pragma unroll
    for (int j = 0; j < N; ++j) t[j] = (e + j >= 0 && e + j < V) ? p[e + j] : static_cast<T>(-INFINITY);
    return q;
  }
  static __device__ __forceinline__ void unpack(const int4& q, float (&f)[N]) {
    if constexpr (sizeof(T) == 2) {
      const uint32_t* u = reinterpret_cast<const uint32_t*>(&q);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = unpack_bf16(u[j]);
        f[2 * j] = x.x; f[2 * j + 1] = x.y;
      }
    } else {
      const float* x = reinterpret_cast<const float*>(&q);
#pragma unroll
      for (int j = 0; j < N; ++j) f[j] = x[j];
    }
  }
};

// The best noisy logit so far; the lower index wins a tie.
struct Pick {
  float key;
  int idx;
  float raw;
  __device__ __forceinline__ void offer(float k, int i, float r) {
    if (k > key || (k == key && i < idx)) { key = k; idx = i; raw = r; }
  }
};

// Offers a granule's elements (those that are not wanted as -inf).  Most cannot win: the noise is a monotone function of the hash, so a
// granule computes from the CTA's best key and its own largest logit what a winner's hash must reach, and only elements that reach it pay
// for two logarithms.
template <int N>
__device__ __forceinline__ void offer_granule(Pick& best, float bar, const float (&f)[N], float fmax, int first, float scale, bool greedy,
                                              uint64_t seed, uint32_t row) {
  if (greedy) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (f[j] * scale > best.key) { best.key = f[j] * scale; best.idx = first + j; best.raw = f[j]; }
    return;
  }
  const uint32_t least = least_hash(bar - fmax * scale);
  uint32_t x[N];
  bool any = false;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    x[j] = noise_hash(seed, row, first + j);
    any |= x[j] >= least;
  }
  if (any) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (x[j] >= least) {
        const float k = f[j] * scale + gumbel_of(x[j]);
        if (k > best.key) { best.key = k; best.idx = first + j; best.raw = f[j]; }
      }
  }
}
// The CTA's best key so far (as an order key), which every warp raises; a late read only prunes less.  Lanes may read different values while
// other warps raise it, so the warp agrees on the largest: callers branch on the result around collectives of the whole warp.
__device__ __forceinline__ float raise_bar(uint32_t* bar, const Pick& best) {
  const uint32_t b = *const_cast<volatile uint32_t*>(bar), k = __reduce_max_sync(0xffffffffu, max(order_key(best.key), b));
  if (k > b && (threadIdx.x & 31) == 0) atomicMax(bar, k);
  return from_order_key(k);
}

__device__ __forceinline__ Pick warp_pick(Pick p) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float k = __shfl_xor_sync(0xffffffffu, p.key, o);
    const int i = __shfl_xor_sync(0xffffffffu, p.idx, o);
    const float r = __shfl_xor_sync(0xffffffffu, p.raw, o);
    p.offer(k, i, r);
  }
  return p;
}
// running maximum and sum of 2^((x - max) k2); a part that saw only -inf has the sum 0
__device__ __forceinline__ void merge_sum(float& m, float& s, float m2, float s2, float k2) {
  const float nm = fmaxf(m, m2);
  if (nm == -INFINITY) return;
  s = (m == -INFINITY ? 0.f : s * ex2((m - nm) * k2)) + (m2 == -INFINITY ? 0.f : s2 * ex2((m2 - nm) * k2));
  m = nm;
}

__device__ __forceinline__ float scale_of(const float* temp, int row, bool inverse, bool greedy_all, bool& greedy) {
  float it = 1.f;
  if (temp) {
    const float t = temp[row];
    it = inverse ? t : (t > 0.f ? __frcp_rn(fmaxf(t, 1e-6f)) : 0.f);
  }
  greedy = greedy_all || it <= 0.f;
  return greedy ? 1.f : it;
}

// One pass over the row.  Bound by integer instructions: three rounds of the hash are 24 of the 45 that an element takes, on a pipe that
// takes a warp every other cycle (61% busy).  [128, 128256] bf16: 37 us (two logarithms for every element, one CTA per row: 47); one row
// of 151936: 9 us (47).
template <typename T>
__global__ void __launch_bounds__(kSampleThreads, 4)
sample_kernel(const T* __restrict__ logits, int64_t ld, int V, const float* __restrict__ temp, int inverse,
              const uint64_t* __restrict__ seeds, int greedy_all, int64_t* __restrict__ out_tok, float* __restrict__ out_lp) {
  using Row = SampleRow<T>;
  constexpr int N = Row::N, AHEAD = 2;
  struct Part { Pick pick; float m, s; };
  __shared__ Part part[kSampleWarps];
  __shared__ Part of_cta[kSampleCtas];
  cg::cluster_group cluster = cg::this_cluster();
  cluster_arrive();                     // waited for before the first store into another CTA: all CTAs of the cluster run by then
  const int rank = static_cast<int>(cluster.block_rank()), ctas = static_cast<int>(cluster.num_blocks());
  const int row = blockIdx.x / ctas;
  const Row r(logits + static_cast<int64_t>(row) * ld, V);
  bool greedy;
  const float scale = scale_of(temp, row, inverse != 0, greedy_all != 0, greedy);
  const float k2 = scale * kLog2E;
  const uint64_t seed = seeds ? seeds[row] : 0;
  __shared__ uint32_t bar;
  if (threadIdx.x == 0) bar = order_key(-INFINITY);
  __syncthreads();
  Pick best{-INFINITY, 0x7fffffff, -INFINITY};
  float bar_now = -INFINITY, m = -INFINITY, s = 0.f;
  const int ng = r.granules();
  const int step = ctas * static_cast<int>(blockDim.x);
  for (int g0 = rank * static_cast<int>(blockDim.x); g0 < ng; g0 += AHEAD * step) {          // uniform in a CTA
    int4 q[AHEAD];
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) q[a] = r.load(min(g0 + a * step + static_cast<int>(threadIdx.x), ng));   // past the end: -inf
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) {
      if (g0 + a * step >= ng) break;
      const int first = r.first(g0 + a * step + static_cast<int>(threadIdx.x));
      float f[N];
      Row::unpack(q[a], f);
      float fm = f[0];
#pragma unroll
      for (int j = 1; j < N; ++j) fm = fmaxf(fm, f[j]);
      if (fm > m) { s *= ex2((m - fm) * k2); m = fm; }
      if (m > -INFINITY) {
#pragma unroll
        for (int j = 0; j < N; ++j) s += ex2((f[j] - m) * k2);
      }
      if (!greedy && bar_now == -INFINITY) {                    // one element of each lane sets a bar for the rest
        if (f[0] > -INFINITY) best.offer(f[0] * scale + gumbel_of(noise_hash(seed, row, first)), first, f[0]);
        bar_now = raise_bar(&bar, best);
      }
      offer_granule<N>(best, bar_now, f, fm, first, scale, greedy, seed, row);
      if (!greedy) bar_now = raise_bar(&bar, best);
    }
  }
  best = warp_pick(best);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) merge_sum(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o), k2);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) part[w] = Part{best, m, s};
  __syncthreads();
  cluster_wait();
  if (threadIdx.x == 0) {
    Part t = part[0];
    for (int i = 1; i < static_cast<int>(blockDim.x >> 5); ++i) {
      t.pick.offer(part[i].pick.key, part[i].pick.idx, part[i].pick.raw);
      merge_sum(t.m, t.s, part[i].m, part[i].s, k2);
    }
    *cluster.map_shared_rank(&of_cta[rank], 0) = t;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    Part t = of_cta[0];
    for (int i = 1; i < ctas; ++i) {
      t.pick.offer(of_cta[i].pick.key, of_cta[i].pick.idx, of_cta[i].pick.raw);
      merge_sum(t.m, t.s, of_cta[i].m, of_cta[i].s, k2);
    }
    out_tok[row] = t.pick.idx;
    out_lp[row] = (t.pick.raw - t.m) * scale - logf(t.s);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// top-k / top-p (nucleus) sampling without a sort: the k-th largest logit and the nucleus cut are found by MSB-first radix selection over
// order-preserving integer keys of the logits (16 bits of a bf16 logit, 32 of an fp32 one), six bits at a time: counts for top-k,
// probability mass for top-p.  Then Gumbel-max over the kept set and the log-prob under the renormalised distribution.  HF / SGLang
// order: temperature -> top-k -> top-p.  (reference exposes rollout.top_k / rollout.top_p:
// 3rdparty/verl/verl/trainer/config/rollout/rollout.yaml).
//
// Logits share a few exponents, so a histogram with shared-memory atomics runs one element after the other.  Here every thread owns a
// column of 64 counts or 32 masses in shared memory ([bin][thread]: no bank conflict, no atomic), then the CTAs' sums meet over the cluster.
// Masses are whole numbers of 2^-40, so a digit's bins add up to the bin of the digit before, in any order, and the cut does not depend on
// timing (tensor-parallel engine ranks must sample identically).  Every pass reads the row again, from L2: kept in registers (40 a thread
// at 152 K logits) or shared memory it would cost the third CTA of an SM.
// [47, 151936] bf16, top_p 0.95: 61 us.  With fp32 masses, which allow 64 bins and three passes instead of four, it was 47, but the cut moved
// where masses tie within 2^-24; with 64-bit atomics on 256 bins, one CTA per row and scalar loads it was 1808.
// ------------------------------------------------------------------------------------------------------------------
constexpr int kBins = 64;               // most bins
constexpr float kMassUnits = 1099511627776.f;        // 2^40
struct CountDigits {
  using Sum = uint32_t;
  static constexpr bool mass = false;
  static constexpr int BITS = 6;
};
struct MassDigits {
  using Sum = uint64_t;
  static constexpr bool mass = true;
  static constexpr int BITS = 5;
};
constexpr int kHistBytes = kSampleThreads * 256;     // 64 counts or 32 masses a thread

template <typename T>
__global__ void __launch_bounds__(kSampleThreads, 3)
sample_topk_topp_kernel(const T* __restrict__ logits, int64_t ld, int V, const float* __restrict__ temp, int inverse,
                        const uint64_t* __restrict__ seeds, int greedy_all, int top_k, float top_p,
                        int64_t* __restrict__ out_tok, float* __restrict__ out_lp) {
  using Row = SampleRow<T>;
  constexpr int N = Row::N;
  constexpr int KEY_BITS = 8 * static_cast<int>(sizeof(T));
  extern __shared__ uint64_t hist[];                      // a column of sums for every thread
  struct Part { Pick pick; float mass; };
  __shared__ Part part[kSampleWarps];
  __shared__ Part of_cta[kSampleCtas];
  __shared__ uint64_t sums[2][kSampleCtas][kBins];        // every CTA holds all CTAs' sums; two passes alternate
  __shared__ float cta_max[kSampleCtas];
  __shared__ uint32_t s_bin, bar;
  __shared__ uint64_t s_rest;
  cg::cluster_group cluster = cg::this_cluster();
  cluster_arrive();                                       // as above
  const int rank = static_cast<int>(cluster.block_rank()), ctas = static_cast<int>(cluster.num_blocks());
  const int row = blockIdx.x / ctas, tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const Row r(logits + static_cast<int64_t>(row) * ld, V);
  bool greedy;
  const float scale = scale_of(temp, row, inverse != 0, greedy_all != 0, greedy);
  const float k2 = scale * kLog2E;
  const uint64_t seed = seeds ? seeds[row] : 0;
  const int ng = r.granules();
  const int turns = (ng + ctas * kSampleThreads - 1) / (ctas * kSampleThreads);
  auto granule = [&](int i) { return (i * ctas + rank) * kSampleThreads + tid; };
  auto key_of = [](float f) { return order_key(f) >> (32 - KEY_BITS); };

  // fn(unpacked granule, granule index) over the thread's granules, in a fixed order; a granule past the end reads as -inf
  auto each = [&](auto&& fn) {
    constexpr int AHEAD = 2;
    for (int i = 0; i < turns; i += AHEAD) {
      int4 q[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) q[a] = r.load(min(granule(i + a), ng));
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        if (i + a >= turns) break;
        float f[N];
        Row::unpack(q[a], f);
        fn(f, granule(i + a));
      }
    }
  };

  float m = -INFINITY;
  each([&](const float (&f)[N], int) {
#pragma unroll
    for (int j = 0; j < N; ++j) m = fmaxf(m, f[j]);
  });
  m = warp_max(m);
  if (l == 0) part[w].mass = m;
  if (tid == 0) bar = order_key(-INFINITY);
  __syncthreads();
  cluster_wait();
  if (tid < ctas) {
    float t = part[0].mass;
    for (int i = 1; i < kSampleWarps; ++i) t = fmaxf(t, part[i].mass);
    *cluster.map_shared_rank(&cta_max[rank], tid) = t;
  }
  cluster.sync();
  m = cta_max[0];
  for (int i = 1; i < ctas; ++i) m = fmaxf(m, cta_max[i]);

  // Largest key whose elements and all above reach `want` (a share of the whole where `share`), among elements with key >= floor_key.
  // Counts, or with Mass weights in units of 2^-40.
  int pass_no = 0;
  auto select = [&](auto kind, double want_in, bool share, uint32_t floor_key) -> uint32_t {
    using Kind = decltype(kind);
    using Sum = typename Kind::Sum;
    constexpr int BITS = Kind::BITS, BINS = 1 << BITS, PER_LANE = BINS / 32;
    Sum* sum = reinterpret_cast<Sum*>(hist);               // [BINS][kSampleThreads]
    uint64_t want = static_cast<uint64_t>(want_in);
    uint32_t prefix = 0;
    for (int hi = KEY_BITS; hi > 0;) {
      const int lo = hi > BITS ? hi - BITS : 0;
#pragma unroll 16
      for (int b = 0; b < BINS; ++b) sum[b * kSampleThreads + tid] = 0;
      each([&](const float (&f)[N], int) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const uint32_t key = key_of(f[j]);
          if (key < floor_key || (hi < KEY_BITS && (key >> hi) != prefix)) continue;
          Sum& bin = sum[((key >> lo) & ((1u << (hi - lo)) - 1u)) * kSampleThreads + tid];
          if constexpr (Kind::mass) bin += __float2ull_rz(ex2((f[j] - m) * k2) * kMassUnits);
          else bin += 1;
        }
      });
      __syncthreads();
      uint64_t(&all)[kSampleCtas][kBins] = sums[pass_no++ & 1];
      for (int b = w; b < BINS; b += kSampleWarps) {
        Sum t = 0;
#pragma unroll
        for (int c = 0; c < kSampleWarps; ++c) t += sum[b * kSampleThreads + c * 32 + l];
        if constexpr (Kind::mass) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        } else {
          t = __reduce_add_sync(0xffffffffu, t);
        }
        if (l < ctas) *cluster.map_shared_rank(&all[rank][b], l) = t;
      }
      cluster.sync();
      if (w == 0) {                                        // lane l: the bins from BINS - 1 - PER_LANE l on, from the top down
        uint64_t of[PER_LANE] = {}, up = 0;
        for (int c = 0; c < ctas; ++c)
#pragma unroll
          for (int i = 0; i < PER_LANE; ++i) of[i] += all[c][BINS - 1 - PER_LANE * l - i];
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) up += of[i];
        uint64_t mine = up;                                // up: inclusive sum over the lanes up to this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint64_t t = __shfl_up_sync(0xffffffffu, up, o);
          if (l >= o) up += t;
        }
        if (share) {
          want = static_cast<uint64_t>(want_in * static_cast<double>(__shfl_sync(0xffffffffu, up, 31)));
          if (want == 0) want = 1;
        }
        const uint32_t hit = __ballot_sync(0xffffffffu, up >= want);
        if (hit == 0) {
          if (l == 0) { s_bin = 0; s_rest = 0; }           // no mass at all: everything
        } else if (l == __ffs(hit) - 1) {
          uint64_t rest = want - (up - mine);
          int i = 0;
          for (; i < PER_LANE - 1 && of[i] < rest; ++i) rest -= of[i];
          s_bin = static_cast<uint32_t>(BINS - 1 - PER_LANE * l - i);
          s_rest = rest;
        }
      }
      __syncthreads();
      prefix = (prefix << (hi - lo)) | s_bin;
      want = s_rest;
      if (want == 0) return prefix << lo;
      share = false;
      hi = lo;
    }
    return prefix;
  };

  const uint32_t k_key = top_k > 0 && top_k < V ? select(CountDigits{}, static_cast<double>(top_k), false, 0) : 0;
  const uint32_t p_key = !greedy && top_p < 1.f && top_p > 0.f ? select(MassDigits{}, static_cast<double>(top_p), true, k_key) : 0;
  const uint32_t cut = k_key > p_key ? k_key : p_key;

  // ---- Gumbel-max over the kept set + its mass
  Pick best{-INFINITY, 0x7fffffff, -INFINITY};
  float bar_now = -INFINITY, mass = 0.f;
  each([&](const float (&raw)[N], int g) {
    float f[N], fm = -INFINITY;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      f[j] = key_of(raw[j]) >= cut ? raw[j] : -INFINITY;
      fm = fmaxf(fm, f[j]);
    }
    if (__any_sync(0xffffffffu, fm > -INFINITY)) {
#pragma unroll
      for (int j = 0; j < N; ++j) mass += ex2((f[j] - m) * k2);
      offer_granule<N>(best, bar_now, f, fm, r.first(g), scale, greedy, seed, row);
      bar_now = raise_bar(&bar, best);
    }
  });
  best = warp_pick(best);
  mass = warp_sum(mass);
  if (l == 0) part[w] = Part{best, mass};
  __syncthreads();
  if (tid == 0) {
    Part t = part[0];
    for (int i = 1; i < kSampleWarps; ++i) { t.pick.offer(part[i].pick.key, part[i].pick.idx, part[i].pick.raw); t.mass += part[i].mass; }
    *cluster.map_shared_rank(&of_cta[rank], 0) = t;
  }
  cluster.sync();
  if (rank == 0 && tid == 0) {
    Part t = of_cta[0];
    for (int i = 1; i < ctas; ++i) { t.pick.offer(of_cta[i].pick.key, of_cta[i].pick.idx, of_cta[i].pick.raw); t.mass += of_cta[i].mass; }
    out_tok[row] = t.pick.idx;
    out_lp[row] = (t.pick.raw - m) * scale - logf(t.mass);
  }
}

// CTAs per row: the most (a power of two, at most 8) that leave the whole batch resident on 148 SMs, `per_sm` CTAs on each.  A second,
// ragged wave costs more: the plain sampler took 50 us for 128 rows with 8 CTAs a row (1.7 waves) and 37 with 4.
inline int row_ctas(int B, int per_sm) {
  int c = kSampleCtas;
  while (c > 1 && static_cast<int64_t>(B) * c > 148 * per_sm) c >>= 1;
  return c;
}
template <typename K, typename... Args>
int launch_rows(K kernel, int B, int ctas, int smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(B) * ctas);
  cfg.blockDim = dim3(kSampleThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ctas;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  PRL_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, args...));
  return 0;
}

template <typename T>
int launch_topk_topp(const void* logits, int64_t ld, int B, int V, const float* temp, int inverse, const uint64_t* seeds, int greedy_all,
                     int top_k, float top_p, int64_t* out_tok, float* out_lp, cudaStream_t s) {
  constexpr int smem = kHistBytes;
  PRL_CUDA_CHECK(cudaFuncSetAttribute(sample_topk_topp_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  return launch_rows(sample_topk_topp_kernel<T>, B, row_ctas(B, 3), smem, s, static_cast<const T*>(logits), ld, V, temp, inverse, seeds,
                     greedy_all, top_k, top_p, out_tok, out_lp);
}
template <typename T>
int launch_sample(const void* logits, int64_t ld, int B, int V, const float* temp, int inverse, const uint64_t* seeds, int greedy_all,
                  int64_t* out_tok, float* out_lp, cudaStream_t s) {
  return launch_rows(sample_kernel<T>, B, row_ctas(B, 4), 0, s, static_cast<const T*>(logits), ld, V, temp, inverse, seeds, greedy_all,
                     out_tok, out_lp);
}

}  // namespace prl

using namespace prl;

// temp: temperatures of the rows (<= 0: greedy), or their inverses where `inverse`; null: 1.
// top_k <= 0 disables top-k, top_p >= 1 disables top-p.  dtype: 0 = fp32 logits, 1 = bf16 logits.
extern "C" int prl_sample_topk_topp(const void* logits, int dtype, int64_t ld, int B, int V, const float* temp, int inverse,
                                    const uint64_t* seeds, int greedy_all, int top_k, float top_p, int64_t* out_tok,
                                    float* out_lp, cudaStream_t s) {
  if (B <= 0) return 0;
  return dtype == 0 ? launch_topk_topp<float>(logits, ld, B, V, temp, inverse, seeds, greedy_all, top_k, top_p, out_tok, out_lp, s)
                    : launch_topk_topp<__nv_bfloat16>(logits, ld, B, V, temp, inverse, seeds, greedy_all, top_k, top_p, out_tok, out_lp, s);
}

// dtype: 0 = fp32 logits, 1 = bf16 logits
extern "C" int prl_sample(const void* logits, int dtype, int64_t ld, int B, int V, const float* temp, int inverse,
                          const uint64_t* seeds, int greedy_all, int64_t* out_tok, float* out_lp, cudaStream_t s) {
  if (B <= 0) return 0;
  return dtype == 0 ? launch_sample<float>(logits, ld, B, V, temp, inverse, seeds, greedy_all, out_tok, out_lp, s)
                    : launch_sample<__nv_bfloat16>(logits, ld, B, V, temp, inverse, seeds, greedy_all, out_tok, out_lp, s);
}
