// polyrl_b200 — what lies between the fused QKV projection and attention, in one pass: optional RMS norm of every query and key head
// (Qwen3), rotary embedding, optional append to the paged cache; and the gradients of the same.
//
// Reference capability: q_norm / k_norm and apply_rotary_pos_emb of the HF decoder layers behind
// 3rdparty/verl/verl/models/transformers/qwen2.py:150-230 (eager: a dozen elementwise kernels over fp32 copies).
//
// A head of d values belongs to d / 16 neighbouring threads of a warp; each holds 8 values of the lower half and the 8 that rotate with
// them in the upper half, so loads and stores are 16 bytes, the rotation needs no exchange and the norm's sum is a few shuffles.
// Bound by HBM: one read and one write of the query and key columns.
#include "common.cuh"

namespace prl {

constexpr int kQrThreads = 256;

struct QkRopeParams {
  const __nv_bfloat16* src;          // [T, ld]: nq query heads, nkv key heads, nkv value heads
  __nv_bfloat16* dst;                // [T, ldo], may be src: receives the query and key heads
  int64_t ld, ldo;
  const int64_t* pos;
  const float* cos_tab;              // [positions, d / 2]
  const float* sin_tab;
  const __nv_bfloat16* qn;           // [d] gains, or null: no norm
  const __nv_bfloat16* kn;
  float eps, sign;
  __nv_bfloat16* k_cache;            // [pages, nkv, block_size, d]
  __nv_bfloat16* v_cache;
  const int64_t* slots;              // [T] or null; a slot below zero appends nothing
  int T, nq, nkv, block_size;
};

__device__ __forceinline__ void unpack8(const int4& v, float (&f)[8]) {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = unpack_bf16(u[j]);
    f[2 * j] = a.x;
    f[2 * j + 1] = a.y;
  }
}
__device__ __forceinline__ int4 pack8(const float (&f)[8]) {
  int4 o;
  o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]); o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
  return o;
}
__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// sum over the L threads of a head (L a power of two that divides the warp; all of them take part)
template <int L>
__device__ __forceinline__ float head_sum(float v) {
  const unsigned mask = L == 32 ? 0xffffffffu : ((1u << L) - 1) << (lane_id() & ~(L - 1));
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

template <int D, bool NORM>
__global__ void __launch_bounds__(kQrThreads) qk_rope_kernel(QkRopeParams p) {
  constexpr int L = D / 16, HALF = D / 2;
  grid_behind();
  const int heads = p.nq + p.nkv + (p.slots != nullptr ? p.nkv : 0);
  const int64_t item = (static_cast<int64_t>(blockIdx.x) * kQrThreads + threadIdx.x) / L;
  if (item >= static_cast<int64_t>(p.T) * heads) return;                  // (whole heads leave together)
  const int t = static_cast<int>(item / heads), h = static_cast<int>(item - static_cast<int64_t>(t) * heads);
  const int j = (threadIdx.x % L) * 8;
  const __nv_bfloat16* s = p.src + static_cast<int64_t>(t) * p.ld + h * D + j;
  const int4 lo = ld_v4(s), hi = ld_v4(s + HALF);
  const int64_t slot = p.slots != nullptr && h >= p.nq ? p.slots[t] : -1;
  const int hk = h < p.nq + p.nkv ? h - p.nq : h - p.nq - p.nkv;
  const int64_t at = slot >= 0 ? ((slot / p.block_size * p.nkv + hk) * p.block_size + slot % p.block_size) * D + j : 0;
  if (h >= p.nq + p.nkv) {                                                // a value head: only the cache takes it
    if (slot >= 0) {
      st_v4(p.v_cache + at, lo);
      st_v4(p.v_cache + at + HALF, hi);
    }
    return;
  }
  float a[8], b[8], c[8], n[8];
  unpack8(lo, a);
  unpack8(hi, b);
  if (NORM) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += a[i] * a[i] + b[i] * b[i];
    const float rstd = rsqrtf(head_sum<L>(ss) / static_cast<float>(D) + p.eps);
    const __nv_bfloat16* g = (h < p.nq ? p.qn : p.kn) + j;
    unpack8(*reinterpret_cast<const int4*>(g), c);
    unpack8(*reinterpret_cast<const int4*>(g + HALF), n);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a[i] *= rstd * c[i];
      b[i] *= rstd * n[i];
    }
  }
  const int64_t row = p.pos[t] * HALF + j;
  load8(p.cos_tab + row, c);
  load8(p.sin_tab + row, n);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = a[i], sn = n[i] * p.sign;
    a[i] = x * c[i] - b[i] * sn;
    b[i] = b[i] * c[i] + x * sn;
  }
  const int4 olo = pack8(a), ohi = pack8(b);
  __nv_bfloat16* d = p.dst + static_cast<int64_t>(t) * p.ldo + h * D + j;
  st_v4(d, olo);
  st_v4(d + HALF, ohi);
  if (slot >= 0) {
    st_v4(p.k_cache + at, olo);
    st_v4(p.k_cache + at + HALF, ohi);
  }
}

// Gradient through rotation and norm, in place on g [T, ldg] (query and key columns): g = R^T g, then with x the heads before the norm and
// xh = x rstd:  dx = rstd (g w - xh mean(g w xh)).  The gains' gradients sum g xh over tokens and heads: a thread keeps its 16 columns in
// registers over all heads it takes, a block writes one row of `part` [blocks, d]; the first q_blocks blocks take query heads, the rest keys.
template <int D>
__global__ void __launch_bounds__(kQrThreads)
qk_norm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, __nv_bfloat16* g, int64_t ldg, const int64_t* __restrict__ pos,
                        const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, const __nv_bfloat16* __restrict__ qn,
                        const __nv_bfloat16* __restrict__ kn, float eps, float* __restrict__ part, int T, int nq, int nkv, int q_blocks) {
  constexpr int L = D / 16, HALF = D / 2, GROUPS = kQrThreads / L;
  __shared__ float red[kQrThreads / 32][D];
  const bool is_q = static_cast<int>(blockIdx.x) < q_blocks;
  const int heads = is_q ? nq : nkv, first = is_q ? 0 : nq;
  const int blk = is_q ? blockIdx.x : blockIdx.x - q_blocks, blocks = is_q ? q_blocks : gridDim.x - q_blocks;
  const int j = (threadIdx.x % L) * 8;
  float wa[8], wb[8], da[8], db[8];
  const __nv_bfloat16* w = (is_q ? qn : kn) + j;
  unpack8(*reinterpret_cast<const int4*>(w), wa);
  unpack8(*reinterpret_cast<const int4*>(w + HALF), wb);
#pragma unroll
  for (int i = 0; i < 8; ++i) { da[i] = 0.f; db[i] = 0.f; }
  const int64_t items = static_cast<int64_t>(T) * heads;
  for (int64_t it = static_cast<int64_t>(blk) * GROUPS + threadIdx.x / L; it < items; it += static_cast<int64_t>(blocks) * GROUPS) {
    const int t = static_cast<int>(it / heads), h = first + static_cast<int>(it - static_cast<int64_t>(t) * heads);
    const __nv_bfloat16* xp = x + static_cast<int64_t>(t) * ldx + h * D + j;
    __nv_bfloat16* gp = g + static_cast<int64_t>(t) * ldg + h * D + j;
    float xa[8], xb[8], ga[8], gb[8], c[8], s[8];
    unpack8(ld_nc_v4(xp), xa);
    unpack8(ld_nc_v4(xp + HALF), xb);
    unpack8(ld_v4(gp), ga);
    unpack8(ld_v4(gp + HALF), gb);
    const int64_t row = pos[t] * HALF + j;
    load8(cos_tab + row, c);
    load8(sin_tab + row, s);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += xa[i] * xa[i] + xb[i] * xb[i];
    const float rstd = rsqrtf(head_sum<L>(ss) / static_cast<float>(D) + eps);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float u = ga[i] * c[i] + gb[i] * s[i], v = gb[i] * c[i] - ga[i] * s[i];
      xa[i] *= rstd;
      xb[i] *= rstd;
      da[i] += u * xa[i];
      db[i] += v * xb[i];
      ga[i] = u * wa[i];
      gb[i] = v * wb[i];
      dot += ga[i] * xa[i] + gb[i] * xb[i];
    }
    dot = head_sum<L>(dot) / static_cast<float>(D);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ga[i] = rstd * (ga[i] - xa[i] * dot);
      gb[i] = rstd * (gb[i] - xb[i] * dot);
    }
    st_v4(gp, pack8(ga));
    st_v4(gp + HALF, pack8(gb));
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int o = L; o < 32; o <<= 1) {
      da[i] += __shfl_xor_sync(0xffffffffu, da[i], o);
      db[i] += __shfl_xor_sync(0xffffffffu, db[i], o);
    }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane < L) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      red[warp][j + i] = da[i];
      red[warp][HALF + j + i] = db[i];
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += kQrThreads) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kQrThreads / 32; ++i) t += red[i][c];
    part[static_cast<int64_t>(blockIdx.x) * D + c] = t;
  }
}

// the gains' gradients: block 0 sums the query blocks' rows of `part`, block 1 the key blocks'; threads = (8, d), in a fixed order
__global__ void qk_norm_dw_kernel(const float* __restrict__ part, int q_blocks, int blocks, __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk) {
  extern __shared__ float sm[];
  const int d = blockDim.x, c = threadIdx.x, y = threadIdx.y;
  const int lo = blockIdx.x ? q_blocks : 0, hi = blockIdx.x ? blocks : q_blocks;
  float s = 0.f;
#pragma unroll 8
  for (int r = lo + y; r < hi; r += blockDim.y) s += part[static_cast<int64_t>(r) * d + c];
  sm[y * d + c] = s;
  __syncthreads();
  if (y == 0) {
    s = 0.f;
    for (int i = 0; i < static_cast<int>(blockDim.y); ++i) s += sm[i * d + c];
    (blockIdx.x ? dk : dq)[c] = __float2bfloat16(s);
  }
}

template <int D>
static void launch_qk_rope(const QkRopeParams& p, cudaStream_t s) {
  const int64_t heads = p.nq + p.nkv + (p.slots != nullptr ? p.nkv : 0), threads = p.T * heads * (D / 16);
  const unsigned grid = static_cast<unsigned>((threads + kQrThreads - 1) / kQrThreads);
  auto kern = p.qn != nullptr ? qk_rope_kernel<D, true> : qk_rope_kernel<D, false>;
  if (p.T <= 256) launch_behind(kern, grid, kQrThreads, 0, s, p);       // a decode step
  else kern<<<grid, kQrThreads, 0, s>>>(p);
}

}  // namespace prl

using namespace prl;

// Head widths of these kernels; the general rotation (elementwise.cu) takes the others.
extern "C" int prl_qk_rope_width_ok(int d) { return d == 32 || d == 64 || d == 128 || d == 256; }

// src, dst: 16-byte aligned rows (pitches multiples of 8); tables 16-byte aligned.  qn, kn: both or neither.
extern "C" int prl_qk_rope(const void* src, void* dst, const int64_t* pos, const float* cos_tab, const float* sin_tab, const void* qn, const void* kn, float eps,
                           int T, int nq, int nkv, int d, int64_t ld, int64_t ldo, float sign, void* k_cache, void* v_cache, const int64_t* slots,
                           int block_size, cudaStream_t s) {
  if (T <= 0) return 0;
  QkRopeParams p{static_cast<const __nv_bfloat16*>(src), static_cast<__nv_bfloat16*>(dst), ld, ldo, pos, cos_tab, sin_tab,
                 static_cast<const __nv_bfloat16*>(qn), static_cast<const __nv_bfloat16*>(kn), eps, sign, static_cast<__nv_bfloat16*>(k_cache),
                 static_cast<__nv_bfloat16*>(v_cache), slots, T, nq, nkv, block_size};
  switch (d) {
    case 32: launch_qk_rope<32>(p, s); break;
    case 64: launch_qk_rope<64>(p, s); break;
    case 128: launch_qk_rope<128>(p, s); break;
    case 256: launch_qk_rope<256>(p, s); break;
    default: return -130;
  }
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}

static int bwd_blocks(int64_t items, int groups) {
  const int64_t want = (items + groups - 1) / groups;
  return static_cast<int>(want < 1 ? 1 : want < 148 * 3 ? want : 148 * 3);
}
// rows of the scratch `part` [rows, d] of prl_qk_norm_rope_bwd
extern "C" int prl_qk_norm_rope_bwd_parts(int T, int nq, int nkv, int d) {
  const int groups = kQrThreads / (d / 16);
  return bwd_blocks(static_cast<int64_t>(T) * nq, groups) + bwd_blocks(static_cast<int64_t>(T) * nkv, groups);
}
extern "C" int prl_qk_norm_rope_bwd(const void* x, int64_t ldx, void* g, int64_t ldg, const int64_t* pos, const float* cos_tab, const float* sin_tab,
                                    const void* qn, const void* kn, float eps, float* part, void* dqn, void* dkn, int T, int nq, int nkv, int d,
                                    cudaStream_t s) {
  if (!prl_qk_rope_width_ok(d)) return -130;
  const int qb = bwd_blocks(static_cast<int64_t>(T) * nq, kQrThreads / (d / 16)), all = prl_qk_norm_rope_bwd_parts(T, nq, nkv, d);
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  const auto* q = static_cast<const __nv_bfloat16*>(qn);
  const auto* k = static_cast<const __nv_bfloat16*>(kn);
  auto* gp = static_cast<__nv_bfloat16*>(g);
  switch (d) {
    case 32: qk_norm_rope_bwd_kernel<32><<<all, kQrThreads, 0, s>>>(xp, ldx, gp, ldg, pos, cos_tab, sin_tab, q, k, eps, part, T, nq, nkv, qb); break;
    case 64: qk_norm_rope_bwd_kernel<64><<<all, kQrThreads, 0, s>>>(xp, ldx, gp, ldg, pos, cos_tab, sin_tab, q, k, eps, part, T, nq, nkv, qb); break;
    case 128: qk_norm_rope_bwd_kernel<128><<<all, kQrThreads, 0, s>>>(xp, ldx, gp, ldg, pos, cos_tab, sin_tab, q, k, eps, part, T, nq, nkv, qb); break;
    default: qk_norm_rope_bwd_kernel<256><<<all, kQrThreads, 0, s>>>(xp, ldx, gp, ldg, pos, cos_tab, sin_tab, q, k, eps, part, T, nq, nkv, qb); break;
  }
  PRL_CUDA_CHECK(cudaGetLastError());
  const int ty = 1024 / d < 8 ? 1024 / d : 8;
  qk_norm_dw_kernel<<<2, dim3(d, ty), d * ty * sizeof(float), s>>>(part, qb, all, static_cast<__nv_bfloat16*>(dqn), static_cast<__nv_bfloat16*>(dkn));
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
