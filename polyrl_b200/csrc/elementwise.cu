// polyrl_b200 — memory-bound transformer kernels: RMSNorm fwd/bwd, RoPE (+ paged-KV append),
// SwiGLU backward, per-row fp8 quantisation.  All are 128-bit vectorised, one pass over HBM.
//
// Reference capability: HF eager RMSNorm/RoPE/SiLU·mul (optionally liger Triton) inside the verl
// FSDP actor (3rdparty/verl/verl/workers/fsdp_workers.py:386-389, models/transformers/*).
#include <cassert>
#include <type_traits>

#include "common.cuh"

namespace prl {

constexpr int kNormThreads = 256;
constexpr int kMaxVPT = 4;   // up to H = 256*8*4 = 8192
constexpr int kStepRows = 256;   // rows of a decode step: launched behind the kernel before

__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < kNormThreads / 32) ? red[l] : 0.f;
  t = warp_sum(t);
  return t;
}

// Sum over the block with one barrier: `parity` alternates from call to call, so a warp that is one call ahead writes the other half.
template <int THREADS>
__device__ __forceinline__ float block_sum_once(float v, float (*red)[THREADS / 32], int parity) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[parity][threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) t += red[parity][i];
  return t;
}

// y = x * rsqrt(mean(x^2)+eps) * w ; rstd saved for backward.
// Bound by HBM.  A block owns whole rows (THREADS x VPT vectors of 16 bytes cover one) and loads the next row before it waits for the sum of
// this one, so the barrier does not drain the loads in flight.  [12287, 4096]: 58 -> 35 us (200 MB, 31 us).
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out, int T, int H, float eps) {
  __shared__ float red[2][THREADS / 32];
  const int nvec = H >> 3;
  int4 wv[VPT], xv[VPT];
  grid_behind();
  auto load = [&](int row) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * THREADS;
      xv[i] = v < nvec ? ld_nc_v4(x + static_cast<int64_t>(row) * H + 8 * v) : make_int4(0, 0, 0, 0);
    }
  };
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * THREADS;
    if (v < nvec) wv[i] = *reinterpret_cast<const int4*>(w + 8 * v);
  }
  int parity = 0;
  load(blockIdx.x);
  for (int row = blockIdx.x; row < T; row += gridDim.x, parity ^= 1) {
    int4 cur[VPT];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      cur[i] = xv[i];
      const uint32_t* u = reinterpret_cast<const uint32_t*>(&cur[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16(u[j]);
        ss += f.x * f.x + f.y * f.y;
      }
    }
    if (row + gridDim.x < T) load(row + gridDim.x);
    ss = block_sum_once<THREADS>(ss, red, parity);
    const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    __nv_bfloat16* yr = y + static_cast<int64_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        const uint32_t* u = reinterpret_cast<const uint32_t*>(&cur[i]);
        const uint32_t* wu = reinterpret_cast<const uint32_t*>(&wv[i]);
        int4 o;
        uint32_t* ou = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16(u[j]);
          const float2 g = unpack_bf16(wu[j]);
          ou[j] = pack_bf16(f.x * rstd * g.x, f.y * rstd * g.y);
        }
        st_v4(yr + 8 * v, o);
      }
    }
  }
}

// Decode-path fusion: x_out = x + r (new residual stream, written in place of x), y = rmsnorm(x_out) * w.
__global__ void __launch_bounds__(kNormThreads)
add_rmsnorm_kernel(__nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ r, const __nv_bfloat16* __restrict__ w,
                   __nv_bfloat16* __restrict__ y, int T, int H, float eps) {
  __shared__ float red[8];
  const int nvec = H >> 3;
  grid_behind();
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    __nv_bfloat16* xr = x + static_cast<int64_t>(row) * H;
    const __nv_bfloat16* rr = r + static_cast<int64_t>(row) * H;
    float v[kMaxVPT][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxVPT; ++i) {
      const int vi = threadIdx.x + i * kNormThreads;
      if (vi < nvec) {
        const int4 a = *reinterpret_cast<const int4*>(xr + 8 * vi);
        const int4 b = ld_nc_v4(rr + 8 * vi);
        const uint32_t* au = reinterpret_cast<const uint32_t*>(&a);
        const uint32_t* bu = reinterpret_cast<const uint32_t*>(&b);
        int4 o;
        uint32_t* ou = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fa = unpack_bf16(au[j]), fb = unpack_bf16(bu[j]);
          ou[j] = pack_bf16(fa.x + fb.x, fa.y + fb.y);
          const float2 s2 = unpack_bf16(ou[j]);          // norm over the bf16-rounded residual stream (what the next op reads)
          v[i][2 * j] = s2.x; v[i][2 * j + 1] = s2.y;
          ss += s2.x * s2.x + s2.y * s2.y;
        }
        st_v4(xr + 8 * vi, o);
      }
    }
    ss = block_sum_256(ss, red);
    const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
    __nv_bfloat16* yr = y + static_cast<int64_t>(row) * H;
#pragma unroll
    for (int i = 0; i < kMaxVPT; ++i) {
      const int vi = threadIdx.x + i * kNormThreads;
      if (vi < nvec) {
        const int4 wq = *reinterpret_cast<const int4*>(w + 8 * vi);
        const uint32_t* wu = reinterpret_cast<const uint32_t*>(&wq);
        int4 o;
        uint32_t* ou = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 g = unpack_bf16(wu[j]);
          ou[j] = pack_bf16(v[i][2 * j] * rstd * g.x, v[i][2 * j + 1] * rstd * g.y);
        }
        st_v4(yr + 8 * vi, o);
      }
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres, the gradient that reaches x past the norm);  part[block] = sum over its rows of dy*xhat.
// Bound by HBM.  Registers are sized for the row length (a block that held the longest row's ran two to the SM and waited for every row),
// the next row is loaded before the sum of this one, and the gain's gradient leaves as one partial row per block, which
// rmsnorm_dw_kernel adds in a fixed order: no atomics, no zero fill.  [12287, 4096]: 223 us and 62 us
// for the sum with dres -> 76 us in one (400 MB, 62 us).
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                   __nv_bfloat16* __restrict__ dx, float* __restrict__ part, int T, int H) {
  __shared__ float red[2][THREADS / 32];
  const int nvec = H >> 3;
  int4 wv[VPT], xv[VPT], dv[VPT];
  float dwacc[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * THREADS;
    wv[i] = v < nvec ? *reinterpret_cast<const int4*>(w + 8 * v) : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
  }
  auto load = [&](int row) {
    const int64_t base = static_cast<int64_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * THREADS;
      xv[i] = v < nvec ? ld_nc_v4(x + base + 8 * v) : make_int4(0, 0, 0, 0);
      dv[i] = v < nvec ? ld_nc_v4(dy + base + 8 * v) : make_int4(0, 0, 0, 0);
    }
  };
  int parity = 0;
  load(blockIdx.x);
  for (int row = blockIdx.x; row < T; row += gridDim.x, parity ^= 1) {
    const float rstd = rstd_in[row];
    int4 cx[VPT], cd[VPT], cr[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      cx[i] = xv[i];
      cd[i] = dv[i];
      const int v = threadIdx.x + i * THREADS;
      cr[i] = dres != nullptr && v < nvec ? ld_nc_v4(dres + static_cast<int64_t>(row) * H + 8 * v) : make_int4(0, 0, 0, 0);
    }
    if (row + gridDim.x < T) load(row + gridDim.x);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const uint32_t* xu = reinterpret_cast<const uint32_t*>(&cx[i]);
      const uint32_t* du = reinterpret_cast<const uint32_t*>(&cd[i]);
      const uint32_t* wu = reinterpret_cast<const uint32_t*>(&wv[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack_bf16(xu[j]), df = unpack_bf16(du[j]), wf = unpack_bf16(wu[j]);
        const float p0 = df.x * (xf.x * rstd), p1 = df.y * (xf.y * rstd);
        dwacc[i][2 * j] += p0;
        dwacc[i][2 * j + 1] += p1;
        dot += p0 * wf.x + p1 * wf.y;
      }
    }
    dot = block_sum_once<THREADS>(dot, red, parity) / static_cast<float>(H);
    __nv_bfloat16* dxr = dx + static_cast<int64_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        const uint32_t* xu = reinterpret_cast<const uint32_t*>(&cx[i]);
        const uint32_t* du = reinterpret_cast<const uint32_t*>(&cd[i]);
        const uint32_t* wu = reinterpret_cast<const uint32_t*>(&wv[i]);
        const uint32_t* ru = reinterpret_cast<const uint32_t*>(&cr[i]);
        int4 o;
        uint32_t* ou = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 xf = unpack_bf16(xu[j]), df = unpack_bf16(du[j]), wf = unpack_bf16(wu[j]), rf = unpack_bf16(ru[j]);
          ou[j] = pack_bf16(rstd * (df.x * wf.x - xf.x * rstd * dot) + rf.x, rstd * (df.y * wf.y - xf.y * rstd * dot) + rf.y);
        }
        st_v4(dxr + 8 * v, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * THREADS;
    if (v < nvec) {
      float* o = part + static_cast<int64_t>(blockIdx.x) * H + 8 * v;
      *reinterpret_cast<float4*>(o) = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
      *reinterpret_cast<float4*>(o + 4) = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
    }
  }
}

// out[c] = sum over rows of part[rows, H], fp32 or bf16: 32 columns a block, 16 threads a column, summed in a fixed order
__global__ void __launch_bounds__(512)
rmsnorm_dw_kernel(const float* __restrict__ part, int rows, int H, float* __restrict__ out32, __nv_bfloat16* __restrict__ out16) {
  __shared__ float red[16][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int r = ty; r < rows; r += 16) s += part[static_cast<int64_t>(r) * H + c];
  }
  red[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < H) {
    s = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += red[i][tx];
    if (out32) out32[c] = s;
    else out16[c] = __float2bfloat16(s);
  }
}

// Rotary embedding (rotate-half / NeoX convention), in place on the q and k heads of a packed
// qkv row [nq*d | nkv*d | nkv*d]; optionally appends the rotated k and the v of each token to a
// paged KV cache laid out [num_blocks, n_kv, block_size, d] at slot_mapping[t] (= block*bs + off).
// `sign` = +1 forward, -1 backward (inverse rotation applied to gradients).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const int64_t* __restrict__ pos,
                            const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int T, int nq,
                            int nkv, int d, int64_t ld, float sign, __nv_bfloat16* __restrict__ k_cache,
                            __nv_bfloat16* __restrict__ v_cache, const int64_t* __restrict__ slot_mapping,
                            int block_size) {
  const int t = blockIdx.x;
  if (t >= T) return;
  const int half = d >> 1;
  const int64_t p = pos[t];
  const float* ct = cos_tab + p * half;
  const float* st = sin_tab + p * half;
  __nv_bfloat16* row = qkv + static_cast<int64_t>(t) * ld;
  const int nrot = (nq + nkv) * half;
  int64_t slot = -1;
  if (slot_mapping) slot = slot_mapping[t];
  const int64_t blk = slot >= 0 ? slot / block_size : 0;
  const int64_t off = slot >= 0 ? slot % block_size : 0;
  for (int i = threadIdx.x; i < nrot; i += blockDim.x) {
    const int h = i / half, j = i - h * half;
    __nv_bfloat16* hp = row + h * d;
    const float x1 = __bfloat162float(hp[j]), x2 = __bfloat162float(hp[j + half]);
    const float c = ct[j], s = st[j] * sign;
    const __nv_bfloat16 o1 = __float2bfloat16(x1 * c - x2 * s);
    const __nv_bfloat16 o2 = __float2bfloat16(x2 * c + x1 * s);
    hp[j] = o1;
    hp[j + half] = o2;
    if (slot >= 0 && h >= nq) {
      __nv_bfloat16* kc = k_cache + ((blk * nkv + (h - nq)) * block_size + off) * d;
      kc[j] = o1;
      kc[j + half] = o2;
    }
  }
  if (slot >= 0) {
    const __nv_bfloat16* vrow = row + (nq + nkv) * d;
    for (int i = threadIdx.x; i < nkv * d; i += blockDim.x) {
      const int h = i / d, j = i - h * d;
      v_cache[((blk * nkv + h) * block_size + off) * d + j] = vrow[i];
    }
  }
}

// Keys and values of cached positions, gathered out of the paged cache for the packed attention: position t of head h is row
// [blk[t], h, off[t], :] of a cache laid out [pages, nkv, page, d].  One thread moves 16 bytes of the key and of the value, so a row is
// read and written in whole 128-byte lines.  Indices below zero count from the end; one outside the cache fails an assertion, as in the
// library's indexing.
// Bound by HBM (13.3 K positions, 8 heads of 128: 109 MB: about 24 us; the library's elementwise index kernels, two launches, took 176 us).
__global__ void __launch_bounds__(256)
gather_pages_kernel(const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc, const int64_t* __restrict__ blk,
                    const int64_t* __restrict__ off, __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v, int T, int64_t pages, int nkv,
                    int page, int units) {
  const int64_t n = static_cast<int64_t>(T) * nkv * units;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const int64_t row = i / units;
    const int u = static_cast<int>(i - row * units);
    const int t = static_cast<int>(row / nkv), h = static_cast<int>(row - static_cast<int64_t>(t) * nkv);
    int64_t b = blk[t], o = off[t];
    b += b < 0 ? pages : 0;
    o += o < 0 ? page : 0;
    assert(b >= 0 && b < pages && o >= 0 && o < page && "index outside the cache");
    const int64_t src = (((b * nkv + h) * page + o) * units + u) * 8;
    const int4 a = ld_nc_v4(kc + src), c = ld_nc_v4(vc + src);
    st_v4(k + i * 8, a);
    st_v4(v + i * 8, c);
  }
}

// SwiGLU backward on the block-interleaved layout ([128 gate | 128 up] per 256 columns):
// dG = dH * u * sig(g) * (1 + g*(1-sig(g))),  dU = dH * silu(g)
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dh,
                                  __nv_bfloat16* __restrict__ dgu, int64_t T, int F) {
  const int64_t nvec = T * (F >> 3);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / (F >> 3);
    const int c = static_cast<int>(i - t * (F >> 3)) * 8;       // column in H
    const int blk = c >> 7, in = c & 127;
    const int64_t gcol = static_cast<int64_t>(blk) * 256 + in;
    const __nv_bfloat16* gp = gu + t * 2 * F + gcol;
    const int4 gq = ld_nc_v4(gp), uq = ld_nc_v4(gp + 128), dq = ld_nc_v4(dh + t * F + c);
    const uint32_t* gu32 = reinterpret_cast<const uint32_t*>(&gq);
    const uint32_t* uu32 = reinterpret_cast<const uint32_t*>(&uq);
    const uint32_t* du32 = reinterpret_cast<const uint32_t*>(&dq);
    int4 og, ou;
    uint32_t* ogu = reinterpret_cast<uint32_t*>(&og);
    uint32_t* ouu = reinterpret_cast<uint32_t*>(&ou);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = unpack_bf16(gu32[j]), u = unpack_bf16(uu32[j]), d = unpack_bf16(du32[j]);
      const float s0 = 1.f / (1.f + __expf(-g.x)), s1 = 1.f / (1.f + __expf(-g.y));
      ogu[j] = pack_bf16(d.x * u.x * s0 * (1.f + g.x * (1.f - s0)), d.y * u.y * s1 * (1.f + g.y * (1.f - s1)));
      ouu[j] = pack_bf16(d.x * g.x * s0, d.y * g.y * s1);
    }
    __nv_bfloat16* op = dgu + t * 2 * F + gcol;
    st_v4(op, og);
    st_v4(op + 128, ou);
  }
}

// Per-row dynamic fp8 (e4m3) quantisation: scale = amax/448; q = x/scale.
__global__ void __launch_bounds__(256)
quant_fp8_rowwise_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale,
                         int T, int H) {
  __shared__ float red[8];
  grid_behind();
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    const __nv_bfloat16* xr = x + static_cast<int64_t>(row) * H;
    float amax = 0.f;
    for (int i = threadIdx.x * 8; i < H; i += 256 * 8) {
      const int4 v = ld_nc_v4(xr + i);
      const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16(u[j]);
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
    amax = warp_max(amax);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
    const float sc = fmaxf(amax, 1e-12f) / 448.f;
    const float inv = 1.f / sc;
    if (threadIdx.x == 0) scale[row] = sc;
    uint8_t* qr = q + static_cast<int64_t>(row) * H;
    for (int i = threadIdx.x * 8; i < H; i += 256 * 8) {
      const int4 v = ld_nc_v4(xr + i);
      const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
      uint32_t o[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 a = unpack_bf16(u[2 * j]), b = unpack_bf16(u[2 * j + 1]);
        uint16_t lo, hi;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(a.y * inv), "f"(a.x * inv));
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(b.y * inv), "f"(b.x * inv));
        o[j] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
      }
      *reinterpret_cast<uint2*>(qr + i) = make_uint2(o[0], o[1]);
    }
  }
}

}  // namespace prl

using namespace prl;

// block shape for a row of H values: the fewest vectors a thread holds
template <class F>
static void norm_shape(int H, F&& f) {
  const int nvec = H / 8;
  if (nvec <= 128) f(std::integral_constant<int, 128>{}, std::integral_constant<int, 1>{});
  else if (nvec <= 256) f(std::integral_constant<int, 256>{}, std::integral_constant<int, 1>{});
  else if (nvec <= 512) f(std::integral_constant<int, 256>{}, std::integral_constant<int, 2>{});
  else f(std::integral_constant<int, 512>{}, std::integral_constant<int, 2>{});
}

extern "C" int prl_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int T, int H, float eps,
                               cudaStream_t s) {
  if (H % 8 != 0 || H > 8 * kNormThreads * kMaxVPT) return -20;
  if (T <= 0) return 0;
  norm_shape(H, [&](auto threads, auto vpt) {
    constexpr int kT = decltype(threads)::value;
    const int most = 148 * (2048 / kT / 2), grid = T < most ? T : most;       // 1024 threads an SM: two rows' loads in flight for each
    auto kern = rmsnorm_fwd_kernel<kT, decltype(vpt)::value>;
    const auto* xb = static_cast<const __nv_bfloat16*>(x);
    const auto* wb = static_cast<const __nv_bfloat16*>(w);
    if (T <= kStepRows) launch_behind(kern, grid, kT, 0, s, xb, wb, static_cast<__nv_bfloat16*>(y), rstd, T, H, eps);
    else kern<<<grid, kT, 0, s>>>(xb, wb, static_cast<__nv_bfloat16*>(y), rstd, T, H, eps);
  });
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
extern "C" int prl_add_rmsnorm(void* x, const void* r, const void* w, void* y, int T, int H, float eps, cudaStream_t s) {
  if (H % 8 != 0 || H > 8 * kNormThreads * kMaxVPT) return -20;
  if (T <= 0) return 0;
  const int grid = T < 148 * 8 ? T : 148 * 8;
  auto* xb = static_cast<__nv_bfloat16*>(x);
  const auto* rb = static_cast<const __nv_bfloat16*>(r);
  const auto* wb = static_cast<const __nv_bfloat16*>(w);
  if (T <= kStepRows) launch_behind(add_rmsnorm_kernel, grid, kNormThreads, 0, s, xb, rb, wb, static_cast<__nv_bfloat16*>(y), T, H, eps);
  else add_rmsnorm_kernel<<<grid, kNormThreads, 0, s>>>(xb, rb, wb, static_cast<__nv_bfloat16*>(y), T, H, eps);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
// blocks of the backward pass, which is the number of rows of `part`: 512 threads an SM, at least two rows a block
extern "C" int prl_rmsnorm_bwd_parts(int T, int H) {
  const int threads = H <= 1024 ? 128 : H <= 4096 ? 256 : 512, most = 148 * (512 / threads);
  const int want = (T + 1) / 2;
  return want < most ? want : most;
}
// part: [prl_rmsnorm_bwd_parts, H] floats of scratch; dres may be null; the gain's gradient goes to dw32 or, if that is null, to dw16
extern "C" int prl_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx, float* part, float* dw32,
                               void* dw16, int T, int H, cudaStream_t s) {
  if (H % 8 != 0 || H > 8 * kNormThreads * kMaxVPT) return -20;
  const int grid = T > 0 ? prl_rmsnorm_bwd_parts(T, H) : 0;
  if (grid > 0)
    norm_shape(H, [&](auto threads, auto vpt) {
      constexpr int kT = decltype(threads)::value;
      rmsnorm_bwd_kernel<kT, decltype(vpt)::value><<<grid, kT, 0, s>>>(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w),
                                                                      static_cast<const __nv_bfloat16*>(dy), rstd,
                                                                      static_cast<const __nv_bfloat16*>(dres), static_cast<__nv_bfloat16*>(dx), part, T, H);
    });
  PRL_CUDA_CHECK(cudaGetLastError());
  rmsnorm_dw_kernel<<<(H + 31) / 32, 512, 0, s>>>(part, grid, H, dw32, static_cast<__nv_bfloat16*>(dw16));
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
extern "C" int prl_rope(void* qkv, const int64_t* pos, const float* cos_tab, const float* sin_tab, int T, int nq,
                        int nkv, int d, int64_t ld, float sign, void* k_cache, void* v_cache,
                        const int64_t* slot_mapping, int block_size, cudaStream_t s) {
  if (T <= 0) return 0;
  rope_kernel<<<T, 256, 0, s>>>(static_cast<__nv_bfloat16*>(qkv), pos, cos_tab, sin_tab, T, nq, nkv, d, ld, sign,
                                static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache),
                                slot_mapping, block_size);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
extern "C" int prl_gather_pages(const void* kc, const void* vc, const int64_t* blk, const int64_t* off, void* k, void* v, int T, int64_t pages, int nkv,
                                int page, int d, cudaStream_t s) {
  if (d % 8 != 0) return -23;
  if (T <= 0 || nkv <= 0) return 0;
  const int64_t blocks = (static_cast<int64_t>(T) * nkv * (d / 8) + 255) / 256;
  gather_pages_kernel<<<static_cast<unsigned>(blocks < 148 * 64 ? blocks : 148 * 64), 256, 0, s>>>(
      static_cast<const __nv_bfloat16*>(kc), static_cast<const __nv_bfloat16*>(vc), blk, off, static_cast<__nv_bfloat16*>(k),
      static_cast<__nv_bfloat16*>(v), T, pages, nkv, page, d / 8);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
extern "C" int prl_swiglu_bwd(const void* gu, const void* dh, void* dgu, int64_t T, int F, cudaStream_t s) {
  if (F % 128 != 0) return -21;
  if (T <= 0) return 0;
  const int64_t nvec = T * (F / 8);
  int grid = static_cast<int>((nvec + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  swiglu_bwd_kernel<<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dh),
                                         static_cast<__nv_bfloat16*>(dgu), T, F);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
extern "C" int prl_quant_fp8_rowwise(const void* x, void* q, float* scale, int T, int H, cudaStream_t s) {
  if (H % 8 != 0) return -22;
  if (T <= 0) return 0;
  const int grid = T < 148 * 8 ? T : 148 * 8;
  const auto* xb = static_cast<const __nv_bfloat16*>(x);
  if (T <= kStepRows) launch_behind(quant_fp8_rowwise_kernel, grid, 256, 0, s, xb, static_cast<uint8_t*>(q), scale, T, H);
  else quant_fp8_rowwise_kernel<<<grid, 256, 0, s>>>(xb, static_cast<uint8_t*>(q), scale, T, H);
  PRL_CUDA_CHECK(cudaGetLastError());
  return 0;
}
