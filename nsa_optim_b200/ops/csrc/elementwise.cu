// Bandwidth-bound kernels: RMSNorm / gated RMSNorm / L2 norm (forward + backward),
// SwiGLU, rotary embedding, causal depthwise conv1d (+SiLU), embedding gather and its
// deterministic scatter-add backward.  bf16 storage, fp32 arithmetic, 16-byte accesses.
//
// Row kernels keep a whole row in registers.  Rows up to 512 elements use one warp per row, longer
// rows (up to 8192) one CTA of 256 threads per row, or of 512 in the norm backward's wider forms.
// Weight gradients of the norms and the convolution are reduced deterministically:
// a persistent grid accumulates per-CTA partial sums into a scratch buffer
// [grid, width] (fp32) that a second kernel adds up in a fixed order.
#include "f32x2.cuh"
#include "host.cuh"
#include <cuda_bf16.h>

namespace {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void store8(bf16* p, const float (&v)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }
// d/dx silu(x)
__device__ __forceinline__ float dsilu_f(float x) {
  float s = sigmoid_f(x);
  return s * (1.f + x * (1.f - s));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sum over the TPR threads that share a row.  TPR == 32: warp; TPR == 256: whole CTA.
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float* red) {
  v = warp_sum(v);
  if (TPR == 32) return v;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < TPR / 32; ++i) t += red[i];
  return t;
}

// ------------------------------------------------------------------------------------
// (gated) RMSNorm.  MODE 0: y = x*rstd*w.   MODE 1: y = x*rstd*w * silu(g)   (norm, then gate)
//                   MODE 2: u = x*silu(g); y = u*rstd(u)*w                    (gate, then norm)
// ------------------------------------------------------------------------------------
template <int TPR, int NV, int MODE>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ g,
                                                          const bf16* __restrict__ w, bf16* __restrict__ y,
                                                          float* __restrict__ rstd_out, long rows, int d, float eps,
                                                          long ldg) {
  __shared__ float red[8];
  const int rows_per_cta = 256 / TPR;
  const long row = static_cast<long>(blockIdx.x) * rows_per_cta + threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const bool active = row < rows;
  float xv[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    if (active && c < d) {
      load8(x + row * d + c, xv[i]);
      if (MODE == 2) {
        float gv[8];
        load8(g + row * ldg + c, gv);
#pragma unroll
        for (int j = 0; j < 8; ++j) xv[i][j] *= silu_f(gv[j]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += xv[i][j] * xv[i][j];
    }
  }
  ss = row_sum<TPR>(ss, red);
  const float rstd = rsqrtf(ss / d + eps);
  if (active && t == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    if (active && c < d) {
      float wv[8], o[8];
      load8(w + c, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = xv[i][j] * rstd * wv[j];
      if (MODE == 1) {
        float gv[8];
        load8(g + row * ldg + c, gv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] *= silu_f(gv[j]);
      }
      store8(y + row * d + c, o);
    }
  }
}

// Residual add fused into the plain norm: h = x + r (rounded to bf16, written out because the
// residual stream continues from it) and y = h * rstd(h) * w, one read of x and r, one write of
// h and y.  The statistics use the rounded h, so the result equals add-then-norm to the bit.
template <int TPR, int NV>
__global__ void __launch_bounds__(256) rmsnorm_add_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ r,
                                                              const bf16* __restrict__ w, bf16* __restrict__ h,
                                                              bf16* __restrict__ y, float* __restrict__ rstd_out,
                                                              long rows, int d, float eps) {
  __shared__ float red[8];
  const int rows_per_cta = 256 / TPR;
  const long row = static_cast<long>(blockIdx.x) * rows_per_cta + threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const bool active = row < rows;
  float hv[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    if (active && c < d) {
      float rv[8];
      load8(x + row * d + c, hv[i]);
      load8(r + row * d + c, rv);
#pragma unroll
      for (int j = 0; j < 8; ++j) hv[i][j] = __bfloat162float(__float2bfloat16(hv[i][j] + rv[j]));
      store8(h + row * d + c, hv[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += hv[i][j] * hv[i][j];
    }
  }
  ss = row_sum<TPR>(ss, red);
  const float rstd = rsqrtf(ss / d + eps);
  if (active && t == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    if (active && c < d) {
      float wv[8], o[8];
      load8(w + c, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = hv[i][j] * rstd * wv[j];
      store8(y + row * d + c, o);
    }
  }
}

// Backward.  Persistent over rows; writes dx (and dg for gated modes) and per-CTA partial
// dw into `partial[gridDim.x][d]`.  `dres` (may be null) is a gradient that reaches the norm's
// input by another route (the residual stream); it is added into dx here instead of by a
// separate pass over both tensors.
//
// Bound by memory traffic, so by the bytes in flight per SM.  A row that a CTA shares ends in two barriers: what helps is the
// next row's operands in flight behind them, as long as a thread's part of a row is one 16-byte piece: TPR 256 up to 2048
// columns, 512 up to 4096 (two pieces a thread ahead leave one CTA of 256 threads per SM: 65536 x 4096, gate first, 757 us,
// 732 without looking ahead, 603 with 512 threads; plain 545, 502, 300).  Above 4096 columns all loads of a row are issued
// together and held (32768 x 8192, plain: 408 us, 752 read where they are used), but with the gate first that
// spills, and 512 threads that read x again take 765 us instead of 1045.  A row of one warp (TPR 32, up to 512 columns) meets
// no barrier: its warps run apart and hide each other's loads, so the registers go to more warps, and x and dres are read
// again where they are used.  1048576 x 128: 260 us plain and 407 norm first (516 and 604 with the next row in registers:
// two CTAs instead of four and three); 262144 x 512: 169 plain, 320 gate first (311 and 415).
// CTAs per SM that the registers leave room for:
template <int TPR, int NV, int MODE>
constexpr int rms_bwd_ctas = TPR == 32    ? (NV == 1 ? (MODE == 0 ? 4 : 3) : (MODE == 0 ? 3 : 2))
                             : NV > 1     ? 1
                             : TPR == 256 ? (MODE == 0 ? 4 : 2)
                                          : (MODE == 0 ? 2 : 1);
template <int TPR>
constexpr int rms_bwd_threads = TPR > 256 ? TPR : 256;
template <int TPR, int NV, int MODE>
__global__ void __launch_bounds__(rms_bwd_threads<TPR>, rms_bwd_ctas<TPR, NV, MODE>)
rmsnorm_bwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ g, const bf16* __restrict__ w, const bf16* __restrict__ dy,
                   const float* __restrict__ rstd_in, bf16* __restrict__ dx, bf16* __restrict__ dg, float* __restrict__ partial,
                   long rows, int d, const bf16* __restrict__ dres = nullptr, long ldg = 0) {
  __shared__ float red[rms_bwd_threads<TPR> / 32];
  __shared__ float dw_sh[(TPR == 32) ? 512 : 1];
  const int rows_per_cta = rms_bwd_threads<TPR> / TPR;
  const int sub = threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  float dwacc[NV][8];
  float wv[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
    if (c < d) load8(w + c, wv[i]);
  }
  // HELD: a row's operands are loaded together and kept as they came; AHEAD: one row early.
  constexpr bool AHEAD = TPR > 32 && NV == 1, HELD = AHEAD || NV == 4;
  uint4 nx[NV], ndy[NV], ng[NV], nr[NV];
  auto fetch = [&](long row) {
    if (row >= rows) return;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (t + i * TPR) * 8;
      if (c >= d) continue;
      nx[i] = *reinterpret_cast<const uint4*>(x + row * d + c);
      ndy[i] = *reinterpret_cast<const uint4*>(dy + row * d + c);
      if (MODE != 0) ng[i] = *reinterpret_cast<const uint4*>(g + row * (ldg ? ldg : d) + c);
      if (dres != nullptr) nr[i] = *reinterpret_cast<const uint4*>(dres + row * d + c);
    }
  };
  const long stride = static_cast<long>(gridDim.x) * rows_per_cta;
  if (AHEAD) fetch(static_cast<long>(blockIdx.x) * rows_per_cta + sub);
  for (long base = static_cast<long>(blockIdx.x) * rows_per_cta; base < rows; base += stride) {
    const long row = base + sub;
    const bool active = row < rows;
    const float rstd = active ? rstd_in[row] : 0.f;
    if (HELD && !AHEAD) fetch(row);
    uint4 cx[NV], cr[NV];
    float xn[NV][8], wdy[NV][8], gv[NV][8], sg[NV][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (t + i * TPR) * 8;
      if (active && c < d) {
        float xv[8], dv[8];
        if (HELD) {
          cx[i] = nx[i];
          cr[i] = nr[i];
          unpack8(nx[i], xv);
          unpack8(ndy[i], dv);
          if (MODE != 0) unpack8(ng[i], gv[i]);
        } else {
          load8(x + row * d + c, xv);
          load8(dy + row * d + c, dv);
          if (MODE != 0) load8(g + row * (ldg ? ldg : d) + c, gv[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float xin = xv[j];
          float dout = dv[j];
          if (MODE == 2) { sg[i][j] = silu_f(gv[i][j]); xin *= sg[i][j]; }
          xn[i][j] = xin * rstd;
          if (MODE == 1) {
            // y = n*w*silu(g): dg = dy*n*w*dsilu(g); upstream for the norm is dy*silu(g)
            const float s = silu_f(gv[i][j]);
            sg[i][j] = dout * xn[i][j] * wv[i][j] * dsilu_f(gv[i][j]);   // dg
            dout *= s;
          }
          dwacc[i][j] += dout * xn[i][j];
          wdy[i][j] = dout * wv[i][j];
          dot += wdy[i][j] * xn[i][j];
        }
      }
    }
    if (AHEAD) fetch(row + stride);
    dot = row_sum<TPR>(dot, red) / d;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (t + i * TPR) * 8;
      if (active && c < d) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (wdy[i][j] - xn[i][j] * dot);   // d/d(norm input)
        if (MODE == 2) {
          // norm input u = x*silu(g): dx = du*silu(g), dg = du*x*dsilu(g)
          float xv[8], og[8];
          if (HELD) unpack8(cx[i], xv);
          else load8(x + row * d + c, xv);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            og[j] = o[j] * xv[j] * dsilu_f(gv[i][j]);
            o[j] *= sg[i][j];
          }
          store8(dg + row * d + c, og);
        } else if (MODE == 1) {
          store8(dg + row * d + c, sg[i]);
        }
        if (dres != nullptr) {
          float rv[8];
          if (HELD) unpack8(cr[i], rv);
          else load8(dres + row * d + c, rv);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rv[j];
        }
        store8(dx + row * d + c, o);
      }
    }
  }
  // per-CTA partial dw
  if (TPR == 32) {
    // 8 sub-rows share columns: combine through shared memory in a fixed order
    for (int i = 0; i < NV; ++i) {
      const int c = (t + i * TPR) * 8;
      for (int s = 0; s < rows_per_cta; ++s) {
        __syncthreads();
        if (sub == s && c < d) {
#pragma unroll
          for (int j = 0; j < 8; ++j) dw_sh[c + j] = (s == 0 ? 0.f : dw_sh[c + j]) + dwacc[i][j];
        }
      }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < d; c += 256) partial[static_cast<long>(blockIdx.x) * d + c] = dw_sh[c];
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (t + i * TPR) * 8;
      if (c < d) {
#pragma unroll
        for (int j = 0; j < 8; ++j) partial[static_cast<long>(blockIdx.x) * d + c + j] = dwacc[i][j];
      }
    }
  }
}

// out[c] = sum_p partial[p][c] in a fixed order; bf16 or fp32 output.  CTA: 32 columns x 32 groups of parts (a thread per
// column walking all parts took 25 us for 592 x 2048: one dependent stream of reads on eight CTAs).
__global__ void __launch_bounds__(1024) reduce_partials_kernel(const float* __restrict__ partial, int parts, int width,
                                                               bf16* __restrict__ out_bf16, float* __restrict__ out_f32) {
  __shared__ float sums[32][33];
  const int l = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.x * 32 + l;
  float s = 0.f;
  if (c < width) {
#pragma unroll 4
    for (int p = g; p < parts; p += 32) s += partial[static_cast<long>(p) * width + c];
  }
  sums[g][l] = s;
  __syncthreads();
  // warp g finishes column g of the tile: 32 group sums meet by shuffles
  s = warp_sum(sums[l][g]);
  const int cg = blockIdx.x * 32 + g;
  if (l == 0 && cg < width) {
    if (out_bf16) out_bf16[cg] = __float2bfloat16(s);
    if (out_f32) out_f32[cg] = s;
  }
}

// ------------------------------------------------------------------------------------
// L2 norm over the last dimension (d <= 512, warp per row)
// ------------------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(256) l2norm_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y,
                                                         float* __restrict__ rinv_out, long rows, int d, float eps) {
  const long row = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int t = threadIdx.x & 31;
  if (row >= rows) return;
  float xv[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * 32) * 8;
    if (c < d) {
      load8(x + row * d + c, xv[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += xv[i][j] * xv[i][j];
    }
  }
  ss = warp_sum(ss);
  const float rinv = rsqrtf(ss + eps);
  if (t == 0) rinv_out[row] = rinv;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * 32) * 8;
    if (c < d) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = xv[i][j] * rinv;
      store8(y + row * d + c, o);
    }
  }
}
template <int NV>
__global__ void __launch_bounds__(256) l2norm_bwd_kernel(const bf16* __restrict__ y, const bf16* __restrict__ dy,
                                                         const float* __restrict__ rinv_in, bf16* __restrict__ dx,
                                                         long rows, int d) {
  const long row = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int t = threadIdx.x & 31;
  if (row >= rows) return;
  float yv[NV][8], dv[NV][8];
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * 32) * 8;
    if (c < d) {
      load8(y + row * d + c, yv[i]);
      load8(dy + row * d + c, dv[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += yv[i][j] * dv[i][j];
    }
  }
  dot = warp_sum(dot);
  const float rinv = rinv_in[row];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * 32) * 8;
    if (c < d) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rinv * (dv[i][j] - yv[i][j] * dot);
      store8(dx + row * d + c, o);
    }
  }
}

// ------------------------------------------------------------------------------------
// SwiGLU
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const bf16* __restrict__ g, const bf16* __restrict__ u,
                                                         bf16* __restrict__ y, long n8, int cols8, long ldg8, long ldu8) {
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long r = i / cols8, c = i - r * cols8;
    float gv[8], uv[8], o[8];
    load8(g + (r * ldg8 + c) * 8, gv);
    load8(u + (r * ldu8 + c) * 8, uv);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = silu_f(gv[j]) * uv[j];
    store8(y + i * 8, o);
  }
}
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const bf16* __restrict__ g, const bf16* __restrict__ u,
                                                         const bf16* __restrict__ dy, bf16* __restrict__ dg,
                                                         bf16* __restrict__ du, long n8, int cols8, long ldg8, long ldu8,
                                                         long ldo8) {
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long r = i / cols8, c = i - r * cols8;
    float gv[8], uv[8], dv[8], o1[8], o2[8];
    load8(g + (r * ldg8 + c) * 8, gv);
    load8(u + (r * ldu8 + c) * 8, uv);
    load8(dy + i * 8, dv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o1[j] = dv[j] * uv[j] * dsilu_f(gv[j]);
      o2[j] = dv[j] * silu_f(gv[j]);
    }
    store8(dg + (r * ldo8 + c) * 8, o1);
    store8(du + (r * ldo8 + c) * 8, o2);
  }
}

// ------------------------------------------------------------------------------------
// Gated combine of the three sparse-attention branches: o = g1 o1 + g2 o2 + g3 o3 with one gate
// per (token, head) row.  Backward: do_i = g_i do and dg_i = sum_d do * o_i.  LANES = D / 8 threads
// share a row (8 elements each); LANES is a power of two <= 32 so a row never straddles a warp.
// ------------------------------------------------------------------------------------
template <int LANES>
__global__ void __launch_bounds__(256) gate_combine_fwd_kernel(const bf16* __restrict__ o1, const bf16* __restrict__ o2,
                                                               const bf16* __restrict__ o3, const bf16* __restrict__ g1,
                                                               const bf16* __restrict__ g2, const bf16* __restrict__ g3,
                                                               bf16* __restrict__ o, long n8, int Hq, long ldg, int sig) {
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long row = i / LANES;
    const long gi = (row / Hq) * ldg + row % Hq;           // gates: [tokens, Hq] with row pitch ldg
    float a = __bfloat162float(g1[gi]), b = __bfloat162float(g2[gi]), c = __bfloat162float(g3[gi]);
    if (sig) { a = sigmoid_f(a); b = sigmoid_f(b); c = sigmoid_f(c); }   // gates given as logits
    float x[8], y[8], z[8], r[8];
    load8(o1 + i * 8, x);
    load8(o2 + i * 8, y);
    load8(o3 + i * 8, z);
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = a * x[j] + b * y[j] + c * z[j];
    store8(o + i * 8, r);
  }
}
// SUMS: e_i also receives rowsum(do_i * o_i), do_i as rounded (2097152 rows of 128: 617 us with, 570 without).
template <int LANES, bool SUMS>
__global__ void __launch_bounds__(256) gate_combine_bwd_kernel(const bf16* __restrict__ o1, const bf16* __restrict__ o2,
                                                               const bf16* __restrict__ o3, const bf16* __restrict__ g1,
                                                               const bf16* __restrict__ g2, const bf16* __restrict__ g3,
                                                               const bf16* __restrict__ d_o, bf16* __restrict__ do1,
                                                               bf16* __restrict__ do2, bf16* __restrict__ do3,
                                                               bf16* __restrict__ dg1, bf16* __restrict__ dg2,
                                                               bf16* __restrict__ dg3, float* __restrict__ e1,
                                                               float* __restrict__ e2, float* __restrict__ e3, long n8, int Hq,
                                                               long ldg, int sig) {
  // the grid is sized so that every thread handles exactly one vector (rows stay inside a warp)
  const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool live = i < n8;
  const long row = (live ? i : 0) / LANES;
  float s1 = 0.f, s2 = 0.f, s3 = 0.f, t1 = 0.f, t2 = 0.f, t3 = 0.f;
  const long gi = (row / Hq) * ldg + row % Hq;
  float a = 0.f, b = 0.f, c = 0.f;
  if (live) {
    a = __bfloat162float(g1[gi]); b = __bfloat162float(g2[gi]); c = __bfloat162float(g3[gi]);
    if (sig) { a = sigmoid_f(a); b = sigmoid_f(b); c = sigmoid_f(c); }
    float x[8], y[8], z[8], d[8], r[8];
    load8(o1 + i * 8, x);
    load8(o2 + i * 8, y);
    load8(o3 + i * 8, z);
    load8(d_o + i * 8, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) { s1 += d[j] * x[j]; s2 += d[j] * y[j]; s3 += d[j] * z[j]; }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      r[j] = a * d[j];
      if (SUMS) { r[j] = __bfloat162float(__float2bfloat16(r[j])); t1 += r[j] * x[j]; }
    }
    store8(do1 + i * 8, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      r[j] = b * d[j];
      if (SUMS) { r[j] = __bfloat162float(__float2bfloat16(r[j])); t2 += r[j] * y[j]; }
    }
    store8(do2 + i * 8, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      r[j] = c * d[j];
      if (SUMS) { r[j] = __bfloat162float(__float2bfloat16(r[j])); t3 += r[j] * z[j]; }
    }
    store8(do3 + i * 8, r);
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    s3 += __shfl_xor_sync(0xffffffffu, s3, o);
  }
  if (SUMS) {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
      t3 += __shfl_xor_sync(0xffffffffu, t3, o);
    }
    if (live && (threadIdx.x % LANES) == 0) { e1[row] = t1; e2[row] = t2; e3[row] = t3; }
  }
  if (live && (threadIdx.x % LANES) == 0) {
    // gates given as logits: the gradient goes back through the sigmoid here
    if (sig) { s1 *= a * (1.f - a); s2 *= b * (1.f - b); s3 *= c * (1.f - c); }
    dg1[gi] = __float2bfloat16(s1);
    dg2[gi] = __float2bfloat16(s2);
    dg3[gi] = __float2bfloat16(s3);
  }
}

// ------------------------------------------------------------------------------------
// Mean pooling of keys / values into compressed blocks (native sparse attention):
//   y[b, i, :] = mean over t in [i*stride, i*stride + block) of x[b, t, :]
// x rows are `width` = Hkv * D elements with row pitch ldx; y is contiguous [B, nC, width].
// Backward: dx[b, t, :] = (1/block) * sum of dy[b, i, :] over the windows i that contain t.
// One thread per 8 elements; fp32 accumulation in a fixed order.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) nsa_pool_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, int T, int nC,
                                                           int width8, long ldx, int block, int stride, long n) {
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int c8 = static_cast<int>(i % width8);
    const long r = i / width8;
    const int ci = static_cast<int>(r % nC);
    const long b = r / nC;
    const bf16* src = x + (b * T + static_cast<long>(ci) * stride) * ldx + c8 * 8;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int t = 0; t < block; ++t) {
      float v[8];
      load8(src + t * ldx, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
    const float inv = 1.f / block;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= inv;
    store8(y + i * 8, acc);
  }
}
__global__ void __launch_bounds__(256) nsa_pool_bwd_kernel(const bf16* __restrict__ dy, bf16* __restrict__ dx, int T, int nC,
                                                           int width8, int block, int stride, long n) {
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int c8 = static_cast<int>(i % width8);
    const long r = i / width8;
    const int t = static_cast<int>(r % T);
    const long b = r / T;
    int lo = t - block + 1;
    lo = lo <= 0 ? 0 : (lo + stride - 1) / stride;
    int hi = t / stride;
    hi = hi < nC - 1 ? hi : nC - 1;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int ci = lo; ci <= hi; ++ci) {
      float v[8];
      load8(dy + ((b * nC + ci) * width8 + c8) * 8, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
    const float inv = 1.f / block;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= inv;
    store8(dx + i * 8, acc);
  }
}

// ------------------------------------------------------------------------------------
// Rotary embedding, halves layout.  x (tokens T per batch, H heads, D); cos/sin (T, D/2).
// sign = +1 forward, -1 backward (rotation by the opposite angle).  In-place safe.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rope_kernel(const bf16* __restrict__ x, const float* __restrict__ cs,
                                                   const float* __restrict__ sn, bf16* __restrict__ y, long n_items,
                                                   int T, int H, int D, float sign) {
  const int d2v = D / 16;   // 8-wide vectors per half
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_items; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % d2v);
    const long bh = i / d2v;            // (b*T + t)*H + h
    const long bt = bh / H;
    const int t = static_cast<int>(bt % T);
    const bf16* px = x + bh * D + v * 8;
    float a[8], b[8], o1[8], o2[8];
    load8(px, a);
    load8(px + D / 2, b);
    const float* pc = cs + static_cast<long>(t) * (D / 2) + v * 8;
    const float* ps = sn + static_cast<long>(t) * (D / 2) + v * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float c = pc[j], s = ps[j] * sign;
      o1[j] = a[j] * c - b[j] * s;
      o2[j] = b[j] * c + a[j] * s;
    }
    bf16* py = y + bh * D + v * 8;
    store8(py, o1);
    store8(py + D / 2, o2);
  }
}

// ------------------------------------------------------------------------------------
// Causal depthwise conv1d, width 4, channel-last (B, T, C), optional bias and SiLU.
// Bound by memory when the arithmetic stays out of the way: a lane owns four channels (8-byte
// accesses, a warp covers 256 contiguous bytes of a row) and walks `rows` consecutive time steps
// with the last three rows in registers, so every element is read and widened once.  The rows ahead
// travel through a ring of shared memory that a lane fills (cp.async) and reads for itself alone: no barriers,
// and 8 rows of a warp stay in flight without holding registers.  Taps, sigmoid and derivative are packed fp32 operations (two
// channels per instruction); groups of rows wholly inside a segment go without a test per row, and addresses are stepped, not formed
// (16384 x 4352, bias and SiLU: forward 64 -> 58 us, 4.9 TB/s, backward 126 -> 105, 4.1 TB/s; 150 instructions a row and warp there,
// now 106, and half of the issue slots: 128 registers leave four warps to a scheduler.  Group-wise order of the steps: 111.  Longer or
// shorter segments and three CTAs per SM with spills: 111, 121, 252).  A CTA is CW channel tiles by 8 / CW time segments: two tiles, or one
// for tensors of up to 128 channels, whose warps would otherwise have nothing to do (four tiles: 108; 4352 channels are 34).
// ------------------------------------------------------------------------------------
constexpr int CT_WARPS = 8, CT_C = 128, CT_U = 4, CT_RING = 3;

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Quad {        // four channels
  float2 a, b;
};
__device__ __forceinline__ Quad quad_unpack(const uint2& u) {
  Quad q;
  q.a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  q.b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return q;
}
__device__ __forceinline__ uint2 quad_pack(const Quad& q) {
  uint2 u;
  *reinterpret_cast<__nv_bfloat162*>(&u.x) = __floats2bfloat162_rn(q.a.x, q.a.y);
  *reinterpret_cast<__nv_bfloat162*>(&u.y) = __floats2bfloat162_rn(q.b.x, q.b.y);
  return u;
}
__device__ __forceinline__ Quad quad_fma(const Quad& x, const Quad& y, const Quad& z) {
  return Quad{fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)};
}
__device__ __forceinline__ Quad quad_zero() { return Quad{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ void conv_taps(const bf16* __restrict__ w, const bf16* __restrict__ bias, int c, bool c_ok,
                                          Quad (&wv)[4], Quad& bv) {
  float t[4][4], s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s[k] = (bias && c_ok) ? __bfloat162float(bias[c + k]) : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j][k] = c_ok ? __bfloat162float(w[(c + k) * 4 + j]) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) wv[j] = Quad{make_float2(t[j][0], t[j][1]), make_float2(t[j][2], t[j][3])};
  bv = Quad{make_float2(s[0], s[1]), make_float2(s[2], s[3])};
}

// Two lanes of silu and of its derivative; the exponential and the reciprocal are the scalar functions'.
__device__ __forceinline__ float2 sigmoid2(const float2& x) {
  const float2 e = mul2(x, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 d = fma2(make_float2(exp2f(e.x), exp2f(e.y)), make_float2(1.f, 1.f), make_float2(1.f, 1.f));
  return make_float2(__fdividef(1.f, d.x), __fdividef(1.f, d.y));
}
__device__ __forceinline__ float2 silu2(const float2& x) { return mul2(x, sigmoid2(x)); }
__device__ __forceinline__ float2 dsilu2(const float2& x) {
  const float2 s = sigmoid2(x), one = make_float2(1.f, 1.f);
  return mul2(s, fma2(x, fma2(s, make_float2(-1.f, -1.f), one), one));
}

// Copies groups of CT_U rows of a lane's four channels into its ring, one after the other; rows past `rows` read as zero.
struct ConvFeed {
  const bf16 *src, *base;
  long pitch;
  int left, slot = 0;
  uint32_t ring;
  __device__ __forceinline__ ConvFeed(const bf16* p, long pitch, int rows, uint2* ring)
      : src(p), base(p), pitch(pitch), left(rows), ring(static_cast<uint32_t>(__cvta_generic_to_shared(ring))) {}
  __device__ __forceinline__ void next(bool commit = true) {
    const uint32_t d = ring + slot * (CT_U * 32 * 8);
    if (left >= CT_U) {
#pragma unroll
      for (int u = 0; u < CT_U; ++u) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + u * 256), "l"(src) : "memory");
        src += pitch;
      }
    } else {
#pragma unroll
      for (int u = 0; u < CT_U; ++u) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + u * 256), "l"(u < left ? src : base), "r"(u < left ? 8 : 0) : "memory");
        src += pitch;
      }
    }
    left -= CT_U;
    slot = (slot + 1) % CT_RING;
    if (commit) cp_async_commit();
  }
};

template <int CW>
__global__ void __launch_bounds__(CT_WARPS * 32, 3) conv1d_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                                      const bf16* __restrict__ bias, bf16* __restrict__ y,
                                                                      int T, int C, long ldx, int act, int rows) {
  __shared__ uint2 ring_all[CT_WARPS][CT_RING * CT_U][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * CW + warp % CW) * CT_C + lane * 4;
  const int t0 = (blockIdx.y * (CT_WARPS / CW) + warp / CW) * rows;
  if (c >= C || t0 >= T) return;
  uint2* ring = &ring_all[warp][0][lane];
  const bf16* xp = x + static_cast<long>(blockIdx.z) * T * ldx + c;
  bf16* yp = y + (static_cast<long>(blockIdx.z) * T + t0) * C + c;
  const int n = min(rows, T - t0);                  // rows of this segment
  const bf16* xs = xp + static_cast<long>(t0) * ldx;
  ConvFeed feed(xs, ldx, n, ring);
#pragma unroll
  for (int g = 0; g < CT_RING - 1; ++g) feed.next();
  auto before = [&](int k) {
    return quad_unpack(t0 >= k ? *reinterpret_cast<const uint2*>(xs - k * ldx) : make_uint2(0u, 0u));
  };
  Quad x0 = before(3), x1 = before(2), x2 = before(1);
  Quad wv[4], bv;
  conv_taps(w, bias, c, true, wv, bv);
  auto row = [&](int u, int g) {
    const Quad x3 = quad_unpack(ring[((g % CT_RING) * CT_U + u) * 32]);
    Quad o = quad_fma(wv[3], x3, quad_fma(wv[2], x2, quad_fma(wv[1], x1, quad_fma(wv[0], x0, bv))));
    x0 = x1; x1 = x2; x2 = x3;
    if (act) o = Quad{silu2(o.a), silu2(o.b)};
    *reinterpret_cast<uint2*>(yp) = quad_pack(o);
    yp += C;
  };
  int g = 0;
  for (; (g + 1) * CT_U <= n; ++g) {
    feed.next();
    cp_async_wait<CT_RING - 1>();
#pragma unroll
    for (int u = 0; u < CT_U; ++u) row(u, g);
  }
  cp_async_wait<0>();
  for (int u = 0; g * CT_U + u < n; ++u) row(u, g);
}

// Backward: dpre[t] = dy[t] (times SiLU'(pre[t]), pre recomputed from x), dx[s] = sum_j w[j] dpre[s + 3 - j],
// dw[j] = sum_t dpre[t] x[t - 3 + j], db = sum_t dpre[t].  The walk of the forward with dx three rows
// behind: a segment also computes dpre on the three rows after its end, which the next one counts.
// Weight and bias gradients stay in registers, the CTA's time segments meet through shared memory in a
// fixed order, and one partial sum leaves per (CTA in time, batch): partial layout [chunk][5][C]
// (row 4 = bias gradient), chunk = blockIdx.z * gridDim.y + blockIdx.y.
struct ConvBwdSmem {
  uint2 x[CT_WARPS][CT_RING * CT_U][32], g[CT_WARPS][CT_RING * CT_U][32];
};
template <int CW>
__global__ void __launch_bounds__(CT_WARPS * 32, 2) conv1d_bwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                                      const bf16* __restrict__ bias, const bf16* __restrict__ dy,
                                                                      bf16* __restrict__ dx, float* __restrict__ partial,
                                                                      int T, int C, long ldx, int act, int rows) {
  extern __shared__ __align__(16) uint8_t conv_smem[];
  ConvBwdSmem& sm = *reinterpret_cast<ConvBwdSmem*>(conv_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * CW + warp % CW) * CT_C + lane * 4;
  const int t0 = (blockIdx.y * (CT_WARPS / CW) + warp / CW) * rows;
  Quad dw[4], db = quad_zero();
#pragma unroll
  for (int j = 0; j < 4; ++j) dw[j] = quad_zero();
  if (c < C && t0 < T) {
    uint2 *rx = &sm.x[warp][0][lane], *rg = &sm.g[warp][0][lane];
    const bf16* xs = x + (static_cast<long>(blockIdx.z) * T + t0) * ldx + c;
    const bf16* gs = dy + (static_cast<long>(blockIdx.z) * T + t0) * C + c;
    bf16* dp = dx + (static_cast<long>(blockIdx.z) * T + t0) * C + c;
    const int n = min(rows, T - t0);             // rows of this segment
    const int ne = min(n + 3, T - t0);           // dpre is needed on [0, ne); rows past T count as zero
    ConvFeed fx(xs, ldx, ne, rx), fg(gs, C, ne, rg);
#pragma unroll
    for (int g = 0; g < CT_RING - 1; ++g) { fx.next(false); fg.next(); }
    auto before = [&](int k) {
      return quad_unpack(t0 >= k ? *reinterpret_cast<const uint2*>(xs - k * ldx) : make_uint2(0u, 0u));
    };
    Quad x0 = before(3), x1 = before(2), x2 = before(1);
    Quad wv[4], bv;
    conv_taps(w, bias, c, true, wv, bv);
    Quad d0 = quad_zero(), d1 = quad_zero(), d2 = quad_zero();
    dp -= 3L * C;
    // row u of group g: the gradients of its taps if it is counted here, dx three rows behind if that is in the segment
    auto row = [&](int u, int g, bool counted, bool behind) {
      const Quad x3 = quad_unpack(rx[((g % CT_RING) * CT_U + u) * 32]);
      Quad d3 = quad_unpack(rg[((g % CT_RING) * CT_U + u) * 32]);   // zero past T, and so is dpre
      if (act) {
        const Quad p = quad_fma(wv[3], x3, quad_fma(wv[2], x2, quad_fma(wv[1], x1, quad_fma(wv[0], x0, bv))));
        d3.a = mul2(d3.a, dsilu2(p.a));
        d3.b = mul2(d3.b, dsilu2(p.b));
      }
      if (counted) {
        dw[0] = quad_fma(d3, x0, dw[0]);
        dw[1] = quad_fma(d3, x1, dw[1]);
        dw[2] = quad_fma(d3, x2, dw[2]);
        dw[3] = quad_fma(d3, x3, dw[3]);
        db = quad_fma(d3, Quad{make_float2(1.f, 1.f), make_float2(1.f, 1.f)}, db);
      }
      if (behind)
        *reinterpret_cast<uint2*>(dp) =
            quad_pack(quad_fma(wv[3], d0, quad_fma(wv[2], d1, quad_fma(wv[1], d2, quad_fma(wv[0], d3, quad_zero())))));
      dp += C;
      x0 = x1; x1 = x2; x2 = x3;
      d0 = d1; d1 = d2; d2 = d3;
    };
    int g = 0;
    if (n >= CT_U) {                             // the first group has nothing three rows behind but in its last row
      fx.next(false); fg.next();
      cp_async_wait<CT_RING - 1>();
#pragma unroll
      for (int u = 0; u < CT_U; ++u) row(u, 0, true, u >= 3);
      g = 1;
    }
    for (; (g + 1) * CT_U <= n; ++g) {
      fx.next(false); fg.next();
      cp_async_wait<CT_RING - 1>();
#pragma unroll
      for (int u = 0; u < CT_U; ++u) row(u, g, true, true);
    }
    cp_async_wait<0>();
    for (int r = g * CT_U; r < n + 3; ++r) {     // at most six rows, all in flight already: three groups are
      const int at = r / CT_U;
      row(r - at * CT_U, at, r < n, r >= 3);
    }
  }
  __syncthreads();                               // the rings become the reduction buffer
  float(*sred)[5][CT_C] = reinterpret_cast<float(*)[5][CT_C]>(conv_smem);
#pragma unroll
  for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(&sred[warp][j][lane * 4]) = make_float4(dw[j].a.x, dw[j].a.y, dw[j].b.x, dw[j].b.y);
  *reinterpret_cast<float4*>(&sred[warp][4][lane * 4]) = make_float4(db.a.x, db.a.y, db.b.x, db.b.y);
  __syncthreads();
  float* pp = partial + (static_cast<long>(blockIdx.z) * gridDim.y + blockIdx.y) * 5 * C;
  for (int e = threadIdx.x; e < 5 * CW * CT_C; e += CT_WARPS * 32) {
    const int j = e / (CW * CT_C), cc = e - j * (CW * CT_C);
    const int cg = blockIdx.x * CW * CT_C + cc;
    if (cg >= C) continue;
    float acc = 0.f;
#pragma unroll
    for (int ti = 0; ti < CT_WARPS / CW; ++ti) acc += sred[ti * CW + cc / CT_C][j][cc % CT_C];
    pp[static_cast<long>(j) * C + cg] = acc;
  }
}

// partial [parts][5][C] -> dw (C, 4) and db (C), fp32 or bf16, in a fixed order.  CTA: 32 channels, G groups of parts: 8 warps for
// a few parts, 32 for more (64 parts of 4352 channels 10.3 -> 4.1 us: the loads of a thread follow one another).
template <typename OT, int G>
__global__ void __launch_bounds__(G * 32) conv1d_dw_kernel(const float* __restrict__ partial, int parts, int C,
                                                           OT* __restrict__ dw, OT* __restrict__ db) {
  __shared__ float s[G][5][32];
  const int cl = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.x * 32 + cl;
  float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < C) {
#pragma unroll 4
    for (int p = g; p < parts; p += G)
#pragma unroll
      for (int j = 0; j < 5; ++j) acc[j] += partial[(static_cast<long>(p) * 5 + j) * C + c];
  }
#pragma unroll
  for (int j = 0; j < 5; ++j) s[g][j][cl] = acc[j];
  __syncthreads();
  if (g >= 5 || c >= C) return;
  float v = 0.f;
#pragma unroll
  for (int k = 0; k < G; ++k) v += s[k][g][cl];
  if (g < 4) dw[static_cast<long>(c) * 4 + g] = static_cast<OT>(v);
  else if (db) db[c] = static_cast<OT>(v);
}

// ------------------------------------------------------------------------------------
// Embedding
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) embedding_fwd_kernel(const long* __restrict__ ids, const bf16* __restrict__ w,
                                                            bf16* __restrict__ y, long n, int d, long vocab,
                                                            KernelStatus* status) {
  const int d8 = d / 8;
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n * d8; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long tok = i / d8;
    const int v = static_cast<int>(i - tok * d8);
    long id = ids[tok];
    if (v == 0) NSA_CHECK_INDEX(id >= 0 && id < vocab, status, id);
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    *reinterpret_cast<uint4*>(y + tok * d + v * 8) = *reinterpret_cast<const uint4*>(w + id * d + v * 8);
  }
}
// ids sorted ascending with `perm` giving the original token position of each sorted entry.
// One CTA column per run start: sums the run's gradient rows in sorted order (deterministic).
__global__ void __launch_bounds__(256) embedding_bwd_kernel(const long* __restrict__ sorted_ids,
                                                            const long* __restrict__ perm, const bf16* __restrict__ dy,
                                                            float* __restrict__ dw, long n, int d) {
  const long i = blockIdx.x;
  const long id = sorted_ids[i];
  if (i > 0 && sorted_ids[i - 1] == id) return;   // not a run start
  for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    for (long j = i; j < n && sorted_ids[j] == id; ++j) {
      float v[8];
      load8(dy + perm[j] * d + c, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += v[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) dw[id * d + c + k] += acc[k];
  }
}

inline int grid_for(long n, int block, int per_sm = 8) {
  long g = (n + block - 1) / block;
  long cap = static_cast<long>(nsa::sm_count()) * per_sm;
  return static_cast<int>(g < cap ? (g < 1 ? 1 : g) : cap);
}

template <int MODE>
int launch_rms_fwd(const void* x, const void* g, const void* w, void* y, float* rstd, long rows, int d, float eps, cudaStream_t st,
                   long ldg = 0) {
  if (ldg == 0) ldg = d;
  if (ldg % 8 || (reinterpret_cast<uintptr_t>(g) & 15)) return nsa::fail(NSA_ERR_ALIGNMENT, "rmsnorm: gate rows must be 16-byte aligned");
  const bf16 *X = (const bf16*)x, *G = (const bf16*)g, *Wt = (const bf16*)w;
  bf16* Y = (bf16*)y;
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width must be a multiple of 8");
  if (d <= 256) rmsnorm_fwd_kernel<32, 1, MODE><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(X, G, Wt, Y, rstd, rows, d, eps, ldg);
  else if (d <= 512) rmsnorm_fwd_kernel<32, 2, MODE><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(X, G, Wt, Y, rstd, rows, d, eps, ldg);
  else if (d <= 2048) rmsnorm_fwd_kernel<256, 1, MODE><<<(unsigned)rows, 256, 0, st>>>(X, G, Wt, Y, rstd, rows, d, eps, ldg);
  else if (d <= 4096) rmsnorm_fwd_kernel<256, 2, MODE><<<(unsigned)rows, 256, 0, st>>>(X, G, Wt, Y, rstd, rows, d, eps, ldg);
  else if (d <= 8192) rmsnorm_fwd_kernel<256, 4, MODE><<<(unsigned)rows, 256, 0, st>>>(X, G, Wt, Y, rstd, rows, d, eps, ldg);
  else return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width above 8192 is not supported");
  nsa::count_launch();
  return 0;
}

// CTAs of the persistent backward: all resident at once (a partial second round would idle most SMs), at most `parts`.
template <int TPR, int NV, int MODE>
int bwd_grid(int parts) {
  static int per_sm = 0;
  if (per_sm == 0) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rmsnorm_bwd_kernel<TPR, NV, MODE>, rms_bwd_threads<TPR>, 0);
    per_sm = n > 0 ? n : 1;
  }
  const int all = per_sm * nsa::sm_count();
  return parts < all ? parts : all;
}
template <int TPR, int NV, int MODE>
void run_rms_bwd(const bf16* X, const bf16* G, const bf16* Wt, const bf16* DY, const float* rstd, bf16* DX, bf16* DG, float* partial,
                 int& grid, long rows, int d, const bf16* DR, long ldg, cudaStream_t st) {
  grid = bwd_grid<TPR, NV, MODE>(grid);
  rmsnorm_bwd_kernel<TPR, NV, MODE><<<grid, rms_bwd_threads<TPR>, 0, st>>>(X, G, Wt, DY, rstd, DX, DG, partial, rows, d, DR, ldg);
}
// `grid` holds the number of partial rows the caller has room for and receives the number written.
template <int MODE>
int launch_rms_bwd(const void* x, const void* g, const void* w, const void* dy, const float* rstd, void* dx, void* dg,
                   float* partial, int& grid, long rows, int d, cudaStream_t st, const void* dres = nullptr, long ldg = 0) {
  const bf16 *X = (const bf16*)x, *G = (const bf16*)g, *Wt = (const bf16*)w, *DY = (const bf16*)dy, *DR = (const bf16*)dres;
  bf16 *DX = (bf16*)dx, *DG = (bf16*)dg;
  if (d <= 256) run_rms_bwd<32, 1, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
  else if (d <= 512) run_rms_bwd<32, 2, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
  else if (d <= 2048) run_rms_bwd<256, 1, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
  else if (d <= 4096) run_rms_bwd<512, 1, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
  else if (d <= 8192) {
    if constexpr (MODE == 2) run_rms_bwd<512, 2, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
    else run_rms_bwd<256, 4, MODE>(X, G, Wt, DY, rstd, DX, DG, partial, grid, rows, d, DR, ldg, st);
  }
  else return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width above 8192 is not supported");
  nsa::count_launch();
  return 0;
}

int launch_rms_add_fwd(const void* x, const void* r, const void* w, void* h, void* y, float* rstd, long rows, int d, float eps,
                       cudaStream_t st) {
  const bf16 *X = (const bf16*)x, *R = (const bf16*)r, *Wt = (const bf16*)w;
  bf16 *H = (bf16*)h, *Y = (bf16*)y;
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width must be a multiple of 8");
  if (d <= 256) rmsnorm_add_fwd_kernel<32, 1><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(X, R, Wt, H, Y, rstd, rows, d, eps);
  else if (d <= 512) rmsnorm_add_fwd_kernel<32, 2><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(X, R, Wt, H, Y, rstd, rows, d, eps);
  else if (d <= 2048) rmsnorm_add_fwd_kernel<256, 1><<<(unsigned)rows, 256, 0, st>>>(X, R, Wt, H, Y, rstd, rows, d, eps);
  else if (d <= 4096) rmsnorm_add_fwd_kernel<256, 2><<<(unsigned)rows, 256, 0, st>>>(X, R, Wt, H, Y, rstd, rows, d, eps);
  else if (d <= 8192) rmsnorm_add_fwd_kernel<256, 4><<<(unsigned)rows, 256, 0, st>>>(X, R, Wt, H, Y, rstd, rows, d, eps);
  else return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width above 8192 is not supported");
  nsa::count_launch();
  return 0;
}

}  // namespace

// mode: 0 plain, 1 norm-then-gate, 2 gate-then-norm.  rstd (rows) fp32 is written for backward.
extern "C" int nsa_rmsnorm_fwd(const void* x, const void* gate, const void* w, void* y, float* rstd, long rows, int d,
                               float eps, int mode, cudaStream_t st) {
  if (mode == 0) return launch_rms_fwd<0>(x, gate, w, y, rstd, rows, d, eps, st);
  if (mode == 1) return launch_rms_fwd<1>(x, gate, w, y, rstd, rows, d, eps, st);
  return launch_rms_fwd<2>(x, gate, w, y, rstd, rows, d, eps, st);
}

// Number of per-CTA partial rows the backward needs in `partial` (fp32 [parts, d]).
extern "C" int nsa_rmsnorm_bwd_parts(long rows, int d) {
  const int rows_per_cta = d <= 512 ? 8 : 1;
  long want = (rows + rows_per_cta - 1) / rows_per_cta;
  long cap = static_cast<long>(nsa::sm_count()) * 4;
  return static_cast<int>(want < cap ? want : cap);
}

// dw_bf16 / dw_f32: either may be null.  `partial` is caller-provided scratch of
// nsa_rmsnorm_bwd_parts(rows, d) * d floats.
extern "C" int nsa_rmsnorm_bwd(const void* x, const void* gate, const void* w, const void* dy, const float* rstd,
                               void* dx, void* dgate, void* dw_bf16, float* dw_f32, float* partial, long rows, int d,
                               int mode, cudaStream_t st) {
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width must be a multiple of 8");
  int parts = nsa_rmsnorm_bwd_parts(rows, d);
  int rc;
  if (mode == 0) rc = launch_rms_bwd<0>(x, gate, w, dy, rstd, dx, dgate, partial, parts, rows, d, st);
  else if (mode == 1) rc = launch_rms_bwd<1>(x, gate, w, dy, rstd, dx, dgate, partial, parts, rows, d, st);
  else rc = launch_rms_bwd<2>(x, gate, w, dy, rstd, dx, dgate, partial, parts, rows, d, st);
  if (rc) return rc;
  reduce_partials_kernel<<<(d + 31) / 32, 1024, 0, st>>>(partial, parts, d, (bf16*)dw_bf16, dw_f32);
  nsa::count_launch();
  return 0;
}

// Gated modes with the gate given as a column slice of a wider row-major matrix: `ldg` is the
// gate's row pitch in elements (a multiple of 8; the slice must start 16-byte aligned).  x, y, dx
// and dgate stay contiguous [rows, d].
extern "C" int nsa_rmsnorm_fwd_ldg(const void* x, const void* gate, long ldg, const void* w, void* y, float* rstd, long rows,
                                   int d, float eps, int mode, cudaStream_t st) {
  if (mode == 1) return launch_rms_fwd<1>(x, gate, w, y, rstd, rows, d, eps, st, ldg);
  if (mode == 2) return launch_rms_fwd<2>(x, gate, w, y, rstd, rows, d, eps, st, ldg);
  return nsa::fail(NSA_ERR_SHAPE, "nsa_rmsnorm_fwd_ldg: gated modes only");
}
extern "C" int nsa_rmsnorm_bwd_ldg(const void* x, const void* gate, long ldg, const void* w, const void* dy, const float* rstd,
                                   void* dx, void* dgate, void* dw_bf16, float* dw_f32, float* partial, long rows, int d,
                                   int mode, cudaStream_t st) {
  if (d % 8 || ldg % 8 || (reinterpret_cast<uintptr_t>(gate) & 15))
    return nsa::fail(NSA_ERR_ALIGNMENT, "rmsnorm: widths multiples of 8 and 16-byte aligned gate rows required");
  int parts = nsa_rmsnorm_bwd_parts(rows, d);
  int rc;
  if (mode == 1) rc = launch_rms_bwd<1>(x, gate, w, dy, rstd, dx, dgate, partial, parts, rows, d, st, nullptr, ldg);
  else if (mode == 2) rc = launch_rms_bwd<2>(x, gate, w, dy, rstd, dx, dgate, partial, parts, rows, d, st, nullptr, ldg);
  else return nsa::fail(NSA_ERR_SHAPE, "nsa_rmsnorm_bwd_ldg: gated modes only");
  if (rc) return rc;
  reduce_partials_kernel<<<(d + 31) / 32, 1024, 0, st>>>(partial, parts, d, (bf16*)dw_bf16, dw_f32);
  nsa::count_launch();
  return 0;
}

// h = x + r and y = rmsnorm(h) * w in one pass (plain mode).  x, r, h, y: [rows, d] bf16 contiguous.
extern "C" int nsa_rmsnorm_add_fwd(const void* x, const void* r, const void* w, void* h, void* y, float* rstd, long rows,
                                   int d, float eps, cudaStream_t st) {
  return launch_rms_add_fwd(x, r, w, h, y, rstd, rows, d, eps, st);
}

// Plain-mode backward that also adds `dres` (the gradient arriving at the norm's input through the
// residual stream, [rows, d] bf16) into dx.  `partial` as for nsa_rmsnorm_bwd.
extern "C" int nsa_rmsnorm_bwd_res(const void* x, const void* w, const void* dy, const float* rstd, const void* dres,
                                   void* dx, void* dw_bf16, float* dw_f32, float* partial, long rows, int d,
                                   cudaStream_t st) {
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "rmsnorm: width must be a multiple of 8");
  int parts = nsa_rmsnorm_bwd_parts(rows, d);
  const int rc = launch_rms_bwd<0>(x, nullptr, w, dy, rstd, dx, nullptr, partial, parts, rows, d, st, dres);
  if (rc) return rc;
  reduce_partials_kernel<<<(d + 31) / 32, 1024, 0, st>>>(partial, parts, d, (bf16*)dw_bf16, dw_f32);
  nsa::count_launch();
  return 0;
}

// ------------------------------------------------------------------------------------
// RMSNorm backward for callers that must not allocate.
//
// Some hosts of this library cannot call cudaMalloc (or anything that may call it) at the
// point where they need a backward pass: an embedding runtime whose device-memory budget is
// fixed when the library is loaded, a worker thread that is forbidden to take the allocator
// lock, a latency-critical loop that cannot afford the implicit device synchronisation an
// allocation may cause.  nsa_rmsnorm_bwd needs a scratch buffer for the per-CTA partial
// sums of the weight gradient; this variant keeps that scratch in the library itself.
//
// The scratch is one file-scope device array of NSA_NOALLOC_SCRATCH_FLOATS floats
// (592 * 4096 floats = 9.25 MiB).  Every GPU that loads the library holds that much from load
// until process exit, whether or not this entry point is ever called.
// ------------------------------------------------------------------------------------
#define NSA_NOALLOC_SCRATCH_FLOATS (592 * 4096)
static __device__ __align__(256) float g_noalloc_scratch[NSA_NOALLOC_SCRATCH_FLOATS];

// Device address of g_noalloc_scratch per device.  In host code the array's name is only a
// handle for the runtime, not an address a kernel can use, so the address is looked up once
// per device with that device current.  The cache is filled without a lock: host threads that
// race on a device's first call all store the same value.
static float* g_noalloc_scratch_addr[64] = {nullptr};

static int noalloc_scratch_for_current_device(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return nsa::fail_cuda(e, "nsa_rmsnorm_bwd_noalloc: cudaGetDevice");
  if (dev < 0 || dev >= 64) return nsa::fail(NSA_ERR_LIMIT, "nsa_rmsnorm_bwd_noalloc: device index above 63");
  if (g_noalloc_scratch_addr[dev] == nullptr) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_scratch);
    if (e != cudaSuccess) return nsa::fail_cuda(e, "nsa_rmsnorm_bwd_noalloc: cudaGetSymbolAddress");
    g_noalloc_scratch_addr[dev] = ptr;
  }
  *out = g_noalloc_scratch_addr[dev];
  return 0;
}

// Same arguments and results as nsa_rmsnorm_bwd, minus `partial`.
//  * Calls no cudaMalloc / cudaFree and no allocating library routine.
//  * The first call on each device looks up the scratch address (a synchronous runtime
//    query); make that first call before any stream capture begins on that device.
//  * Limit: nsa_rmsnorm_bwd_parts(rows, d) * d must not exceed NSA_NOALLOC_SCRATCH_FLOATS
//    (true whenever sm_count * 4 * d <= 592 * 4096, e.g. d <= 4096 on a 148-SM part); larger
//    problems are rejected with NSA_ERR_LIMIT and
//    nothing is launched.
//  * All calls on a device share the one scratch array, which keeps whatever the previous
//    call left in it.  Nothing in it has to start at zero: the backward kernel overwrites
//    every (part, column) entry that the reduction then reads.  Two calls whose kernels can
//    overlap on the GPU (different streams, or concurrent host threads) race on the array;
//    serialise them on one stream.
extern "C" int nsa_rmsnorm_bwd_noalloc(const void* x, const void* gate, const void* w, const void* dy,
                                       const float* rstd, void* dx, void* dgate, void* dw_bf16, float* dw_f32,
                                       long rows, int d, int mode, cudaStream_t st) {
  if (rows <= 0 || d <= 0) return nsa::fail(NSA_ERR_SHAPE, "nsa_rmsnorm_bwd_noalloc: empty problem");
  const long need = static_cast<long>(nsa_rmsnorm_bwd_parts(rows, d)) * d;
  if (need > static_cast<long>(NSA_NOALLOC_SCRATCH_FLOATS))
    return nsa::fail(NSA_ERR_LIMIT,
                     "nsa_rmsnorm_bwd_noalloc: problem needs more than the 592*4096-float built-in scratch "
                     "(use nsa_rmsnorm_bwd with caller-provided scratch)");
  float* scratch = nullptr;
  const int rc = noalloc_scratch_for_current_device(&scratch);
  if (rc) return rc;
  return nsa_rmsnorm_bwd(x, gate, w, dy, rstd, dx, dgate, dw_bf16, dw_f32, scratch, rows, d, mode, st);
}

extern "C" int nsa_l2norm_fwd(const void* x, void* y, float* rinv, long rows, int d, float eps, cudaStream_t st) {
  if (d % 8 || d > 512) return nsa::fail(NSA_ERR_SHAPE, "l2norm: width must be a multiple of 8, at most 512");
  const unsigned grid = (unsigned)((rows + 7) / 8);
  if (d <= 256) l2norm_fwd_kernel<1><<<grid, 256, 0, st>>>((const bf16*)x, (bf16*)y, rinv, rows, d, eps);
  else l2norm_fwd_kernel<2><<<grid, 256, 0, st>>>((const bf16*)x, (bf16*)y, rinv, rows, d, eps);
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_l2norm_bwd(const void* y, const void* dy, const float* rinv, void* dx, long rows, int d, cudaStream_t st) {
  if (d % 8 || d > 512) return nsa::fail(NSA_ERR_SHAPE, "l2norm: width must be a multiple of 8, at most 512");
  const unsigned grid = (unsigned)((rows + 7) / 8);
  if (d <= 256) l2norm_bwd_kernel<1><<<grid, 256, 0, st>>>((const bf16*)y, (const bf16*)dy, rinv, (bf16*)dx, rows, d);
  else l2norm_bwd_kernel<2><<<grid, 256, 0, st>>>((const bf16*)y, (const bf16*)dy, rinv, (bf16*)dx, rows, d);
  nsa::count_launch();
  return 0;
}

// gate / up: [rows, cols] with row pitches ldg / ldu (elements, multiples of 8); y contiguous.
extern "C" int nsa_swiglu_fwd(const void* g, const void* u, void* y, long rows, int cols, long ldg, long ldu, cudaStream_t st) {
  if ((cols % 8) || (ldg % 8) || (ldu % 8)) return nsa::fail(NSA_ERR_SHAPE, "swiglu: sizes must be multiples of 8");
  const long n8 = rows * (cols / 8);
  swiglu_fwd_kernel<<<grid_for(n8, 256), 256, 0, st>>>((const bf16*)g, (const bf16*)u, (bf16*)y, n8, cols / 8, ldg / 8, ldu / 8);
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_swiglu_bwd(const void* g, const void* u, const void* dy, void* dg, void* du, long rows, int cols,
                              long ldg, long ldu, long ldo, cudaStream_t st) {
  if ((cols % 8) || (ldg % 8) || (ldu % 8) || (ldo % 8)) return nsa::fail(NSA_ERR_SHAPE, "swiglu: sizes must be multiples of 8");
  const long n8 = rows * (cols / 8);
  swiglu_bwd_kernel<<<grid_for(n8, 256), 256, 0, st>>>((const bf16*)g, (const bf16*)u, (const bf16*)dy, (bf16*)dg, (bf16*)du,
                                                        n8, cols / 8, ldg / 8, ldu / 8, ldo / 8);
  nsa::count_launch();
  return 0;
}

// o, o1..o3: [rows, D] bf16 contiguous; g1..g3: [rows] bf16.  D in {64, 128, 256}.
extern "C" int nsa_gate_combine_fwd(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2,
                                    const void* g3, void* o, long rows, int D, cudaStream_t st) {
  if (D != 64 && D != 128 && D != 256) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: head_dim must be 64, 128 or 256");
  const long n8 = rows * (D / 8);
  const int grid = grid_for(n8, 256);
#define NSA_GC_FWD(L) gate_combine_fwd_kernel<L><<<grid, 256, 0, st>>>((const bf16*)o1, (const bf16*)o2, (const bf16*)o3, \
    (const bf16*)g1, (const bf16*)g2, (const bf16*)g3, (bf16*)o, n8, 1, 1L, 0)
  if (D == 64) NSA_GC_FWD(8); else if (D == 128) NSA_GC_FWD(16); else NSA_GC_FWD(32);
#undef NSA_GC_FWD
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_gate_combine_bwd(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2,
                                    const void* g3, const void* d_o, void* do1, void* do2, void* do3, void* dg1,
                                    void* dg2, void* dg3, long rows, int D, cudaStream_t st) {
  if (D != 64 && D != 128 && D != 256) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: head_dim must be 64, 128 or 256");
  const long n8 = rows * (D / 8);
  const long blocks = (n8 + 255) / 256;
  if (blocks > 2147483647L) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: problem too large for one launch");
#define NSA_GC_BWD(L) gate_combine_bwd_kernel<L, false><<<(unsigned)blocks, 256, 0, st>>>((const bf16*)o1, (const bf16*)o2, \
    (const bf16*)o3, (const bf16*)g1, (const bf16*)g2, (const bf16*)g3, (const bf16*)d_o, (bf16*)do1, (bf16*)do2, (bf16*)do3, \
    (bf16*)dg1, (bf16*)dg2, (bf16*)dg3, nullptr, nullptr, nullptr, n8, 1, 1L, 0)
  if (D == 64) NSA_GC_BWD(8); else if (D == 128) NSA_GC_BWD(16); else NSA_GC_BWD(32);
#undef NSA_GC_BWD
  nsa::count_launch();
  return 0;
}

// The same with the three gates as columns of one [tokens, >= 3*Hq] bf16 matrix (row pitch ldg, the
// gate projection's output as it stands) and, with sig != 0, given as logits: the sigmoid and its
// derivative are applied here.  rows = tokens * Hq.  dg1..dg3 use the same pitch.  e1..e3 (all or none): fp32 [rows].
extern "C" int nsa_gate_combine_fwd_ex(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2,
                                       const void* g3, long ldg, int Hq, int sig, void* o, long rows, int D, cudaStream_t st) {
  if (D != 64 && D != 128 && D != 256) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: head_dim must be 64, 128 or 256");
  if (Hq <= 0 || rows % Hq) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: rows must be tokens * heads");
  const long n8 = rows * (D / 8);
  const int grid = grid_for(n8, 256);
#define NSA_GC_FWD(L) gate_combine_fwd_kernel<L><<<grid, 256, 0, st>>>((const bf16*)o1, (const bf16*)o2, (const bf16*)o3, \
    (const bf16*)g1, (const bf16*)g2, (const bf16*)g3, (bf16*)o, n8, Hq, ldg, sig)
  if (D == 64) NSA_GC_FWD(8); else if (D == 128) NSA_GC_FWD(16); else NSA_GC_FWD(32);
#undef NSA_GC_FWD
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_gate_combine_bwd_ex(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2,
                                       const void* g3, long ldg, int Hq, int sig, const void* d_o, void* do1, void* do2,
                                       void* do3, void* dg1, void* dg2, void* dg3, float* e1, float* e2, float* e3,
                                       long rows, int D, cudaStream_t st) {
  if (D != 64 && D != 128 && D != 256) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: head_dim must be 64, 128 or 256");
  if (Hq <= 0 || rows % Hq) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: rows must be tokens * heads");
  const long n8 = rows * (D / 8);
  const long blocks = (n8 + 255) / 256;
  if (blocks > 2147483647L) return nsa::fail(NSA_ERR_SHAPE, "gate_combine: problem too large for one launch");
#define NSA_GC_BWD(L, S) gate_combine_bwd_kernel<L, S><<<(unsigned)blocks, 256, 0, st>>>((const bf16*)o1, (const bf16*)o2, \
    (const bf16*)o3, (const bf16*)g1, (const bf16*)g2, (const bf16*)g3, (const bf16*)d_o, (bf16*)do1, (bf16*)do2, (bf16*)do3, \
    (bf16*)dg1, (bf16*)dg2, (bf16*)dg3, e1, e2, e3, n8, Hq, ldg, sig)
  if (e1 != nullptr) { if (D == 64) NSA_GC_BWD(8, true); else if (D == 128) NSA_GC_BWD(16, true); else NSA_GC_BWD(32, true); }
  else { if (D == 64) NSA_GC_BWD(8, false); else if (D == 128) NSA_GC_BWD(16, false); else NSA_GC_BWD(32, false); }
#undef NSA_GC_BWD
  nsa::count_launch();
  return 0;
}

// Block mean pooling (see nsa_pool_fwd_kernel).  x: [B, T, width] bf16 with row pitch ldx; y: [B, nC, width]
// contiguous, nC = (T - block) / stride + 1.  dx is contiguous [B, T, width].
extern "C" int nsa_pool_fwd(const void* x, void* y, int B, int T, int width, long ldx, int block, int stride, cudaStream_t st) {
  if (width % 8 || ldx % 8 || T < block || block <= 0 || stride <= 0)
    return nsa::fail(NSA_ERR_SHAPE, "nsa_pool: width and pitch multiples of 8, T >= block required");
  const int nC = (T - block) / stride + 1;
  const long n = static_cast<long>(B) * nC * (width / 8);
  nsa_pool_fwd_kernel<<<grid_for(n, 256), 256, 0, st>>>((const bf16*)x, (bf16*)y, T, nC, width / 8, ldx, block, stride, n);
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_pool_bwd(const void* dy, void* dx, int B, int T, int width, int block, int stride, cudaStream_t st) {
  if (width % 8 || T < block || block <= 0 || stride <= 0)
    return nsa::fail(NSA_ERR_SHAPE, "nsa_pool: width multiple of 8, T >= block required");
  const int nC = (T - block) / stride + 1;
  const long n = static_cast<long>(B) * T * (width / 8);
  nsa_pool_bwd_kernel<<<grid_for(n, 256), 256, 0, st>>>((const bf16*)dy, (bf16*)dx, T, nC, width / 8, block, stride, n);
  nsa::count_launch();
  return 0;
}

extern "C" int nsa_rope(const void* x, const float* cos_t, const float* sin_t, void* y, long batch, int T, int H, int D,
                        int backward, cudaStream_t st) {
  if (D % 16) return nsa::fail(NSA_ERR_SHAPE, "rope: head_dim must be a multiple of 16");
  const long n = batch * T * H * (D / 16);
  rope_kernel<<<grid_for(n, 256), 256, 0, st>>>((const bf16*)x, cos_t, sin_t, (bf16*)y, n, T, H, D, backward ? -1.f : 1.f);
  nsa::count_launch();
  return 0;
}

// Channel tiles of a CTA.
static int conv_tiles(int C) { return C <= CT_C ? 1 : 2; }
// Time steps per warp: 64 keeps the rows read twice (3 of x ahead of a segment, 3 of dpre behind it) under
// a tenth; short sequences take 32, 16 or 8 so that every SM still finds 32 warps; beyond 16.8 M steps (of four segments
// a CTA, eight up to 128 channels) 128 or 256, so that the grid's second dimension (at most 65535) reaches as far as 67 M.
static int conv_rows(int B, int T, int C) {
  int rows = 64;
  while (rows < 256 && static_cast<long>(rows) * (CT_WARPS / conv_tiles(C)) * 65535 < T) rows <<= 1;
  auto warps = [&](int r) { return static_cast<long>(B) * ((C + CT_C - 1) / CT_C) * ((T + r - 1) / r); };
  while (rows > 8 && warps(rows) < 32L * nsa::sm_count()) rows >>= 1;
  return rows;
}
static dim3 conv_grid(int B, int T, int C, int rows) {
  const int cw = conv_tiles(C), steps = CT_WARPS / cw * rows;
  return dim3((C + cw * CT_C - 1) / (cw * CT_C), static_cast<unsigned>((static_cast<long>(T) + steps - 1) / steps), B);
}
extern "C" int nsa_conv1d_fwd(const void* x, const void* w, const void* bias, void* y, int B, int T, int C, long ldx,
                              int width, int act, cudaStream_t st) {
  if (C % 8 || ldx % 8 || width != 4) return nsa::fail(NSA_ERR_SHAPE, "conv1d: channels multiple of 8 and width 4 required");
  const int rows = conv_rows(B, T, C);
  const dim3 grid = conv_grid(B, T, C, rows);
#define NSA_CONV_FWD(CW) \
  conv1d_fwd_kernel<CW><<<grid, CT_WARPS * 32, 0, st>>>((const bf16*)x, (const bf16*)w, (const bf16*)bias, (bf16*)y, T, C, ldx, act, rows)
  const int cw = conv_tiles(C);
  if (cw == 1) NSA_CONV_FWD(1); else NSA_CONV_FWD(2);
#undef NSA_CONV_FWD
  nsa::count_launch();
  return 0;
}
extern "C" long nsa_conv1d_bwd_parts(int B, int T, int C) {
  return static_cast<long>(B) * conv_grid(B, T, C, conv_rows(B, T, C)).y;
}
// partial: scratch of nsa_conv1d_bwd_parts(B, T, C) * 5 * C floats.  dw: [C][4]; db: [C] or null; both fp32
// (dw_fp32 = 1) or bf16.
extern "C" int nsa_conv1d_bwd(const void* x, const void* w, const void* bias, const void* dy, void* dx, float* partial,
                              void* dw, void* db, int dw_fp32, int B, int T, int C, long ldx, int width, int act, cudaStream_t st) {
  if (C % 8 || ldx % 8 || width != 4) return nsa::fail(NSA_ERR_SHAPE, "conv1d: channels multiple of 8 and width 4 required");
  const int rows = conv_rows(B, T, C);
  const dim3 grid = conv_grid(B, T, C, rows);
  static_assert(sizeof(ConvBwdSmem) >= CT_WARPS * 5 * CT_C * 4, "conv1d: reduction buffer");
  const int cw = conv_tiles(C);
  auto* kernel = cw == 1 ? conv1d_bwd_kernel<1> : conv1d_bwd_kernel<2>;
  static bool cfg[2] = {};
  if (!cfg[cw - 1]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(ConvBwdSmem));
    if (e != cudaSuccess) return nsa::fail_cuda(e, "conv1d_bwd: shared memory attribute");
    cfg[cw - 1] = true;
  }
  kernel<<<grid, CT_WARPS * 32, sizeof(ConvBwdSmem), st>>>((const bf16*)x, (const bf16*)w, (const bf16*)bias, (const bf16*)dy, (bf16*)dx,
                                                    partial, T, C, ldx, act, rows);
  const int parts = static_cast<int>(nsa_conv1d_bwd_parts(B, T, C));
#define NSA_CONV_DW(OT, G) conv1d_dw_kernel<OT, G><<<(C + 31) / 32, G * 32, 0, st>>>(partial, parts, C, (OT*)dw, (OT*)db)
  if (parts <= 32) { if (dw_fp32) NSA_CONV_DW(float, 8); else NSA_CONV_DW(bf16, 8); }
  else { if (dw_fp32) NSA_CONV_DW(float, 32); else NSA_CONV_DW(bf16, 32); }
#undef NSA_CONV_DW
  nsa::count_launch(2);
  return 0;
}

extern "C" int nsa_embedding_fwd(const long* ids, const void* w, void* y, long n, int d, long vocab, cudaStream_t st) {
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "embedding: width must be a multiple of 8");
  embedding_fwd_kernel<<<grid_for(n * (d / 8), 256), 256, 0, st>>>(ids, (const bf16*)w, (bf16*)y, n, d, vocab, nsa::status_ptr());
  nsa::count_launch();
  return 0;
}
// dw (fp32 [vocab, d]) must be zero-initialised by the caller; rows of absent ids stay zero.
extern "C" int nsa_embedding_bwd(const long* sorted_ids, const long* perm, const void* dy, float* dw, long n, int d, cudaStream_t st) {
  if (d % 8) return nsa::fail(NSA_ERR_SHAPE, "embedding: width must be a multiple of 8");
  embedding_bwd_kernel<<<(unsigned)n, 256, 0, st>>>(sorted_ids, perm, (const bf16*)dy, dw, n, d);
  nsa::count_launch();
  return 0;
}
