// Optimizer and loss kernels.
//   * fused AdamW (decoupled weight decay, bias correction, optional fp32 master copy);
//   * 8-bit AdamW: moments stored as uint8 codes of a 256-entry dynamic-tree code book with
//     one fp32 absmax per 256-element block (signed map for the first moment, unsigned for
//     the second); one warp per block: dequantise, update, block absmax, requantise;
//   both over lists of tensors in one launch;
//   * sum of squares for the global gradient norm (deterministic two-stage reduction);
//   * softmax cross-entropy over a (rows, vocab) bf16 logits block: per-row loss and the
//     logits overwritten in place by d(loss)/d(logits).
// Gradients may be bf16 or fp32; an optional device scalar `grad_scale` multiplies them
// (clip coefficient), so no host synchronisation is needed between norm and update.
#include <algorithm>

#include "codebook.cuh"
#include "host.cuh"
#include <cuda_bf16.h>

namespace {
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct AdamArgs {
  float lr, beta1, beta2, eps, wd, bc1, bc2_sqrt;   // bc1 = 1-beta1^t, bc2_sqrt = sqrt(1-beta2^t)
};

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
  const float2 c = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
  v[0] = a.x; v[1] = a.y; v[2] = c.x; v[3] = c.y;
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(bf16* p, const float (&v)[4]) {
  uint2 x;
  *reinterpret_cast<__nv_bfloat162*>(&x.x) = __floats2bfloat162_rn(v[0], v[1]);
  *reinterpret_cast<__nv_bfloat162*>(&x.y) = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = x;
}

// ------------------------------------------------------------------------------------
// AdamW updates over a list of tensors.  A model has hundreds of parameters and most of them (norms,
// per-head vectors, convolution taps) are too small to fill the GPU for the time a launch takes, so one
// launch updates up to kMaxItems of them: the work is numbered through all tensors, and a CTA that
// walks it moves on in the list (uniform constant-memory reads) whenever its number passes an end.
// ------------------------------------------------------------------------------------
constexpr int kMaxItems = 48;         // 48 x 64 bytes of kernel arguments
struct AdamItem {
  void* p;
  const void* g;
  void* m;             // fp32, or uint8 codes
  void* v;
  float* a;            // fp32 master copy or null; 8-bit: scales of the first moment
  float* b;            // 8-bit: scales of the second moment
  long n;              // elements
  long end;            // units (chunks, blocks) up to and including this tensor; -end - 1 for tensors whose
};                     //   addresses do not allow 16-byte accesses (fp32 state only)
struct AdamList {
  AdamItem item[kMaxItems];
  int count;
};

// fp32 state: bound by memory (12 to 28 bytes per element).  A unit is 1024 elements, four consecutive ones
// per thread with 8- or 16-byte accesses.
template <typename PT, typename GT>
__global__ void __launch_bounds__(256) adamw_kernel(const __grid_constant__ AdamList list, const float* __restrict__ grad_scale,
                                                    long units, AdamArgs a) {
  const float gs = grad_scale ? *grad_scale : 1.f;
  const float decay = 1.f - a.lr * a.wd, step_size = a.lr / a.bc1;
  int k = 0;
  long first = 0;                     // first unit of item k
  for (long u = blockIdx.x; u < units; u += gridDim.x) {
    long end = list.item[k].end;
    while (u >= (end < 0 ? -end - 1 : end)) {
      first = end < 0 ? -end - 1 : end;
      end = list.item[++k].end;
    }
    const AdamItem& it = list.item[k];
    PT* p = static_cast<PT*>(it.p);
    const GT* g = static_cast<const GT*>(it.g);
    float *m = static_cast<float*>(it.m), *v = static_cast<float*>(it.v), *master = it.a;
    const long i = (u - first) * 1024 + threadIdx.x * 4;
    auto update = [&](float& w, float gr, float& mm, float& vv) {
      gr *= gs;
      w *= decay;
      mm = a.beta1 * mm + (1.f - a.beta1) * gr;
      vv = a.beta2 * vv + (1.f - a.beta2) * gr * gr;
      w -= step_size * mm / (sqrtf(vv) / a.bc2_sqrt + a.eps);
    };
    if (end > 0 && i + 4 <= it.n) {
      float w[4], gr[4], mm[4], vv[4];
      load4(g + i, gr);
      load4(m + i, mm);
      load4(v + i, vv);
      if (master) load4(master + i, w);
      else load4(p + i, w);
#pragma unroll
      for (int j = 0; j < 4; ++j) update(w[j], gr[j], mm[j], vv[j]);
      store4(m + i, mm);
      store4(v + i, vv);
      if (master) store4(master + i, w);
      store4(p + i, w);
    } else {
      // Scalar accesses.  The last elements of an aligned tensor: the thread's own four; an unaligned tensor: neighbouring
      // threads take neighbouring elements (2^26 bf16 parameters one element off: 315 us, 473 with a thread's own four one by one, 311 in a
      // kernel of scalar accesses alone).
      const long e0 = end > 0 ? i : (u - first) * 1024 + threadIdx.x, step = end > 0 ? 1 : 256;
      float w[4], gr[4], mm[4], vv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long e = min(e0 + j * step, it.n - 1);             // no branch between the loads: all four are in flight
        gr[j] = static_cast<float>(g[e]);
        mm[j] = m[e];
        vv[j] = v[e];
        w[j] = master ? master[e] : static_cast<float>(p[e]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long e = e0 + j * step;
        if (e >= it.n) break;
        update(w[j], gr[j], mm[j], vv[j]);
        m[e] = mm[j];
        v[e] = vv[j];
        if (master) master[e] = w[j];
        p[e] = static_cast<PT>(w[j]);
      }
    }
  }
}

// 8-bit state.  A warp owns a 256-element quantisation block (two groups of four consecutive elements per
// lane), so the block's absolute maximum is a warp reduction and the CTA never synchronises; decoding
// is one shared-memory read per value and encoding two (codebook.cuh).
template <typename PT, typename GT>
__global__ void __launch_bounds__(256, 4) adamw8bit_kernel(const __grid_constant__ AdamList list,
                                                           const float* __restrict__ cb_signed,
                                                           const float* __restrict__ cb_unsigned,
                                                           const float* __restrict__ grad_scale, long nblocks, AdamArgs a) {
  __shared__ cbk::Book<true> cs;
  __shared__ cbk::Book<false> cu;
  cs.build(cb_signed);
  cu.build(cb_unsigned);
  const float gs = grad_scale ? *grad_scale : 1.f;
  const int lane = threadIdx.x & 31;
  const float decay = 1.f - a.lr * a.wd, step_size = a.lr / a.bc1;
  int k = 0;
  long first = 0;                     // first block of item k
  for (long u = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5); u < nblocks; u += static_cast<long>(gridDim.x) * 8) {
    while (u >= list.item[k].end) first = list.item[k++].end;
    const AdamItem& it = list.item[k];
    PT* p = static_cast<PT*>(it.p);
    const GT* g = static_cast<const GT*>(it.g);
    uint8_t *mq = static_cast<uint8_t*>(it.m), *vq = static_cast<uint8_t*>(it.v);
    const long b = u - first, i = b * 256 + lane * 4;
    float gr[2][4], wt[2][4], mm[2][4], vv[2][4];
    uchar4 mc[2], vc[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      load4(g + i + h * 128, gr[h]);
      load4(p + i + h * 128, wt[h]);
      mc[h] = *reinterpret_cast<const uchar4*>(mq + i + h * 128);
      vc[h] = *reinterpret_cast<const uchar4*>(vq + i + h * 128);
    }
    const float ms = it.a[b], vs = it.b[b];
    float am = 0.f, av = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float m0[4] = {cs.value[mc[h].x], cs.value[mc[h].y], cs.value[mc[h].z], cs.value[mc[h].w]};
      const float v0[4] = {cu.value[vc[h].x], cu.value[vc[h].y], cu.value[vc[h].z], cu.value[vc[h].w]};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = gr[h][e] * gs;
        mm[h][e] = a.beta1 * (m0[e] * ms) + (1.f - a.beta1) * x;
        vv[h][e] = a.beta2 * (v0[e] * vs) + (1.f - a.beta2) * x * x;
        wt[h][e] = wt[h][e] * decay - step_size * mm[h][e] / (sqrtf(vv[h][e]) / a.bc2_sqrt + a.eps);
        am = fmaxf(am, fabsf(mm[h][e]));
        av = fmaxf(av, vv[h][e]);
      }
      store4(p + i + h * 128, wt[h]);
    }
    am = warp_max(am);
    av = warp_max(av);
    const float dm = fmaxf(am, 1e-30f), dv = fmaxf(av, 1e-30f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mc[h] = make_uchar4(cs.nearest(mm[h][0] / dm), cs.nearest(mm[h][1] / dm), cs.nearest(mm[h][2] / dm), cs.nearest(mm[h][3] / dm));
      vc[h] = make_uchar4(cu.nearest(vv[h][0] / dv), cu.nearest(vv[h][1] / dv), cu.nearest(vv[h][2] / dv), cu.nearest(vv[h][3] / dv));
      *reinterpret_cast<uchar4*>(mq + i + h * 128) = mc[h];
      *reinterpret_cast<uchar4*>(vq + i + h * 128) = vc[h];
    }
    if (lane == 0) { it.a[b] = am; it.b[b] = av; }
  }
}

template <typename GT>
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const GT* __restrict__ g, long n, float* __restrict__ partial) {
  __shared__ float red[8];
  float s = 0.f;
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float x = static_cast<float>(g[i]);
    s += x * x;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += red[k];
    partial[blockIdx.x] = t;
  }
}
__global__ void sumsq_final_kernel(const float* __restrict__ partial, int parts, float* __restrict__ out, int accumulate) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    float t = accumulate ? *out : 0.f;
    for (int k = 0; k < parts; ++k) t += partial[k];
    *out = t;
  }
}

// One CTA per row.  loss_out[row] = lse - logit[label] (0 for ignored rows); the row is then
// overwritten with (softmax - onehot) * (*inv_count) (zeros for ignored rows).
__global__ void __launch_bounds__(256) cross_entropy_kernel(bf16* __restrict__ logits, const long* __restrict__ labels,
                                                            float* __restrict__ loss_out, const float* __restrict__ inv_count,
                                                            int V, long ld, long ignore_index, int write_grad,
                                                            KernelStatus* status) {
  __shared__ float red[8], red2[8];
  const long row = blockIdx.x;
  bf16* lp = logits + row * ld;
  const long label = labels[row];
  const bool ignored = (label == ignore_index) || label < 0 || label >= V;
  if (threadIdx.x == 0) NSA_CHECK_INDEX(label == ignore_index || (label >= 0 && label < V), status, label);
  const int V8 = V / 8;
  // pass 1: online max / sum-exp
  float mx = -INFINITY, sum = 0.f;
  for (int i = threadIdx.x; i < V8; i += blockDim.x) {
    uint4 u = *reinterpret_cast<const uint4*>(lp + i * 8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    float x[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) { float2 f = __bfloat1622float2(h[k]); x[2 * k] = f.x; x[2 * k + 1] = f.y; }
    float lm = x[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) lm = fmaxf(lm, x[k]);
    const float nm = fmaxf(mx, lm);
    float ls = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ls += __expf(x[k] - nm);
    sum = sum * __expf(mx - nm) + ls;
    mx = nm;
  }
  for (int i = V8 * 8 + threadIdx.x; i < V; i += blockDim.x) {
    const float x = __bfloat162float(lp[i]);
    const float nm = fmaxf(mx, x);
    sum = sum * __expf(mx - nm) + __expf(x - nm);
    mx = nm;
  }
  // combine across the CTA
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  float gm = warp_max(mx);
  if (l == 0) red[w] = gm;
  __syncthreads();
  gm = red[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) gm = fmaxf(gm, red[k]);
  float s = (mx == -INFINITY) ? 0.f : sum * __expf(mx - gm);
  s = warp_sum(s);
  if (l == 0) red2[w] = s;
  __syncthreads();
  s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += red2[k];
  const float lse = gm + __logf(s);
  if (threadIdx.x == 0) loss_out[row] = ignored ? 0.f : lse - __bfloat162float(lp[label]);
  if (!write_grad) return;
  __syncthreads();      // the label logit has been read before anyone overwrites it
  const float scale = ignored ? 0.f : *inv_count;
  for (int i = threadIdx.x; i < V8; i += blockDim.x) {
    uint4 u = *reinterpret_cast<const uint4*>(lp + i * 8);
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 f = __bfloat1622float2(h[k]);
      const int c = i * 8 + 2 * k;
      f.x = (__expf(f.x - lse) - (c == label ? 1.f : 0.f)) * scale;
      f.y = (__expf(f.y - lse) - (c + 1 == label ? 1.f : 0.f)) * scale;
      h[k] = __floats2bfloat162_rn(f.x, f.y);
    }
    *reinterpret_cast<uint4*>(lp + i * 8) = u;
  }
  for (int i = V8 * 8 + threadIdx.x; i < V; i += blockDim.x) {
    const float x = __bfloat162float(lp[i]);
    lp[i] = __float2bfloat16((__expf(x - lse) - (i == label ? 1.f : 0.f)) * scale);
  }
}

// dst = src * (*scale), rounded once to bf16; 8 elements per thread and iteration.
template <typename ST>
__global__ void __launch_bounds__(256) scale_kernel(const ST* __restrict__ src, bf16* __restrict__ dst, const float* __restrict__ scale, long n) {
  const float sc = *scale;
  const long step = static_cast<long>(gridDim.x) * 256 * 8;
  for (long i = (static_cast<long>(blockIdx.x) * 256 + threadIdx.x) * 8; i < n; i += step) {
    if (i + 8 <= n) {
      float a[4], b[4];
      load4(src + i, a);
      load4(src + i + 4, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) { a[k] *= sc; b[k] *= sc; }
      store4(dst + i, a);
      store4(dst + i + 4, b);
    } else {
      for (long e = i; e < n; ++e) dst[e] = __float2bfloat16(static_cast<float>(src[e]) * sc);
    }
  }
}

inline int grid_cap(long want, int per_sm) {
  long cap = static_cast<long>(nsa::sm_count()) * per_sm;
  return static_cast<int>(want < cap ? (want < 1 ? 1 : want) : cap);
}
AdamArgs make_args(int step, float lr, float b1, float b2, float eps, float wd) {
  AdamArgs a;
  a.lr = lr; a.beta1 = b1; a.beta2 = b2; a.eps = eps; a.wd = wd;
  a.bc1 = 1.f - powf(b1, (float)step);
  a.bc2_sqrt = sqrtf(1.f - powf(b2, (float)step));
  return a;
}
// ------------------------------------------------------------------------------------
// Asymmetric affine block quantisation of SOAP's eigenbases: every row is cut into blocks of
// q_block columns; a block stores uint8 codes q = round(x / scale + zero) with
// scale = (max - min) / (2^bits - 1) and zero = round(-min / scale) kept as a float.  One warp per block.
// Divisions are IEEE (not the fast-math approximations) so the codes match the PyTorch form.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) affine_quant_kernel(const float* __restrict__ t, uint8_t* __restrict__ q,
                                                           float* __restrict__ scale, float* __restrict__ zero, long rows,
                                                           int cols, int q_block, int nblk, float qmax) {
  const int lane = threadIdx.x & 31;
  const long wid = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (wid >= rows * nblk) return;
  const long row = wid / nblk;
  const int blk = static_cast<int>(wid - row * nblk);
  const float* src = t + row * cols;
  const int c0 = blk * q_block;
  float lo = INFINITY, hi = -INFINITY;
  for (int j = lane; j < q_block; j += 32) {
    const int c = min(c0 + j, cols - 1);            // the padded tail repeats the last column
    const float x = src[c];
    lo = fminf(lo, x);
    hi = fmaxf(hi, x);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const float sc = fmaxf(__fdiv_rn(hi - lo, qmax), 1e-12f);
  const float zp = rintf(__fdiv_rn(-lo, sc));        // not clamped: a one-signed block has its zero outside the code range
  if (lane == 0) { scale[wid] = sc; zero[wid] = zp; }
  uint8_t* dst = q + (row * nblk + blk) * static_cast<long>(q_block);
  for (int j = lane; j < q_block; j += 32) {
    const int c = min(c0 + j, cols - 1);
    const float v = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(src[c], sc), zp)), 0.f), qmax);
    dst[j] = static_cast<uint8_t>(v);
  }
}
__global__ void __launch_bounds__(256) affine_dequant_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scale,
                                                             const float* __restrict__ zero, float* __restrict__ out,
                                                             long rows, int cols, int q_block, int nblk) {
  const long n = rows * cols;
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long row = i / cols;
    const int c = static_cast<int>(i - row * cols);
    const long b = row * nblk + c / q_block;
    out[i] = (static_cast<float>(q[row * static_cast<long>(nblk) * q_block + c]) - zero[b]) * scale[b];
  }
}
}  // namespace

// Seven 64-bit words per tensor: p, g, m, v, a, b (addresses; see AdamItem) and the element count.
static bool next_item(const long long* w, AdamItem& it) {
  it.p = reinterpret_cast<void*>(w[0]);
  it.g = reinterpret_cast<const void*>(w[1]);
  it.m = reinterpret_cast<void*>(w[2]);
  it.v = reinterpret_cast<void*>(w[3]);
  it.a = reinterpret_cast<float*>(w[4]);
  it.b = reinterpret_cast<float*>(w[5]);
  it.n = w[6];
  return it.n > 0;
}

// fp32 state.  p: bf16 (p_fp32 = 0) or fp32; g: bf16 (g_fp32 = 0) or fp32; m, v fp32; a: fp32 master or null.
extern "C" int nsa_adamw_multi(const long long* words, int tensors, const float* grad_scale, int p_fp32, int g_fp32, int step,
                               float lr, float b1, float b2, float eps, float wd, cudaStream_t st) {
  const AdamArgs a = make_args(step, lr, b1, b2, eps, wd);
  for (int t = 0; t < tensors;) {
    AdamList list;
    list.count = 0;
    long units = 0;
    for (; t < tensors && list.count < kMaxItems; ++t) {
      AdamItem& it = list.item[list.count];
      if (!next_item(words + 7 * t, it)) continue;
      const uintptr_t all = reinterpret_cast<uintptr_t>(it.m) | reinterpret_cast<uintptr_t>(it.v) | reinterpret_cast<uintptr_t>(it.a);
      const bool wide = !(all & 15) && !(reinterpret_cast<uintptr_t>(it.p) & (p_fp32 ? 15 : 7)) &&
                        !(reinterpret_cast<uintptr_t>(it.g) & (g_fp32 ? 15 : 7));
      units += (it.n + 1023) / 1024;
      it.end = wide ? units : -units - 1;
      ++list.count;
    }
    if (units == 0) continue;
    const int grid = grid_cap(units, 8);
    if (p_fp32 && g_fp32) adamw_kernel<float, float><<<grid, 256, 0, st>>>(list, grad_scale, units, a);
    else if (p_fp32) adamw_kernel<float, bf16><<<grid, 256, 0, st>>>(list, grad_scale, units, a);
    else if (g_fp32) adamw_kernel<bf16, float><<<grid, 256, 0, st>>>(list, grad_scale, units, a);
    else adamw_kernel<bf16, bf16><<<grid, 256, 0, st>>>(list, grad_scale, units, a);
    nsa::count_launch();
  }
  return 0;
}
extern "C" int nsa_adamw_step(void* p, const void* g, float* m, float* v, float* master, const float* grad_scale,
                              long n, int p_fp32, int g_fp32, int step, float lr, float b1, float b2, float eps, float wd,
                              cudaStream_t st) {
  const long long w[7] = {(long long)p, (long long)g, (long long)m, (long long)v, (long long)master, 0, n};
  return nsa_adamw_multi(w, 1, grad_scale, p_fp32, g_fp32, step, lr, b1, b2, eps, wd, st);
}

// 8-bit state: m, v codes; a, b their scales.  Element counts must be multiples of 256.
// cb_signed / cb_unsigned: device pointers to 256 fp32 entries.
extern "C" int nsa_adamw8bit_multi(const long long* words, int tensors, const float* cb_signed, const float* cb_unsigned,
                                   const float* grad_scale, int p_fp32, int g_fp32, int step, float lr, float b1, float b2,
                                   float eps, float wd, cudaStream_t st) {
  for (int t = 0; t < tensors; ++t)
    if (words[7 * t + 6] > 0 && words[7 * t + 6] % 256)
      return nsa::fail(NSA_ERR_SHAPE, "adamw8bit: element count must be a multiple of 256");
  const AdamArgs a = make_args(step, lr, b1, b2, eps, wd);
  for (int t = 0; t < tensors;) {
    AdamList list;
    list.count = 0;
    long nb = 0;
    for (; t < tensors && list.count < kMaxItems; ++t) {
      AdamItem& it = list.item[list.count];
      if (!next_item(words + 7 * t, it)) continue;
      nb += it.n / 256;
      it.end = nb;
      ++list.count;
    }
    if (nb == 0) continue;
    const int grid = grid_cap((nb + 7) / 8, 4);
    if (p_fp32 && g_fp32) adamw8bit_kernel<float, float><<<grid, 256, 0, st>>>(list, cb_signed, cb_unsigned, grad_scale, nb, a);
    else if (p_fp32) adamw8bit_kernel<float, bf16><<<grid, 256, 0, st>>>(list, cb_signed, cb_unsigned, grad_scale, nb, a);
    else if (g_fp32) adamw8bit_kernel<bf16, float><<<grid, 256, 0, st>>>(list, cb_signed, cb_unsigned, grad_scale, nb, a);
    else adamw8bit_kernel<bf16, bf16><<<grid, 256, 0, st>>>(list, cb_signed, cb_unsigned, grad_scale, nb, a);
    nsa::count_launch();
  }
  return 0;
}
extern "C" int nsa_adamw8bit_step(void* p, const void* g, uint8_t* mq, float* mabs, uint8_t* vq, float* vabs,
                                  const float* cb_signed, const float* cb_unsigned, const float* grad_scale, long n,
                                  int p_fp32, int g_fp32, int step, float lr, float b1, float b2, float eps, float wd,
                                  cudaStream_t st) {
  const long long w[7] = {(long long)p, (long long)g, (long long)mq, (long long)vq, (long long)mabs, (long long)vabs, n};
  return nsa_adamw8bit_multi(w, 1, cb_signed, cb_unsigned, grad_scale, p_fp32, g_fp32, step, lr, b1, b2, eps, wd, st);
}

// out (device scalar) = [out +] sum(g^2).  partial: scratch of nsa_sumsq_parts() floats.
extern "C" int nsa_sumsq_parts() { return nsa::sm_count() * 4; }
extern "C" int nsa_sumsq(const void* g, long n, int g_fp32, float* partial, float* out, int accumulate, cudaStream_t st) {
  const int parts = grid_cap((n + 255) / 256, 4);
  if (g_fp32) sumsq_partial_kernel<float><<<parts, 256, 0, st>>>((const float*)g, n, partial);
  else sumsq_partial_kernel<bf16><<<parts, 256, 0, st>>>((const bf16*)g, n, partial);
  sumsq_final_kernel<<<1, 32, 0, st>>>(partial, parts, out, accumulate);
  nsa::count_launch(2);
  return 0;
}

extern "C" int nsa_cross_entropy(void* logits, const long* labels, float* loss_rows, const float* inv_count, long rows,
                                 int V, long ld, long ignore_index, int write_grad, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (ld % 8) return nsa::fail(NSA_ERR_SHAPE, "cross_entropy: row pitch must be a multiple of 8");
  cross_entropy_kernel<<<(unsigned)rows, 256, 0, st>>>((bf16*)logits, labels, loss_rows, inv_count, V, ld, ignore_index, write_grad,
                                                       nsa::status_ptr());
  nsa::count_launch();
  return 0;
}

// dst (bf16) = src (fp32 or bf16) * (*scale); bases 16-byte aligned.
extern "C" int nsa_scale_bf16(const void* src, void* dst, const float* scale, long n, int src_fp32, cudaStream_t st) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) return nsa::fail(NSA_ERR_ALIGNMENT, "scale: 16-byte aligned bases required");
  const int grid = grid_cap((n + 2047) / 2048, 8);
  if (src_fp32) scale_kernel<float><<<grid, 256, 0, st>>>((const float*)src, (bf16*)dst, scale, n);
  else scale_kernel<bf16><<<grid, 256, 0, st>>>((const bf16*)src, (bf16*)dst, scale, n);
  nsa::count_launch();
  return 0;
}

// t: [rows, cols] fp32 -> q: [rows, nblk * q_block] uint8, scale / zero: [rows, nblk] with nblk = ceil(cols / q_block).
extern "C" int nsa_affine_quant(const float* t, uint8_t* q, float* scale, float* zero, long rows, int cols, int q_block,
                                int bits, cudaStream_t st) {
  if (rows <= 0 || cols <= 0 || q_block <= 0 || bits < 1 || bits > 8) return nsa::fail(NSA_ERR_SHAPE, "affine_quant: bad shape");
  const int nblk = (cols + q_block - 1) / q_block;
  const long warps = rows * nblk;
  affine_quant_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(t, q, scale, zero, rows, cols, q_block, nblk,
                                                                   static_cast<float>((1 << bits) - 1));
  nsa::count_launch();
  return 0;
}
extern "C" int nsa_affine_dequant(const uint8_t* q, const float* scale, const float* zero, float* out, long rows, int cols,
                                  int q_block, cudaStream_t st) {
  if (rows <= 0 || cols <= 0 || q_block <= 0) return nsa::fail(NSA_ERR_SHAPE, "affine_dequant: bad shape");
  const int nblk = (cols + q_block - 1) / q_block;
  const long n = rows * cols;
  const long blocks = std::min<long>((n + 255) / 256, 148L * 16);
  affine_dequant_kernel<<<(unsigned)blocks, 256, 0, st>>>(q, scale, zero, out, rows, cols, q_block, nblk);
  nsa::count_launch();
  return 0;
}
