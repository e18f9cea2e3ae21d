// Mamba-2 SSD (state-space duality) on tcgen05 tensor cores.  Chunk length 128, state width
// N = 128, head width P = 64, one group of B/C shared by all heads.
//
// For one (batch, head) with a_t = dt_t * A (<= 0), cum = inclusive cumsum of a inside the
// chunk, tot = cum at the chunk end, and H the N x P state entering the chunk:
//     P_ij    = (C_i . B_j) exp(cum_i - cum_j) dt_j   (j <= i)          "decayed scores"
//     y_i     = sum_j P_ij x_j + exp(cum_i) C_i H + D x_i
//     H_next  = exp(tot) H + sum_j exp(tot - cum_j) dt_j B_j (outer) x_j
// Kernels (chunk_state: one CTA per (chunk, head, batch)):
//   chunk_state : the sum in H_next (mode 0), or G = sum_i exp(cum_i) C_i (outer) dy_i (mode 1,
//                 the per-chunk term of the state gradient);   fp32 [.., N, P]
//   state pass  : the recurrence over chunks (forward) / its reverse (backward), elementwise
//   chunk_out   : y for the chunk (three MMAs: C B^T, P x, C H)
//   chunk_grad  : dx, dB / dC summed over the heads that a CTA has of a chunk, and the two row
//                 scalars dy.(y - D x) and x.dx from which d(dt) and dA follow by a suffix sum.
// chunk_out and chunk_grad are persistent: a CTA walks a run of (chunk, head) items.
// Decay factors are formed per element in registers (exp2 of a difference that is <= 0), never
// stored; the [128 x 128] P and dS tiles live only on chip, as bf16 MMA operands.
#include <algorithm>
#include "f32x2.cuh"
#include "host.cuh"
#include "tc5.cuh"

namespace {
typedef __nv_bfloat16 bf16;
constexpr int L = 128;      // chunk length
constexpr int NS = 128;     // state width
constexpr int PD = 64;      // head width
constexpr int BOXB = 16384; // bytes of a [128 rows][64 bf16] swizzled box
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void st_row64(uint8_t* kblock, int row, const uint32_t (&pk)[32]) {
  uint8_t* base = kblock + row * 128;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(base + ((j ^ (row & 7)) << 4)) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
}
__device__ __forceinline__ void ld_row64(const uint8_t* kblock, int row, float (&out)[64]) {
  const uint8_t* base = kblock + row * 128;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint4 v = *reinterpret_cast<const uint4*>(base + ((j ^ (row & 7)) << 4));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 f = __bfloat1622float2(h[k]);
      out[8 * j + 2 * k] = f.x;
      out[8 * j + 2 * k + 1] = f.y;
    }
  }
}
// 32 columns col0.. of a tile of [128][64] boxes; the row's 16-byte pieces are swizzled as above
__device__ __forceinline__ void st_row32(uint8_t* tile, int row, int col0, const uint32_t (&pk)[16]) {
  uint8_t* base = tile + (col0 >> 6) * BOXB + row * 128;
  const int j0 = (col0 & 63) >> 3;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    *reinterpret_cast<uint4*>(base + (((j0 + j) ^ (row & 7)) << 4)) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
}
template <int N>
__device__ __forceinline__ void ld_row(const uint8_t* tile, int row, int col0, float (&out)[N]) {
  const uint8_t* base = tile + (col0 >> 6) * BOXB + row * 128;
  const int j0 = (col0 & 63) >> 3;
#pragma unroll
  for (int j = 0; j < N / 8; ++j) {
    const uint4 v = *reinterpret_cast<const uint4*>(base + (((j0 + j) ^ (row & 7)) << 4));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(h[k]);
      out[8 * j + 2 * k] = f.x;
      out[8 * j + 2 * k + 1] = f.y;
    }
  }
}
__device__ __forceinline__ void tld32(uint32_t taddr, float (&out)[32]) {
  uint32_t a[32];
  tc5::tmem_ld_x32(taddr, a);
  tc5::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; ++j) out[j] = __uint_as_float(a[j]);
}
__device__ __forceinline__ void tld16(uint32_t taddr, float (&out)[16]) {
  uint32_t a[16];
  tc5::tmem_ld_x16(taddr, a);
  tc5::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 16; ++j) out[j] = __uint_as_float(a[j]);
}
__device__ __forceinline__ void tld64(uint32_t taddr, float (&out)[64]) {
  uint32_t a[32], b[32];
  tc5::tmem_ld_x32(taddr, a);
  tc5::tmem_ld_x32(taddr + 32, b);
  tc5::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; ++j) { out[j] = __uint_as_float(a[j]); out[32 + j] = __uint_as_float(b[j]); }
}

__device__ __forceinline__ float2 unpack2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }

// OR over the sixteen computing warps of a kernel that has one more
__device__ __forceinline__ bool compute_any(bool bad) {
  int any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 1, 512, p;\n\tselp.s32 %0, 1, 0, q;\n\t}\n"
               : "=r"(any) : "r"(static_cast<int>(bad)) : "memory");
  return any != 0;
}

struct SsdParams {
  const float* dt;     // [B, T, H] (after softplus)
  const float* A;      // [H] (negative)
  const float* Dskip;  // [H] or null
  int B, T, H, nc, c0; // c0: first chunk of the launch
  // chunk_state
  float* S_out;        // [B, nc, H, NS, PD] fp32
  float* gamma_out;    // [B, nc, H] or null
  // chunk_out, chunk_grad (y and dx leave through their tensor maps)
  int quota;           // (chunk, head) items per CTA
  int slots;           // partial tiles of dB and dC per chunk: one per CTA that has heads of it
  float* dB_part;      // [B, T, slots, NS] sums over a CTA's heads of the chunk
  float* dC_part;
  float* q_out;        // [B, T, H]  dy . (y - D x)
  float* k_out;        // [B, T, H]  x . dx (without the D term)
  float* r_out;        // [B, T, H]  dy . x (gradient of the skip weight D before the sum over tokens), or null
  KernelStatus* status;
};

// dt of four neighbouring rows per lane of a chunk that starts at t0 (one warp)
__device__ __forceinline__ float4 load_dt4(const SsdParams& p, int b, int t0, int h) {
  const int t = t0 + 4 * (threadIdx.x & 31);
  const float* src = p.dt + (static_cast<long>(b) * p.T + t) * p.H + h;
  return make_float4(t < p.T ? src[0] : 0.f, t + 1 < p.T ? src[p.H] : 0.f, t + 2 < p.T ? src[2 * p.H] : 0.f,
                     t + 3 < p.T ? src[3 * p.H] : 0.f);
}
// One warp: inclusive sums of dt A over the chunk, in units of log 2.  Every kernel forms its decays from these, as differences of
// sums: the gradients of dt and A are differences of terms that different kernels compute, and cancel as far as the decays agree.
// (The sum before a lane comes from the lane before.  Taking this lane's own part off its sum instead would give rows in front of
// a long or non-finite step that step's rounding error, or a NaN.)
__device__ __forceinline__ float4 chunk_sums(float4 dt, float a) {
  const int lane = threadIdx.x & 31;
  float4 v = make_float4(dt.x * a, dt.y * a, dt.z * a, dt.w * a);
  v.y += v.x;
  v.z += v.y;
  v.w += v.z;
  float run = v.w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float n = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += n;
  }
  float off = __shfl_up_sync(0xffffffffu, run, 1);
  if (lane == 0) off = 0.f;
  // products of their own: fused with the subtractions that follow they would round differently from one kernel to the next
  return make_float4(__fmul_rn(off + v.x, LOG2E), __fmul_rn(off + v.y, LOG2E), __fmul_rn(off + v.z, LOG2E), __fmul_rn(run, LOG2E));
}

// ---------------------------------------------------------------------------------------
// chunk_state.  MODE 0: rows of Bm scaled by exp(tot - cum_j) dt_j, values = x.
//               MODE 1: rows of Cm scaled by exp(cum_i),            values = dy.
// out[N, P] = scaled^T [N x 128] * values [128 x P]
// ---------------------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(128, 2)
ssd_chunk_state_kernel(const __grid_constant__ CUtensorMap tm_bc, const __grid_constant__ CUtensorMap tm_v,
                       const SsdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sBC = smem;                 // [2 chunks][128 t][64]  raw rows, then scaled in place
  uint8_t* sV = sBC + 2 * BOXB;        // [128 t][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + BOXB);
  uint64_t* full = bars;
  uint64_t* done = bars + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* cum = reinterpret_cast<float*>(bars + 4);
  float* dts = cum + L;

  const int r = threadIdx.x, warp = r >> 5;
  const int h = blockIdx.x, c = p.c0 + blockIdx.y, b = blockIdx.z;    // see each_slab
  const int t0 = c * L;
  if (r == 0) {
    *abort_flag = 0;
    tc5::mbar_init(full, 1);
    tc5::mbar_init(done, 1);
    tc5::fence_barrier_init();
    tc5::mbar_expect_tx(full, 3 * BOXB);
    tc5::tma_load_3d(sBC, &tm_bc, full, 0, t0, b);
    tc5::tma_load_3d(sBC + BOXB, &tm_bc, full, 64, t0, b);
    tc5::tma_load_4d(sV, &tm_v, full, 0, h, t0, b);
  }
  if (warp == 1) { tc5::tmem_alloc(tmem_slot, 64); tc5::tmem_relinquish(); }
  if (warp == 0) {
    const float4 dt = load_dt4(p, b, t0, h);
    reinterpret_cast<float4*>(cum)[r] = chunk_sums(dt, p.A[h]);
    reinterpret_cast<float4*>(dts)[r] = dt;
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const float tot = cum[L - 1];
  bool ok = tc5::mbar_wait(full, 0, abort_flag, p.status, STATUS_TIMEOUT_SMEM_FULL);
  if (ok) {
    const float sc = MODE == 0 ? exp2f(tot - cum[r]) * dts[r] : exp2f(cum[r]);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float v[64];
      ld_row64(sBC + half * BOXB, r, v);
      uint32_t pk[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) pk[j] = tc5::pack_bf16(v[2 * j] * sc, v[2 * j + 1] * sc);
      st_row64(sBC + half * BOXB, r, pk);
    }
  }
  tc5::fence_proxy_async();
  tc5::fence_before_sync();
  if (__syncthreads_or(!ok)) ok = false;
  if (ok && warp == 0) {
    // the whole warp stays converged and one elected lane issues: descriptors then live in uniform
    // registers and an MMA costs the issuing thread a few cycles instead of 70 to 100
    const bool lead = tc5::elect_one();
    tc5::fence_after_sync();
    constexpr uint32_t idesc = tc5::make_idesc_bf16(128, PD, 1, 1);
    const uint64_t a0 = tc5::desc_mnmajor(tc5::smem_u32(sBC), BOXB), v0 = tc5::desc_mnmajor(tc5::smem_u32(sV), BOXB);
    if (lead) {
#pragma unroll
      for (int kk = 0; kk < L / 16; ++kk)
        tc5::mma_ss(tmem, a0 + static_cast<uint64_t>((kk * 2048) >> 4), v0 + static_cast<uint64_t>((kk * 2048) >> 4), idesc, kk > 0 ? 1u : 0u);
      tc5::mma_commit(done);
    }
    __syncwarp();
  }
  if (ok && !tc5::mbar_wait(done, 0, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) ok = false;
  if (!__syncthreads_or(!ok)) {
    tc5::fence_after_sync();
    float o[64];
    tld64(tmem + (static_cast<uint32_t>(warp * 32) << 16), o);
    // The tile is contiguous in memory but a thread owns a row of it, and direct stores would put 16 bytes into
    // 32 rows per instruction: it is turned through the operand tile (free now), pieces swizzled by row.
    float4* stage = reinterpret_cast<float4*>(sBC);
#pragma unroll
    for (int j = 0; j < 16; ++j) stage[r * 16 + (j ^ (r & 15))] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
    __syncthreads();
    float4* dst = reinterpret_cast<float4*>(p.S_out + ((static_cast<long>(b) * p.nc + c) * p.H + h) * NS * PD);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = j * 128 + r;
      dst[i] = stage[(i & ~15) + ((i ^ (i >> 4)) & 15)];
    }
    if (MODE == 0 && r == 0 && p.gamma_out) p.gamma_out[(static_cast<long>(b) * p.nc + c) * p.H + h] = exp2f(tot);
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 1) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 64); }
}

// ---------------------------------------------------------------------------------------
// Items (chunk, head), heads fastest, in runs of p.quota per CTA: what a chunk's heads share (B, C and the scores C B^T)
// is loaded and computed once per run of one chunk ("segment"), and the next items' tiles are in flight meanwhile.
// ---------------------------------------------------------------------------------------
struct Items {
  int n, h, t0, b, H, rows;            // items of the run; head, first token and sequence of the current one; padded length
  __device__ explicit Items(const SsdParams& p) : H(p.H), rows(p.nc * L) {
    const int total = p.B * p.nc * p.H, first = blockIdx.x * p.quota;
    n = min(p.quota, total - first);
    h = first % H;
    t0 = first / H % p.nc * L;
    b = first / H / p.nc;
  }
  __device__ void next() {
    if (++h < H) return;
    h = 0;
    t0 += L;
    if (t0 == rows) { t0 = 0; ++b; }
  }
  __device__ bool opens(int k) const { return k == 0 || h == 0; }              // first item of a segment
  __device__ bool closes(int k) const { return k + 1 == n || h + 1 == H; }     // last one
};

// One warp: cum[] = inclusive sums of dt A in units of log 2, dts[] = dt, for 128 rows.  Pairs of rows in different blocks of
// 32 need no exponential of their own: with m the sum at the end of an earlier block, exp(c_i - c_j) = exp(c_i - m)
// exp(m - c_j), and both exponents are <= 0.  colf[] receives the factors that belong to columns:
//   FWD  (columns j, rows i): for row block q = 1..3, m = end of block q - 1: exp(m - c_j) dt_j, j < 32 q, at 16 q (q - 1) + j
//   !FWD (columns i, rows j): for row block q = 0..2, m = end of block q:     exp(c_i - m), i >= 32 (q + 1), at later_block(q) + i
__device__ __forceinline__ int later_block(int q) { return 16 * q * (7 - q) - 32 * (q + 1); }   // 0, 96, 160 at the block's first row
template <bool FWD>
__device__ __forceinline__ void chunk_scan_warp(float4 dt, float a, float* cum, float* dts, float* colf) {
  const int lane = threadIdx.x & 31, blk = lane >> 3;
  const float4 v = chunk_sums(dt, a);
  *reinterpret_cast<float4*>(cum + 4 * lane) = v;
  *reinterpret_cast<float4*>(dts + 4 * lane) = dt;
  auto ex = [](float x) { return exp2f(fminf(x, 0.f)); };
#pragma unroll
  for (int q = 0; q < 3; ++q) {                      // m = sum at the end of block q
    const float m = __shfl_sync(0xffffffffu, v.w, 8 * q + 7);
    if (FWD) {
      if (blk <= q)
        *reinterpret_cast<float4*>(colf + 16 * q * (q + 1) + 4 * lane) =
            make_float4(ex(m - v.x) * dt.x, ex(m - v.y) * dt.y, ex(m - v.z) * dt.z, ex(m - v.w) * dt.w);
    } else if (blk > q) {
      *reinterpret_cast<float4*>(colf + later_block(q) + 4 * lane) = make_float4(ex(v.x - m), ex(v.y - m), ex(v.z - m), ex(v.w - m));
    }
  }
}

// ---------------------------------------------------------------------------------------
// chunk_out: y = P x + exp(cum) (C H) + D x.
// Sixteen warps compute the weights of one item, then finish the rows of the item before, whose products ran meanwhile;
// three more issue, copy and scan the step sizes.  C B^T stays in registers for all heads of a segment, P goes to tensor
// memory as the A operand, y leaves from the place of x.  16384 tokens x 64 heads x 64: 179 us as a CTA per (chunk, head), 102 with one
// warp for issue, copies and scan, 94 with three; x, H and y (403 MB) take 62 at the copy rate.
// ---------------------------------------------------------------------------------------
constexpr int OUT_ST = 4;                             // stages of (x, H)
constexpr int OUT_SMEM = 1024 + (4 + 2 * OUT_ST) * BOXB + 2 * (2 * L + 192) * 4 + 256;
__global__ void __launch_bounds__(608, 1)
ssd_chunk_out_kernel(const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ CUtensorMap tm_b,
                     const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_h,
                     const __grid_constant__ CUtensorMap tm_y, const SsdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sC = smem;                  // [2 k-blocks][128][64]
  uint8_t* sB = sC + 2 * BOXB;
  uint8_t* stages = sB + 2 * BOXB;     // x [128 t][64], H [128 n][64]
  float* scan = reinterpret_cast<float*>(stages + 2 * OUT_ST * BOXB);   // even and odd items: cum, dts, colf
  uint64_t* bars = reinterpret_cast<uint64_t*>(scan + 2 * (2 * L + 192));
  uint64_t *full = bars, *cb = bars + OUT_ST, *ms = cb + 1, *sread = cb + 2;
  uint64_t *scanned = cb + 3, *ready = cb + 5, *done = cb + 7;        // even and odd items
  uint64_t* left = cb + 9;                             // per stage
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(left + OUT_ST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = tc5::warp_index();
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < OUT_ST; ++i) { tc5::mbar_init(full + i, 1); tc5::mbar_init(left + i, 16); }
    tc5::mbar_init(cb, 1);
    tc5::mbar_init(ms, 1);
    tc5::mbar_init(sread, 16);
    for (int i = 0; i < 2; ++i) {
      tc5::mbar_init(scanned + i, 1);
      tc5::mbar_init(ready + i, 16);
      tc5::mbar_init(done + i, 1);
    }
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 512); tc5::tmem_relinquish(); }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t cS = 0, cP = 128, cYi = 256, cYo = 384;     // the last three: 64 columns for even and odd items each
  auto wait = [&](uint64_t* bar, int phase, int code) {
    return tc5::mbar_wait_warp(bar, phase & 1, abort_flag, p.status, code);
  };
  if (warp == 16) {                                    // products
    constexpr uint32_t id_s = tc5::make_idesc_bf16(128, 128, 0, 0);
    constexpr uint32_t id_y = tc5::make_idesc_bf16(128, PD, 0, 1);
    const bool lead = tc5::elect_one();                // converged warp, elected lane issues (see ssd_chunk_state_kernel)
    Items cur(p);
    const int n = cur.n;
    const uint64_t cc = tc5::desc_kmajor(tc5::smem_u32(sC)), bb = tc5::desc_kmajor(tc5::smem_u32(sB));
    int seg = 0;
    for (int k = 0; k < n; ++k, cur.next()) {
      const int buf = k & 1, s = k % OUT_ST;
      if (cur.opens(k)) {
        if (k > 0 && !wait(sread, seg - 1, STATUS_TIMEOUT_TMEM_EMPTY)) break;
        if (!wait(cb, seg, STATUS_TIMEOUT_SMEM_FULL)) break;
        tc5::fence_after_sync();
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < NS / 16; ++kk) {
            const uint64_t off = static_cast<uint64_t>(((kk >> 2) * BOXB + (kk & 3) * 32) >> 4);
            tc5::mma_ss(tmem + cS, cc + off, bb + off, id_s, kk > 0 ? 1u : 0u);
          }
          tc5::mma_commit(ms);
        }
        __syncwarp();
        ++seg;
      }
      if (k > 1 && !wait(left + (k - 2) % OUT_ST, (k - 2) / OUT_ST, STATUS_TIMEOUT_TMEM_EMPTY)) break;      // its columns are free
      if (!wait(full + s, k / OUT_ST, STATUS_TIMEOUT_SMEM_FULL)) break;
      tc5::fence_after_sync();
      const uint64_t xx = tc5::desc_mnmajor(tc5::smem_u32(stages + s * 2 * BOXB), BOXB);
      const uint64_t hh = tc5::desc_mnmajor(tc5::smem_u32(stages + s * 2 * BOXB + BOXB), BOXB);
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < NS / 16; ++kk)
          tc5::mma_ss(tmem + cYi + buf * 64, cc + static_cast<uint64_t>(((kk >> 2) * BOXB + (kk & 3) * 32) >> 4),
                      hh + static_cast<uint64_t>((kk * 2048) >> 4), id_y, kk > 0 ? 1u : 0u);
      }
      __syncwarp();
      if (!wait(ready + buf, k >> 1, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk)
          tc5::mma_ts(tmem + cYo + buf * 64, tmem + cP + buf * 64 + kk * 8, xx + static_cast<uint64_t>((kk * 2048) >> 4), id_y, kk > 0 ? 1u : 0u);
        tc5::mma_commit(done + buf);
      }
      __syncwarp();
    }
  } else if (warp == 17) {                             // loads and stores
    const bool lead = tc5::elect_one();
    Items cur(p), ahead(p), behind(p);                 // the item of a step, the next to be loaded, the next to be stored
    const int n = cur.n, item0 = blockIdx.x * p.quota;
    auto load = [&](int k) {                           // item k, which is `ahead`
      const int s = k % OUT_ST;
      uint8_t* st = stages + s * 2 * BOXB;
      tc5::mbar_expect_tx(full + s, 2 * BOXB);
      tc5::tma_load_4d(st, &tm_x, full + s, 0, ahead.h, ahead.t0, ahead.b);
      tc5::tma_load_2d(st + BOXB, &tm_h, full + s, 0, (item0 + k) * NS);
    };
    auto store = [&](int k) {                          // item k, which is `behind`; rows past T are clipped by the copy engine
      tc5::tma_store_4d(&tm_y, stages + (k % OUT_ST) * 2 * BOXB, 0, behind.h, behind.t0, behind.b);
      tc5::tma_store_commit();
    };
    bool ok = true;
    for (int k = 0; k < n; ++k, cur.next()) {
      if (cur.opens(k)) {                              // C and B of its chunk, over those that the products of item k - 1 read
        if (k > 0 && !(ok = wait(done + ((k - 1) & 1), (k - 1) >> 1, STATUS_TIMEOUT_TMEM_FULL))) break;
        if (lead) {
          tc5::mbar_expect_tx(cb, 4 * BOXB);
          tc5::tma_load_3d(sC, &tm_c, cb, 0, cur.t0, cur.b);
          tc5::tma_load_3d(sC + BOXB, &tm_c, cb, 64, cur.t0, cur.b);
          tc5::tma_load_3d(sB, &tm_b, cb, 0, cur.t0, cur.b);
          tc5::tma_load_3d(sB + BOXB, &tm_b, cb, 64, cur.t0, cur.b);
        }
        __syncwarp();
      }
      if (k == 0) {
        for (int i = 0; i < 2 && i < n; ++i, ahead.next())
          if (lead) load(i);
      } else {
        if (!(ok = wait(left + (k - 1) % OUT_ST, (k - 1) / OUT_ST, STATUS_TIMEOUT_TMEM_EMPTY))) break;
        if (lead) store(k - 1);
        behind.next();
      }
      if (lead && k + 2 < n) {                         // over the stage of item k - 2, stored one step ago
        tc5::tma_store_wait_read<1>();
        load(k + 2);
      }
      ahead.next();
      __syncwarp();
    }
    if (ok && wait(left + (n - 1) % OUT_ST, (n - 1) / OUT_ST, STATUS_TIMEOUT_TMEM_EMPTY)) {
      if (lead) store(n - 1);
    } else if (lead) {                                 // loads may still be in flight
      for (int i = 0; i < OUT_ST; ++i) tc5::mbar_drain(full + i);
      tc5::mbar_drain(cb);
    }
    if (lead) tc5::tma_store_wait_read<0>();
    __syncwarp();
  } else if (warp == 18) {                             // sums of step sizes, two items ahead
    Items cur(p);
    const int n = cur.n;
    float4 dt = load_dt4(p, cur.b, cur.t0, cur.h);
    float a = p.A[cur.h];
    for (int k = 0; k < n; ++k) {
      float4 dt_next = make_float4(0.f, 0.f, 0.f, 0.f);
      float a_next = 0.f;
      cur.next();
      if (k + 1 < n) { dt_next = load_dt4(p, cur.b, cur.t0, cur.h); a_next = p.A[cur.h]; }
      if (k > 1 && !wait(ready + (k & 1), (k >> 1) - 1, STATUS_TIMEOUT_TMEM_EMPTY)) break;       // those of item k - 2 have been read
      float* at = scan + (k & 1) * (2 * L + 192);
      chunk_scan_warp<true>(dt, a, at, at + L, at + 2 * L);
      tc5::arrive_warp(scanned + (k & 1));
      dt = dt_next;
      a = a_next;
    }
  } else {
    const int r = threadIdx.x & 127, lane = r & 31, quad = warp & 3, grp = warp >> 2;    // row, its block of 32, column block
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    float s[32];                                       // C_i . B_j of the segment: row i = r, columns j = 32 grp ..
    float e_open = 0.f, dsk_open = 0.f;                // exp(cum) and skip weight of the item whose rows are still open
    Items cur(p);
    const int n = cur.n;
    int seg = 0;
    for (int k = 0; k <= n; ++k, cur.next()) {
      float e = 0.f, dsk = 0.f;
      if (k < n) {
        const int buf = k & 1;
        if (p.Dskip) dsk = p.Dskip[cur.h];             // in flight until the item's rows are finished
        if (cur.opens(k)) {
          if (!wait(ms, seg, STATUS_TIMEOUT_TMEM_FULL)) break;
          tc5::fence_after_sync();
          tld32(lanes + cS + grp * 32, s);
          tc5::fence_before_sync();
          tc5::arrive_warp(sread);
          ++seg;
        }
        if (!wait(scanned + buf, k >> 1, STATUS_TIMEOUT_SMEM_FULL)) break;
        const float* cum = scan + buf * (2 * L + 192);
        const float *dts = cum + L + grp * 32, *cols = cum + grp * 32;
        const float ci = cum[r];
        e = exp2f(ci);
        uint32_t pk[16];
        if (grp < quad) {                              // every column is before every row
          const float rowf = exp2f(fminf(ci - cum[32 * quad - 1], 0.f));
          const float* f = cum + 2 * L + 16 * quad * (quad - 1) + grp * 32;          // see chunk_scan_warp
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 w = *reinterpret_cast<const float4*>(f + j);
            pk[j / 2] = tc5::pack_bf16(s[j] * (rowf * w.x), s[j + 1] * (rowf * w.y));
            pk[j / 2 + 1] = tc5::pack_bf16(s[j + 2] * (rowf * w.z), s[j + 3] * (rowf * w.w));
          }
        } else if (grp == quad) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            // operands fetched and the weight computed for every j, then selected: a conditional around
            // the loads costs a branch per element
            const float2 c = *reinterpret_cast<const float2*>(cols + j), d = *reinterpret_cast<const float2*>(dts + j);
            const float w0 = exp2f(fminf(ci - c.x, 0.f)) * d.x, w1 = exp2f(fminf(ci - c.y, 0.f)) * d.y;
            pk[j / 2] = tc5::pack_bf16(j <= lane ? s[j] * w0 : 0.f, j + 1 <= lane ? s[j + 1] * w1 : 0.f);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = 0u;
        }
        tc5::tmem_st_x16(lanes + cP + buf * 64 + grp * 16, pk);
        tc5::tmem_st_wait();
        tc5::fence_before_sync();
        tc5::arrive_warp(ready + buf);
      }
      if (k > 0) {                                     // rows of the item before, whose products ran meanwhile
        const int q = k - 1, buf = q & 1;
        if (!wait(full + q % OUT_ST, q / OUT_ST, STATUS_TIMEOUT_SMEM_FULL) || !wait(done + buf, q >> 1, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        uint8_t* sX = stages + (q % OUT_ST) * 2 * BOXB;
        float xf[16], yo[16], yi[16];
        ld_row(sX, r, grp * 16, xf);
        tld16(lanes + cYo + buf * 64 + grp * 16, yo);
        tld16(lanes + cYi + buf * 64 + grp * 16, yi);
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2)
          o[i / 2] = tc5::pack_bf16(yo[i] + e_open * yi[i] + dsk_open * xf[i], yo[i + 1] + e_open * yi[i + 1] + dsk_open * xf[i + 1]);
        uint8_t* base = sX + r * 128;                  // the thread's own piece of x, which the products have read
#pragma unroll
        for (int j = 0; j < 2; ++j)
          *reinterpret_cast<uint4*>(base + (((grp * 2 + j) ^ (r & 7)) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        tc5::fence_proxy_async();
        tc5::fence_before_sync();
        tc5::arrive_warp(left + q % OUT_ST);
      }
      e_open = e;
      dsk_open = dsk;
    }
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 512); }
}

// ---------------------------------------------------------------------------------------
// chunk_grad for one (chunk, head, batch), given dy, the state entering the chunk (H) and
// the gradient of the state leaving it (dHn):
//   S = C B^T, R = dy x^T;  P = S w, dS = R w  with w_ij = exp(cum_i - cum_j) dt_j (j <= i)
//   dx_j  = sum_i P_ij dy_i + s_j B_j dHn + D dy_j          (s_j = exp(tot - cum_j) dt_j)
//   dC_i  = sum_j dS_ij B_j + (exp(cum_i) dy_i) H^T         summed over the heads of a segment in tensor memory
//   dB_j  = sum_i dS_ij C_i + (s_j x_j) dHn^T               likewise
//   q_i   = dy_i . (y_i - D x_i) = sum_j P_ij R_ij + exp(cum_i) dy_i . (C_i H),   k_j = x_j . (dx_j - D dy_j),   r = dy . x
// Scores are held transposed (lanes j, columns i): P^T, dS^T and the scaled rows of x and dy are A operands in tensor memory, and
// only dS needs a tile in shared memory.  Sixteen warps compute, a quarter of the columns each; the seventeenth loads the
// next item (64 KB in flight during a whole item), scans its step sizes, issues the products and stores.
// The sums over heads leave once per segment, as fp32 tiles that nsa_ssd_finish adds up.
// 16384 tokens x 64 heads x 64, 128 states: 563 us and 95 for the sum over heads as a CTA per (chunk, head), 309 and 9 now.  Bound by the
// phases of an item (scores, weights, products, rows), each waiting for the one before; the next item's loads and scan run beside
// them.  A warp of its own for the scan (320) or for the row sums (312) gives nothing.
// ---------------------------------------------------------------------------------------
constexpr int GRAD_SMEM = 1024 + 14 * BOXB + (2 * L + 192) * 4 + 128;
__global__ void __launch_bounds__(544, 1)
ssd_chunk_grad_kernel(const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ CUtensorMap tm_b,
                      const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_dy,
                      const __grid_constant__ CUtensorMap tm_h, const __grid_constant__ CUtensorMap tm_dh,
                      const __grid_constant__ CUtensorMap tm_dx, const SsdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sC = smem;                  // 2 boxes
  uint8_t* sB = sC + 2 * BOXB;         // 2 boxes
  uint8_t* sDS = sB + 2 * BOXB;        // 2 boxes: dS^T [j][i]
  uint8_t* stages = sDS + 2 * BOXB;    // 2 x (x, dy, H [n][p], dHn [n][p])
  float* cum = reinterpret_cast<float*>(stages + 8 * BOXB);
  float* dts = cum + L;
  float* colf = dts + L;
  uint64_t* bars = reinterpret_cast<uint64_t*>(colf + 192);
  uint64_t *full = bars, *cb = bars + 2, *ms = bars + 3, *sread = bars + 4, *scanned = bars + 5;
  uint64_t *m0 = bars + 6, *m1 = bars + 7, *ready = bars + 8, *m2 = bars + 9, *m3 = bars + 10, *sums = bars + 11, *left = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = tc5::warp_index();
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    tc5::mbar_init(full, 1);
    tc5::mbar_init(full + 1, 1);
    tc5::mbar_init(cb, 1);
    tc5::mbar_init(ms, 1);
    tc5::mbar_init(sread, 16);
    tc5::mbar_init(scanned, 1);
    tc5::mbar_init(m0, 1);
    tc5::mbar_init(m1, 1);
    tc5::mbar_init(ready, 16);
    tc5::mbar_init(m2, 1);
    tc5::mbar_init(m3, 1);
    tc5::mbar_init(sums, 1);
    tc5::mbar_init(left, 16);
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 512); tc5::tmem_relinquish(); }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // TMEM columns.  R^T [0, 128): of each 16 columns, the first 8 become P^T and the others dS^T (bf16 pairs, 16 i).
  // B dHn, then dx [128, 192).  C H [192, 256): of each 16, 8 become exp(cum) dy and 8 s x (16 p).  dB, dC [256, 512).
  const uint32_t cR = 0, cX = 128, cY = 192, cDB = 256, cDC = 384;
  auto wait = [&](uint64_t* bar, int phase, int code) {
    return tc5::mbar_wait_warp(bar, phase & 1, abort_flag, p.status, code);
  };
  if (warp == 16) {
    constexpr uint32_t id_s = tc5::make_idesc_bf16(128, 128, 0, 0);     // K-major x K-major -> [128 x 128]
    constexpr uint32_t id_kn64 = tc5::make_idesc_bf16(128, PD, 0, 1);   // K-major A, MN-major B -> [128 x 64]
    constexpr uint32_t id_kn128 = tc5::make_idesc_bf16(128, NS, 0, 1);  // K-major A, MN-major B -> [128 x 128]
    constexpr uint32_t id_tn128 = tc5::make_idesc_bf16(128, NS, 1, 1);  // MN-major A, MN-major B -> [128 x 128]
    const bool lead = tc5::elect_one();                // converged warp, elected lane issues (see ssd_chunk_state_kernel)
    Items cur(p), ahead(p), behind(p);                 // the item of a step, the next to be loaded and scanned, the next to be stored
    const int n = cur.n, item0 = blockIdx.x * p.quota;
    auto load = [&](int k) {                           // item k, which is `ahead`
      uint8_t* st = stages + (k & 1) * 4 * BOXB;
      uint64_t* bar = full + (k & 1);
      tc5::mbar_expect_tx(bar, 4 * BOXB);
      tc5::tma_load_4d(st, &tm_x, bar, 0, ahead.h, ahead.t0, ahead.b);
      tc5::tma_load_4d(st + BOXB, &tm_dy, bar, 0, ahead.h, ahead.t0, ahead.b);
      tc5::tma_load_2d(st + 2 * BOXB, &tm_h, bar, 0, (item0 + k) * NS);
      tc5::tma_load_2d(st + 3 * BOXB, &tm_dh, bar, 0, (item0 + k) * NS);
    };
    auto store = [&](int k) {                          // dx of item k, `behind`, from the place of x; rows past T are clipped by the copy engine
      tc5::tma_store_4d(&tm_dx, stages + (k & 1) * 4 * BOXB, 0, behind.h, behind.t0, behind.b);
      tc5::tma_store_commit();
      tc5::tma_store_wait_read<0>();                   // the next item but one goes there
    };
    const uint64_t ck = tc5::desc_kmajor(tc5::smem_u32(sC)), bk = tc5::desc_kmajor(tc5::smem_u32(sB));
    const uint64_t cm = tc5::desc_mnmajor(tc5::smem_u32(sC), BOXB), bm = tc5::desc_mnmajor(tc5::smem_u32(sB), BOXB);
    const uint64_t dsm = tc5::desc_mnmajor(tc5::smem_u32(sDS), BOXB);
    auto kblock = [](int kk) { return static_cast<uint64_t>(((kk >> 2) * BOXB + (kk & 3) * 32) >> 4); };
    auto kcols = [](int kk) { return static_cast<uint64_t>((kk * 32) >> 4); };
    auto krow = [](int kk) { return static_cast<uint64_t>((kk * 2048) >> 4); };
    auto box = [&](int k, int i) { return tc5::smem_u32(stages + ((k & 1) * 4 + i) * BOXB); };      // x, dy, H, dHn of item k
    int seg = 0;
    auto load_chunk = [&]() {                          // C and B of the chunk of `cur`
      if (lead) {
        tc5::mbar_expect_tx(cb, 4 * BOXB);
        tc5::tma_load_3d(sC, &tm_c, cb, 0, cur.t0, cur.b);
        tc5::tma_load_3d(sC + BOXB, &tm_c, cb, 64, cur.t0, cur.b);
        tc5::tma_load_3d(sB, &tm_b, cb, 0, cur.t0, cur.b);
        tc5::tma_load_3d(sB + BOXB, &tm_b, cb, 64, cur.t0, cur.b);
      }
      __syncwarp();
    };
    auto open_segment = [&]() {                        // S^T = B C^T
      if (!wait(cb, seg, STATUS_TIMEOUT_SMEM_FULL)) return false;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < NS / 16; ++kk) tc5::mma_ss(tmem + cR, bk + kblock(kk), ck + kblock(kk), id_s, kk > 0 ? 1u : 0u);
        tc5::mma_commit(ms);
      }
      __syncwarp();
      if (!wait(sread, seg, STATUS_TIMEOUT_TMEM_EMPTY)) return false;
      tc5::fence_after_sync();
      ++seg;
      return true;
    };
    auto scores = [&](int k) {                         // R^T = x dy^T, over P^T and dS^T of the item before
      if (lead) {
        const uint64_t xk = tc5::desc_kmajor(box(k, 0)), dyk = tc5::desc_kmajor(box(k, 1));
#pragma unroll
        for (int kk = 0; kk < PD / 16; ++kk) tc5::mma_ss(tmem + cR, xk + kcols(kk), dyk + kcols(kk), id_s, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m0);
      }
      __syncwarp();
    };
    auto state_rows = [&](int k) {                     // C H, over the scaled rows of the item before
      if (lead) {
        const uint64_t hm = tc5::desc_mnmajor(box(k, 2), BOXB);
#pragma unroll
        for (int kk = 0; kk < NS / 16; ++kk) tc5::mma_ss(tmem + cY, ck + kblock(kk), hm + krow(kk), id_kn64, kk > 0 ? 1u : 0u);
      }
      __syncwarp();
    };
    load_chunk();
    if (lead) load(0);
    chunk_scan_warp<false>(load_dt4(p, ahead.b, ahead.t0, ahead.h), p.A[ahead.h], cum, dts, colf);
    tc5::arrive_warp(scanned);
    ahead.next();
    // A step issues the rest of item k and the first products of item k + 1 between them, so that the scores of k + 1 are
    // there when the warps have finished the rows of k, and the sums over heads run behind their work.
    bool ok = open_segment() && wait(full, 0, STATUS_TIMEOUT_SMEM_FULL);
    if (ok) {
      tc5::fence_after_sync();
      scores(0);
      state_rows(0);
    }
    for (int k = 0; k < n && ok; ++k) {
      const bool opens = cur.opens(k), closes = cur.closes(k), more = k + 1 < n;
      if (k > 0) {
        if (!(ok = wait(left, k - 1, STATUS_TIMEOUT_TMEM_EMPTY))) break;
        tc5::fence_after_sync();
      }
      if (lead) {
        const uint64_t dhm = tc5::desc_mnmajor(box(k, 3), BOXB);
#pragma unroll
        for (int kk = 0; kk < NS / 16; ++kk)           // B dHn, over dx of the item before
          tc5::mma_ss(tmem + cX, bk + kblock(kk), dhm + krow(kk), id_kn64, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m1);
        if (k > 0) store(k - 1);
      }
      if (k > 0) behind.next();
      __syncwarp();
      if (more) {                                      // over item k - 1, whose last products are complete when these are
        if (!(ok = wait(m1, k, STATUS_TIMEOUT_TMEM_FULL))) break;
        if (lead) load(k + 1);
        __syncwarp();
      }
      float4 dt_next = make_float4(0.f, 0.f, 0.f, 0.f);
      float a_next = 0.f;
      if (more) { dt_next = load_dt4(p, ahead.b, ahead.t0, ahead.h); a_next = p.A[ahead.h]; }
      ahead.next();
      if (!(ok = wait(ready, k, STATUS_TIMEOUT_TMEM_EMPTY))) break;
      tc5::fence_after_sync();
      const uint32_t sum = opens ? 0u : 1u;
      if (lead) {
        const uint64_t dym = tc5::desc_mnmajor(box(k, 1), BOXB);
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk)            // dx += P^T dy
          tc5::mma_ts(tmem + cX, tmem + cR + 16 * kk, dym + krow(kk), id_kn64, 1u);
        tc5::mma_commit(m2);
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk)            // dB += dS^T C
          tc5::mma_ts(tmem + cDB, tmem + cR + 16 * kk + 8, cm + krow(kk), id_kn128, kk > 0 ? 1u : sum);
      }
      __syncwarp();
      const bool same = more && !closes;               // item k + 1 is of the same chunk
      if (same) {
        if (!(ok = wait(full + ((k + 1) & 1), (k + 1) >> 1, STATUS_TIMEOUT_SMEM_FULL))) break;
        tc5::fence_after_sync();
        scores(k + 1);
      }
      if (lead) {
        const uint64_t hk = tc5::desc_kmajor(box(k, 2)), dhk = tc5::desc_kmajor(box(k, 3));
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk)            // dC += dS B
          tc5::mma_ss(tmem + cDC, dsm + krow(kk), bm + krow(kk), id_tn128, kk > 0 ? 1u : sum);
        tc5::mma_commit(m3);
#pragma unroll
        for (int kk = 0; kk < PD / 16; ++kk)           // dC += (exp(cum) dy) H^T
          tc5::mma_ts(tmem + cDC, tmem + cY + 16 * kk, hk + kcols(kk), id_s, 1u);
#pragma unroll
        for (int kk = 0; kk < PD / 16; ++kk)           // dB += (s x) dHn^T
          tc5::mma_ts(tmem + cDB, tmem + cY + 16 * kk + 8, dhk + kcols(kk), id_s, 1u);
        if (closes) tc5::mma_commit(sums);
      }
      __syncwarp();
      if (more) {                                      // this item's sums of step sizes have been read
        chunk_scan_warp<false>(dt_next, a_next, cum, dts, colf);
        tc5::arrive_warp(scanned);
      }
      cur.next();
      if (same) {
        state_rows(k + 1);
      } else if (more) {                               // every product and every reader of the segment is through: C and B may go
        if (!(ok = wait(left, k, STATUS_TIMEOUT_TMEM_EMPTY))) break;
        load_chunk();
        if (!(ok = open_segment() && wait(full + ((k + 1) & 1), (k + 1) >> 1, STATUS_TIMEOUT_SMEM_FULL))) break;
        tc5::fence_after_sync();
        scores(k + 1);
        state_rows(k + 1);
      }
    }
    if (ok && wait(left, n - 1, STATUS_TIMEOUT_TMEM_EMPTY)) {
      if (lead) store(n - 1);
    } else if (lead) {                                 // copies may still be in flight
      tc5::mbar_drain(full);
      tc5::mbar_drain(full + 1);
      tc5::mbar_drain(cb);
      tc5::tma_store_wait_read<0>();
    }
    __syncwarp();
  } else {
    const int r = threadIdx.x & 127, lane = r & 31, quad = warp & 3, grp = warp >> 2;    // row, its block of 32, column block
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    float s[32];                                       // B_j . C_i of the segment: row j = r, columns i = 32 grp ..
    bool ok = true;
    int seg = 0;
    Items cur(p);
    const int n = cur.n;
    for (int k = 0; k < n; ++k, cur.next()) {
      const int t = cur.t0 + r;
      const float dsk = p.Dskip ? p.Dskip[cur.h] : 0.f;          // in flight until the item's last phase
      uint8_t* sX = stages + (k & 1) * 4 * BOXB;
      uint8_t* sDY = sX + BOXB;
      if (cur.opens(k)) {
        ok = ok && wait(ms, seg, STATUS_TIMEOUT_TMEM_FULL);
        if (ok) {
          tc5::fence_after_sync();
          tld32(lanes + cR + grp * 32, s);
          tc5::fence_before_sync();
          tc5::arrive_warp(sread);
        }
        ++seg;
      }
      ok = ok && wait(scanned, k, STATUS_TIMEOUT_SMEM_FULL) && wait(full + (k & 1), k >> 1, STATUS_TIMEOUT_SMEM_FULL) &&
           wait(m0, k, STATUS_TIMEOUT_TMEM_FULL);
      float q_intra = 0.f;      // sum_j P_ij R_ij with P as rounded for the MMA (pairs exactly with x.dx): of column i = 32 grp + lane
      float q_inter = 0.f, e = 0.f;
      if (ok) {
        tc5::fence_after_sync();
        const float cj = cum[r], dtj = dts[r];
        const float s_row = exp2f(cum[L - 1] - cj) * dtj;
        e = exp2f(cj);
        // 16 columns: weights -> P^T, dS^T and the column sums of P^T R^T over this warp's 32 rows
        auto sixteen = [&](const int hf, auto weight) {
          float rr[16], g[16];
          tld16(lanes + cR + grp * 32 + hf * 16, rr);
          uint32_t pk[8], ds[8];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 w = weight(hf * 16 + i);
            pk[i / 2] = tc5::pack_bf16(s[hf * 16 + i] * w.x, s[hf * 16 + i + 1] * w.y);
            ds[i / 2] = tc5::pack_bf16(rr[i] * w.x, rr[i + 1] * w.y);
            const float2 pr = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk[i / 2]));
            g[i] = pr.x * rr[i];
            g[i + 1] = pr.y * rr[i + 1];
          }
          tc5::tmem_st_x8(lanes + cR + grp * 32 + hf * 16, pk);
          tc5::tmem_st_x8(lanes + cR + grp * 32 + hf * 16 + 8, ds);
          tc5::tmem_st_wait();
          if (hf == 0 && k > 0) ok = wait(m3, k - 1, STATUS_TIMEOUT_TMEM_FULL);     // dS of the item before has been read
          const int c0 = grp * 32 + hf * 16, j0 = (c0 & 63) >> 3;
          uint8_t* base = sDS + (c0 >> 6) * BOXB + r * 128;
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<uint4*>(base + (((j0 + j) ^ (r & 7)) << 4)) = make_uint4(ds[4 * j], ds[4 * j + 1], ds[4 * j + 2], ds[4 * j + 3]);
          // halves of the columns change hands between lanes until a lane holds the sum of one column
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < o; ++i) {
              const float send = up ? g[i] : g[i + o];
              g[i] = (up ? g[i + o] : g[i]) + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          g[0] += __shfl_xor_sync(0xffffffffu, g[0], 16);
          if ((lane >> 4) == hf) q_intra = g[0];
        };
        if (grp > quad) {                              // every column i is behind every row j
          const float rowf = exp2f(fminf(cum[32 * quad + 31] - cj, 0.f)) * dtj;
          const float* f = colf + later_block(quad) + grp * 32;
          auto weight = [&](int i) {
            const float2 c = *reinterpret_cast<const float2*>(f + i);
            return make_float2(rowf * c.x, rowf * c.y);
          };
          sixteen(0, weight);
          sixteen(1, weight);
        } else if (grp == quad) {
          auto weight = [&](int i) {                   // computed for every i, then selected (no branch per element)
            const float2 c = *reinterpret_cast<const float2*>(cum + grp * 32 + i);
            const float w0 = exp2f(fminf(c.x - cj, 0.f)) * dtj, w1 = exp2f(fminf(c.y - cj, 0.f)) * dtj;
            return make_float2(i >= lane ? w0 : 0.f, i + 1 >= lane ? w1 : 0.f);
          };
          sixteen(0, weight);
          sixteen(1, weight);
        } else {                                       // masked: zero operands
          uint32_t z[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) z[i] = 0u;
          tc5::tmem_st_x16(lanes + cR + grp * 32, z);
          tc5::tmem_st_x16(lanes + cR + grp * 32 + 16, z);
          tc5::tmem_st_wait();
          if (k > 0) ok = wait(m3, k - 1, STATUS_TIMEOUT_TMEM_FULL);
          st_row32(sDS, r, grp * 32, z);
        }
        ok = ok && wait(m1, k, STATUS_TIMEOUT_TMEM_FULL);
        if (ok) {
          tc5::fence_after_sync();
          // dx starts from s_j B_j dHn; rows of dy and x, scaled, take the place of C H.  (The sources of a tcgen05.st must
          // stay as they are until it is waited for: all three leave together.)
          float v[16], u[16];
          uint32_t w[16], a[8], c[8];
          tld16(lanes + cX + grp * 16, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(s_row * v[i]);
          tld16(lanes + cY + grp * 16, v);
          ld_row(sDY, r, grp * 16, u);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            q_inter += u[i] * v[i] + u[i + 1] * v[i + 1];
            a[i / 2] = tc5::pack_bf16(e * u[i], e * u[i + 1]);
          }
          ld_row(sX, r, grp * 16, u);
#pragma unroll
          for (int i = 0; i < 16; i += 2) c[i / 2] = tc5::pack_bf16(s_row * u[i], s_row * u[i + 1]);
          tc5::tmem_st_x16(lanes + cX + grp * 16, w);
          tc5::tmem_st_x8(lanes + cY + grp * 16, a);
          tc5::tmem_st_x8(lanes + cY + grp * 16 + 8, c);
          tc5::tmem_st_wait();
          tc5::fence_proxy_async();
          tc5::fence_before_sync();
          tc5::arrive_warp(ready);
        }
      }
      ok = ok && wait(m2, k, STATUS_TIMEOUT_TMEM_FULL);
      if (ok) {
        tc5::fence_after_sync();
        float kacc = 0.f, racc = 0.f;
        float g[16], xf[16], df[16];
        tld16(lanes + cX + grp * 16, g);
        ld_row(sX, r, grp * 16, xf);
        ld_row(sDY, r, grp * 16, df);
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          kacc += xf[i] * g[i] + xf[i + 1] * g[i + 1];
          racc += xf[i] * df[i] + xf[i + 1] * df[i + 1];
          o[i / 2] = tc5::pack_bf16(g[i] + dsk * df[i], g[i + 1] + dsk * df[i + 1]);
        }
        uint8_t* base = sX + r * 128;                  // the thread's own piece of x, which the products have read
#pragma unroll
        for (int j = 0; j < 2; ++j)
          *reinterpret_cast<uint4*>(base + (((grp * 2 + j) ^ (r & 7)) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        // the sums of its row and column on their way to one: over its own piece of dy
        *reinterpret_cast<float4*>(sDY + r * 128 + (((grp * 2) ^ (r & 7)) << 4)) = make_float4(kacc, racc, q_inter, q_intra);
      }
      if (compute_any(!ok)) { ok = false; break; }     // all sixteen warps leave together
      const long tok = static_cast<long>(cur.b) * p.T + t;
      if (t < p.T && grp < 3) {                        // the four pieces add up in a fixed order; group g finishes sum g
        auto piece = [&](int row, int g) { return reinterpret_cast<const float*>(sDY + row * 128 + (((g * 2) ^ (row & 7)) << 4)); };
        auto row_sum = [&](int i) { return (piece(r, 0)[i] + piece(r, 1)[i]) + (piece(r, 2)[i] + piece(r, 3)[i]); };
        const long o = tok * p.H + cur.h;
        if (grp == 0) p.k_out[o] = row_sum(0);
        else if (grp == 1) { if (p.r_out) p.r_out[o] = row_sum(1); }
        else p.q_out[o] = ((piece(lane, quad)[3] + piece(32 + lane, quad)[3]) + (piece(64 + lane, quad)[3] + piece(96 + lane, quad)[3])) +
                          e * row_sum(2);
      }
      if (cur.closes(k)) {                             // the segment's sums over heads
        ok = wait(sums, seg - 1, STATUS_TIMEOUT_TMEM_FULL);
        if (ok) {
          tc5::fence_after_sync();
          const long chunk = static_cast<long>(cur.b) * p.nc + cur.t0 / L;
          const int slot = blockIdx.x - static_cast<int>(chunk * p.H / p.quota);
          // Sixteen columns at a time through the warp's own piece of dS (its products are complete), so that four lanes write 64 bytes
          // of a row: a lane that writes its own row leaves 16 bytes in each of 32 rows, which took 5 of 16 us of a CTA with one item.
          uint8_t* piece = sDS + (grp >> 1) * BOXB + quad * 32 * 128;
          const int j0 = (grp & 1) * 4, col = lane & 3;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float v[32];
            tld32(lanes + (q ? cDC : cDB) + grp * 32, v);
            float* part = q ? p.dC_part : p.dB_part;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(piece + lane * 128 + (((j0 + j) ^ (lane & 7)) << 4)) =
                    make_float4(v[hf * 16 + 4 * j], v[hf * 16 + 4 * j + 1], v[hf * 16 + 4 * j + 2], v[hf * 16 + 4 * j + 3]);
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int row = i * 8 + (lane >> 2), tr = cur.t0 + quad * 32 + row;
                const float4 w = *reinterpret_cast<const float4*>(piece + row * 128 + (((j0 + col) ^ (row & 7)) << 4));
                if (tr < p.T)
                  *reinterpret_cast<float4*>(part + ((static_cast<long>(cur.b) * p.T + tr) * p.slots + slot) * NS + grp * 32 + hf * 16 + col * 4) = w;
              }
              __syncwarp();
            }
          }
        }
      }
      if (!ok) continue;                               // the next item's vote ends the walk
      tc5::fence_proxy_async();
      tc5::fence_before_sync();
      tc5::arrive_warp(left);
    }
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 512); }
}

// ---------------------------------------------------------------------------------------
// States entering the chunks (BACK: gradients of the states leaving them) in one pass: a CTA walks the chunks of one (head,
// sequence), the state in registers; only its bf16 copies reach memory, where chunk_state and the state pass move 20 bytes per element
// of it.  Two groups of four warps scale the rows of B (C) of every other chunk in place, eight warps add the product of the chunk before to
// the state; the others issue, load, and scan the step sizes, two warps with every other chunk.  (Rows of x are half as many elements, but
// scaled x rounds differently from what the gradients pair it with: dA was a quarter further from its 64-bit value.)
// Bound by the latency of a chunk's steps in each role (waits, proxy fences, loads): 16384 tokens x 64 heads 141 us with one group
// of scaling warps, one scan (its loads alone 1.1 K cycles a chunk), two products in flight and one output buffer; 121 now, and 90 with the
// state's rows in halves on two CTAs.
// ---------------------------------------------------------------------------------------
__host__ __device__ constexpr int walk_stages(int parts) { return parts == 1 ? 4 : 6; }       // of B (C) and x (dy)
constexpr int WALK_ACC = 4;                            // products in tensor memory
constexpr int walk_smem(int parts) { return (2 / parts + 1) * walk_stages(parts) * BOXB + 2 * BOXB / parts + walk_stages(parts) * (L + 4) * 4 + 256; }
// PARTS 2: a CTA has half of the state's rows (blockIdx.x = 2 head + part), so that few heads use twice the SMs and a chunk's steps are
// shorter.
template <bool BACK, int PARTS>
__global__ void __launch_bounds__(PARTS == 1 ? 672 : 640, 1)
ssd_walk_kernel(const __grid_constant__ CUtensorMap tm_bc, const __grid_constant__ CUtensorMap tm_v,
                const __grid_constant__ CUtensorMap tm_out, const SsdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_walk[];     // the stages leave no room to align by hand
  uint8_t* smem = smem_walk;
  if (tc5::smem_u32(smem) & 1023u) {                   // the swizzle needs it; never seen otherwise
    if (threadIdx.x == 0) status_report(p.status, STATUS_BAD_ARGUMENT, blockIdx.x, static_cast<int>(tc5::smem_u32(smem)));
    return;
  }
  constexpr int WALK_ST = walk_stages(PARTS), OUT = BOXB / PARTS;
  constexpr int ROWS = NS / PARTS, BOXES = 2 / PARTS, STAGE = (BOXES + 1) * BOXB;      // of the state, of B (C), of both operands
  uint8_t* sOut = smem + WALK_ST * STAGE;              // [2][ROWS n][64 p]
  float* scale = reinterpret_cast<float*>(sOut + 2 * OUT);      // per stage: row scales, decay of the chunk
  uint64_t* bars = reinterpret_cast<uint64_t*>(scale + WALK_ST * (L + 4));
  uint64_t *full = bars, *empty = bars + WALK_ST, *ready = bars + 2 * WALK_ST, *done = ready + WALK_ACC, *taken = done + WALK_ACC;   // a product's
  uint64_t *written = taken + WALK_ACC, *left = written + 2;       // an output buffer's
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(left + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* decay = reinterpret_cast<float*>(tmem_slot + 2);        // [WALK_ACC]
  const int warp = tc5::warp_index(), lane = threadIdx.x & 31, h = blockIdx.x / PARTS, n0 = blockIdx.x % PARTS * ROWS,
            b = blockIdx.y, nc = p.nc;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < WALK_ST; ++i) { tc5::mbar_init(full + i, 2); tc5::mbar_init(empty + i, 1); }
    for (int i = 0; i < WALK_ACC; ++i) { tc5::mbar_init(ready + i, 4); tc5::mbar_init(done + i, 1); tc5::mbar_init(taken + i, 8); }
    for (int i = 0; i < 2; ++i) { tc5::mbar_init(written + i, 8 / PARTS); tc5::mbar_init(left + i, 1); }
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, WALK_ACC * 64); tc5::tmem_relinquish(); }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, int phase, int code) {
    return tc5::mbar_wait_warp(bar, phase & 1, abort_flag, p.status, code);
  };
  auto chunk_of = [&](int i) { return BACK ? nc - 1 - i : i; };
  auto leave = [&](int i) {                            // chunk i's buffer to memory, one thread
    tc5::tma_store_2d(&tm_out, sOut + (i & 1) * OUT, 0, ((b * nc + chunk_of(i)) * p.H + h) * NS + n0);
    tc5::tma_store_commit();
  };
  const int r = threadIdx.x & 127, half = (warp >> 2) & 1;      // row and half of its columns, for the first sixteen warps
  if (PARTS == 2 && warp < 8) {
    // State, twice: the four warps of either half keep all of it and store that of every other chunk, which takes as long as the rest
    // (the proxy fence alone a quarter).  64 rows are sixteen lanes of each quarter of tensor memory; see the load for the layout.
    const uint32_t acc = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int n = (warp & 3) * 16 + (lane >> 2);
    uint8_t* out = sOut + half * OUT;
    float2 st[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) st[j] = make_float2(0.f, 0.f);
    for (int i = 0; i < nc; ++i) {
      if (i > 0) {
        uint32_t a[32];
        if (!wait(done + (i - 1) % WALK_ACC, (i - 1) / WALK_ACC, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        const float g = decay[(i - 1) % WALK_ACC];            // of the chunk before
        tc5::tmem_ld_16x256b_x8(acc + (i - 1) % WALK_ACC * 64, a);
        tc5::tmem_ld_wait();
        tc5::fence_before_sync();
        tc5::arrive_warp(taken + (i - 1) % WALK_ACC);
        const float2 g2 = make_float2(g, g);
#pragma unroll
        for (int j = 0; j < 16; ++j) st[j] = fma2(g2, st[j], make_float2(__uint_as_float(a[2 * j]), __uint_as_float(a[2 * j + 1])));
      }
      if ((i & 1) != half) continue;
      const bool first = (warp & 3) == 0;              // of the four: sees to their stores
      if (i > 1) {
        if (first) {
          if (lane == 0) tc5::tma_store_wait_read<0>();
          tc5::arrive_warp(left + half);
        }
        if (!wait(left + half, (i >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY)) break;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {                   // columns 8 (j / 2) + 2 (lane % 4), rows n and n + 8
        const int row = n + (j & 1) * 8;
        *reinterpret_cast<uint32_t*>(out + row * 128 + (((j >> 1) ^ (row & 7)) << 4) + (lane & 3) * 4) = tc5::pack_bf16(st[j].x, st[j].y);
      }
      tc5::fence_proxy_async();
      tc5::arrive_warp(written + half);
      if (!first) continue;
      if (!wait(written + half, i >> 1, STATUS_TIMEOUT_SMEM_FULL)) break;
      if (lane == 0) leave(i);
      __syncwarp();
    }
    if ((warp & 3) == 0 && lane == 0) tc5::tma_store_wait_read<0>();
    __syncwarp();
  } else if (warp < 8) {                               // state: row r, columns p = 32 half ..
    const uint32_t acc = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * 32;
    float2 st[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) st[j] = make_float2(0.f, 0.f);
    for (int i = 0; i < nc; ++i) {
      if (i > 0) {
        float a[32];
        if (!wait(done + (i - 1) % WALK_ACC, (i - 1) / WALK_ACC, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        const float g = decay[(i - 1) % WALK_ACC];            // of the chunk before
        tld32(acc + (i - 1) % WALK_ACC * 64, a);
        tc5::fence_before_sync();
        tc5::arrive_warp(taken + (i - 1) % WALK_ACC);
        const float2 g2 = make_float2(g, g);
#pragma unroll
        for (int j = 0; j < 16; ++j) st[j] = fma2(g2, st[j], make_float2(a[2 * j], a[2 * j + 1]));
      }
      uint32_t pk[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) pk[j] = tc5::pack_bf16(st[j].x, st[j].y);
      if (i > 1 && !wait(left + (i & 1), (i >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY)) break;
      st_row32(sOut + (i & 1) * OUT, r, half * 32, pk);
      tc5::fence_proxy_async();
      tc5::arrive_warp(written + (i & 1));
    }
  } else if (warp < 16) {                              // row t of B (C), of every other chunk
    for (int i = half; i + 1 < nc; i += 2) {
      const int s = i % WALK_ST;
      if (!wait(full + s, i / WALK_ST, STATUS_TIMEOUT_SMEM_FULL)) break;
      const float sc = scale[s * (L + 4) + r];
      const float2 f = make_float2(sc, sc);
#pragma unroll
      for (int k = 0; k < BOXES; ++k) {
        uint8_t* row = smem + s * STAGE + k * BOXB + r * 128;
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = *reinterpret_cast<const uint4*>(row + ((j ^ (r & 7)) << 4));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 a = mul2(unpack2(v[j].x), f), c = mul2(unpack2(v[j].y), f), d = mul2(unpack2(v[j].z), f), e = mul2(unpack2(v[j].w), f);
          *reinterpret_cast<uint4*>(row + ((j ^ (r & 7)) << 4)) =
              make_uint4(tc5::pack_bf16(a.x, a.y), tc5::pack_bf16(c.x, c.y), tc5::pack_bf16(d.x, d.y), tc5::pack_bf16(e.x, e.y));
        }
      }
      tc5::fence_proxy_async();
      // the decay goes along to the product's readers, who have taken the one that was in its place
      if (i >= WALK_ACC && !wait(taken + i % WALK_ACC, i / WALK_ACC - 1, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      if (r == 0) decay[i % WALK_ACC] = scale[s * (L + 4) + L];
      tc5::arrive_warp(ready + i % WALK_ACC);
    }
  } else if (warp == 16) {
    constexpr uint32_t idesc = tc5::make_idesc_bf16(ROWS, PD, 1, 1);
    const bool lead = tc5::elect_one();                // converged warp, elected lane issues (see ssd_chunk_state_kernel)
    for (int i = 0; i + 1 < nc; ++i) {                 // nothing follows the last chunk
      const int s = i % WALK_ST;
      const uint64_t a0 = tc5::desc_mnmajor(tc5::smem_u32(smem + s * STAGE), BOXB);
      const uint64_t v0 = tc5::desc_mnmajor(tc5::smem_u32(smem + s * STAGE + BOXES * BOXB), BOXB);
      if (!wait(ready + i % WALK_ACC, i / WALK_ACC, STATUS_TIMEOUT_TMEM_EMPTY)) break;       // also: its place in tensor memory is free
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk)
          tc5::mma_ss(tmem + i % WALK_ACC * 64, a0 + static_cast<uint64_t>((kk * 2048) >> 4), v0 + static_cast<uint64_t>((kk * 2048) >> 4), idesc, kk > 0 ? 1u : 0u);
        tc5::mma_commit(done + i % WALK_ACC);
        tc5::mma_commit(empty + s);
      }
      __syncwarp();
    }
  } else if (warp == 17) {
    const bool lead = tc5::elect_one();
    // into L2 a few chunks ahead: the stages alone leave a load from memory less time than it takes
    constexpr int AHEAD = 8;
    auto prefetch = [&](int i) {
      if (i + 1 >= nc || !lead) return;
      const int t0 = chunk_of(i) * L;
      tc5::tma_prefetch_4d(&tm_v, 0, h, t0, b);
      if (i % p.H != h) return;                        // shared by all heads
#pragma unroll
      for (int k = 0; k < BOXES; ++k) tc5::tma_prefetch_3d(&tm_bc, n0 + k * 64, t0, b);
    };
    for (int i = WALK_ST; i < AHEAD; ++i) prefetch(i);
    bool ok = true;
    for (int i = 0; i + 1 < nc; ++i) {
      const int s = i % WALK_ST, t0 = chunk_of(i) * L;
      uint8_t* st = smem + s * STAGE;
      if (i >= WALK_ST && !(ok = wait(empty + s, i / WALK_ST - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full + s, STAGE);
#pragma unroll
        for (int k = 0; k < BOXES; ++k) tc5::tma_load_3d(st + k * BOXB, &tm_bc, full + s, n0 + k * 64, t0, b);
        tc5::tma_load_4d(st + BOXES * BOXB, &tm_v, full + s, 0, h, t0, b);
      }
      prefetch(i + AHEAD);
      __syncwarp();
    }
    // stages whose last use was not waited for above
    for (int i = nc > WALK_ST + 1 ? nc - WALK_ST : 0; i + 1 < nc && ok; ++i) ok = wait(empty + i % WALK_ST, i / WALK_ST, STATUS_TIMEOUT_SMEM_EMPTY);
    if (!ok && lead)                                   // loads may still be in flight
      for (int i = 0; i < WALK_ST; ++i) tc5::mbar_drain(full + i);
    __syncwarp();
  } else if (warp < 20) {                              // row scales and decay of every other chunk, the next one's step sizes in flight
    const float a = p.A[h];
    auto load_dt = [&](int i) { return load_dt4(p, b, chunk_of(min(i, nc - 1)) * L, h); };
    float4 dt = load_dt(warp - 18), next = load_dt(warp - 16);
    for (int i = warp - 18; i + 1 < nc; i += 2) {
      const int s = i % WALK_ST;
      const float4 c = chunk_sums(dt, a);
      const float tot = __shfl_sync(0xffffffffu, c.w, 31);
      auto weight = [&](float cum, float d) { return BACK ? exp2f(cum) : exp2f(tot - cum) * d; };
      const float4 w = make_float4(weight(c.x, dt.x), weight(c.y, dt.y), weight(c.z, dt.z), weight(c.w, dt.w));
      dt = next;
      next = load_dt(i + 4);
      if (i >= WALK_ST && !wait(empty + s, i / WALK_ST - 1, STATUS_TIMEOUT_SMEM_EMPTY)) break;
      float* sc = scale + s * (L + 4);
      *reinterpret_cast<float4*>(sc + 4 * lane) = w;
      if (lane == 0) sc[L] = exp2f(tot);
      tc5::arrive_warp(full + s);
    }
  } else {                                             // PARTS 1: the stores of all eight state warps
    for (int i = 0; i < nc; ++i) {
      if (!wait(written + (i & 1), i >> 1, STATUS_TIMEOUT_SMEM_FULL)) break;
      if (lane == 0) {
        leave(i);
        tc5::tma_store_wait_read<1>();                 // the one before has left its buffer
      }
      if (i > 0) tc5::arrive_warp(left + ((i - 1) & 1));
    }
    if (lane == 0) tc5::tma_store_wait_read<0>();
    __syncwarp();
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, WALK_ACC * 64); }
}

// ---------------------------------------------------------------------------------------
// State passing over chunks (elementwise).  Layout [B, nc, H, E], E = NS * PD.
// ---------------------------------------------------------------------------------------
// A thread walks the chunks of VEC neighbouring elements.  The recurrence itself is one FMA per chunk; what takes time is
// memory, so the terms of the next eight chunks are always in flight (512 chunks x 64 heads x 8192, bf16 out: 348 us without,
// 268 now).  Few elements leave one warp per scheduler, and then a step is as long as its instructions: pointers move by a
// step, and the bounds are tested outside the unrolled walk (1000 chunks x 3 heads x 63: 87 us with an address computed per
// access, 53 without chunks in flight, 32 now).
template <int VEC>
struct Elems { float v[VEC]; };
template <int VEC>
__device__ __forceinline__ void st_bf16(bf16* p, const Elems<VEC>& x) {
  if constexpr (VEC == 4) *reinterpret_cast<uint2*>(p) = make_uint2(tc5::pack_bf16(x.v[0], x.v[1]), tc5::pack_bf16(x.v[2], x.v[3]));
  else *p = __float2bfloat16(x.v[0]);
}
template <int VEC>
__device__ __forceinline__ Elems<VEC> ld_f32(const float* p) {
  Elems<VEC> e;
  if constexpr (VEC == 4) { const float4 f = *reinterpret_cast<const float4*>(p); e.v[0] = f.x; e.v[1] = f.y; e.v[2] = f.z; e.v[3] = f.w; }
  else e.v[0] = *p;
  return e;
}
template <int VEC>
__device__ __forceinline__ void st_f32(float* p, const Elems<VEC>& x) {
  if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
  else *p = x.v[0];
}
// out[c] = state entering chunk c; step: state <- gamma[c] state + in[c].  BACK walks the chunks in reverse.
template <int VEC, bool BACK>
__global__ void __launch_bounds__(256, 3) ssd_state_kernel(const float* __restrict__ in, const float* __restrict__ gamma,
                                                        float* __restrict__ out, bf16* __restrict__ out_bf,
                                                        float* __restrict__ last, int nc, int H, long E) {
  constexpr int U = 8;
  const long e = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) * VEC;
  if (e >= E) return;
  const int h = blockIdx.y, b = blockIdx.z;
  const long first = (static_cast<long>(b) * nc + (BACK ? nc - 1 : 0)) * H + h;
  const long gstep = BACK ? -H : H, step = gstep * E;              // from one chunk to the next
  in += first * E + e;
  gamma += first;
  if (out) out += first * E + e;
  if (out_bf) out_bf += first * E + e;
  Elems<VEC> st{}, next[U];
  float g_next[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u < nc) { next[u] = ld_f32<VEC>(in + u * step); g_next[u] = gamma[u * gstep]; }
  in += U * step;
  gamma += U * gstep;
  auto advance = [&](int u, bool more) {
    if (out) { st_f32<VEC>(out, st); out += step; }
    if (out_bf) { st_bf16<VEC>(out_bf, st); out_bf += step; }
#pragma unroll
    for (int k = 0; k < VEC; ++k) st.v[k] = g_next[u] * st.v[k] + next[u].v[k];
    if (more) { next[u] = ld_f32<VEC>(in); g_next[u] = *gamma; in += step; gamma += gstep; }
  };
  int i = 0;
  for (; i + 2 * U <= nc; i += U)
#pragma unroll
    for (int u = 0; u < U; ++u) advance(u, true);
  for (; i < nc; i += U)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u < nc) advance(u, i + u + U < nc);
  if (last) st_f32<VEC>(last + (static_cast<long>(b) * H + h) * E + e, st);
}
template <bool BACK>
int launch_state(const float* in, const float* gamma, float* out, void* out_bf, float* last, int B, int nc, int H, long E,
                 cudaStream_t st) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(last) |
                        (reinterpret_cast<uintptr_t>(out_bf) << 1);
  if (E % 4 == 0 && all % 16 == 0)
    ssd_state_kernel<4, BACK><<<dim3((unsigned)((E / 4 + 255) / 256), H, B), 256, 0, st>>>(in, gamma, out, (bf16*)out_bf, last, nc, H, E);
  else
    ssd_state_kernel<1, BACK><<<dim3((unsigned)((E + 255) / 256), H, B), 256, 0, st>>>(in, gamma, out, (bf16*)out_bf, last, nc, H, E);
  nsa::count_launch();
  return 0;
}

// ---------------------------------------------------------------------------------------
// What follows the chunk gradients: sums over heads and over time.
// ---------------------------------------------------------------------------------------
// dB (blockIdx.y = 0) and dC: a token's partial rows, fp32 sums in a fixed order, bf16 out.  A chunk has one partial per CTA of the
// gradient kernel that had heads of it.  A warp owns a token, 16 bytes per lane, FLY partials in flight (see nsa_ssd_finish).
template <int FLY>
__global__ void __launch_bounds__(256) ssd_sum_parts_kernel(const float* __restrict__ dB_part, const float* __restrict__ dC_part,
                                                            bf16* __restrict__ dB, bf16* __restrict__ dC, long rows, int T, int H,
                                                            int nc, int quota, int slots) {
  const long row = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const long first = (row / T * nc + (row % T) / L) * H;           // the chunk's first item
  const int n = static_cast<int>((first + H - 1) / quota - first / quota) + 1;
  const float4* src = reinterpret_cast<const float4*>((blockIdx.y ? dC_part : dB_part) + row * slots * NS) + lane;
  float4 acc = src[0];
  auto add = [&](const float4& v) { acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; };
  if (FLY == 4) {
#pragma unroll 4
    for (int i = 1; i < n; ++i) add(src[i * (NS / 4)]);
  } else {
    for (int i0 = 1; i0 < n; i0 += FLY) {
      float4 v[FLY];
#pragma unroll
      for (int i = 0; i < FLY; ++i)
        if (i0 + i < n) v[i] = src[(i0 + i) * (NS / 4)];
#pragma unroll
      for (int i = 0; i < FLY; ++i)
        if (i0 + i < n) add(v[i]);
    }
  }
  reinterpret_cast<uint2*>((blockIdx.y ? dC : dB) + row * NS)[lane] = make_uint2(tc5::pack_bf16(acc.x, acc.y), tc5::pack_bf16(acc.z, acc.w));
}

// With da_t = sum over t' >= t of (q - k)_t' :  ddt = da A + k / dt,  dA = sum da dt,  dD = sum r  (sums over tokens and batch).
// Chunks of 128 tokens in parallel: one kernel leaves each chunk's totals, the next adds up the totals of the chunks
// behind its own (a few KB from L2) and walks the chunk from its end, a third sums the per-chunk dA and dD.
// Thread = (head of 64, quarter of the chunk).  totals, pA, pD: [B * nc][H].  There are few CTAs, so what bounds them is latency:
// a thread asks for 16 or 32 steps before it adds (16384 tokens x 64 heads: with eight steps in flight 10.8 and 17.4 us, now 5.9 and 8.2; 300 x 32 7.6 and 8.3, now 4.0 and 4.7).
constexpr int QT = L / 4;
__global__ void __launch_bounds__(256, 2) ssd_totals_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                         const float* __restrict__ r, float* __restrict__ totals,
                                                         float* __restrict__ pD, int T, int H, int nc) {
  __shared__ float ss[4][64], sd[4][64];
  const int hl = threadIdx.x & 63, part = threadIdx.x >> 6, c = blockIdx.x, b = blockIdx.y;
  const int t0 = c * L + part * QT, n = min(QT, T - t0);
  for (int h0 = 0; h0 < H; h0 += 64) {
    const int h = h0 + hl;
    float s = 0.f, d = 0.f;
    {
      const long at = (static_cast<long>(b) * T + t0) * H + h;
      const float *qh = q + at, *kh = k + at, *rh = r ? r + at : nullptr;
      const int live = h < H ? n : 0;
#pragma unroll 1
      for (int i0 = 0; i0 < QT; i0 += 16) {                // all 32 at once take 255 registers
        float x[16], y[16], z[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const bool in = i0 + i < live;
          x[i] = in ? qh[static_cast<long>(i0 + i) * H] : 0.f;
          y[i] = in ? kh[static_cast<long>(i0 + i) * H] : 0.f;
          z[i] = r && in ? rh[static_cast<long>(i0 + i) * H] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          s += x[i] - y[i];
          d += z[i];
        }
      }
    }
    ss[part][hl] = s;
    sd[part][hl] = d;
    __syncthreads();
    if (part == 0 && h < H) {
      const long o = (static_cast<long>(b) * nc + c) * H + h;
      totals[o] = (ss[0][hl] + ss[1][hl]) + (ss[2][hl] + ss[3][hl]);
      if (r) pD[o] = (sd[0][hl] + sd[1][hl]) + (sd[2][hl] + sd[3][hl]);
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) ssd_ddt_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                      const float* __restrict__ dt, const float* __restrict__ A,
                                                      const float* __restrict__ totals, float* __restrict__ ddt,
                                                      float* __restrict__ pA, int T, int H, int nc) {
  __shared__ float ss[4][64], sb[4][64], sa[4][64];
  const int hl = threadIdx.x & 63, part = threadIdx.x >> 6, c = blockIdx.x, b = blockIdx.y;
  const int t0 = c * L + part * QT, n = min(QT, T - t0);
  for (int h0 = 0; h0 < H; h0 += 64) {
    const int h = h0 + hl, live = h < H ? n : 0;
    const long i0 = (static_cast<long>(b) * T + t0) * H + h;
    float s = 0.f, behind = 0.f, x[QT], y[QT], z[QT];
#pragma unroll
    for (int i = 0; i < QT; ++i) {
      const long at = i0 + static_cast<long>(i) * H;
      x[i] = i < live ? q[at] : 0.f;
      y[i] = i < live ? k[at] : 0.f;
      z[i] = i < live ? dt[at] : 0.f;
    }
    if (h < H) {
#pragma unroll 16
      for (int cc = c + 1 + part; cc < nc; cc += 4) behind += totals[(static_cast<long>(b) * nc + cc) * H + h];
    }
#pragma unroll
    for (int i = 0; i < QT; ++i) s += x[i] - y[i];
    ss[part][hl] = s;
    sb[part][hl] = behind;
    __syncthreads();
    float da = (sb[0][hl] + sb[1][hl]) + (sb[2][hl] + sb[3][hl]), acc = 0.f;
    for (int p = 3; p > part; --p) da += ss[p][hl];
    const float a = h < H ? A[h] : 0.f;
#pragma unroll
    for (int i = QT - 1; i >= 0; --i)
      if (i < live) {
        da += x[i] - y[i];
        ddt[i0 + static_cast<long>(i) * H] = da * a + y[i] / fmaxf(z[i], 1e-20f);
        acc += da * z[i];
      }
    sa[part][hl] = acc;
    __syncthreads();
    if (part == 0 && h < H) pA[(static_cast<long>(b) * nc + c) * H + h] = (sa[0][hl] + sa[1][hl]) + (sa[2][hl] + sa[3][hl]);
    __syncthreads();
  }
}
// dA[h], dD[h] = sums over the rows of pA, pD in a fixed order.  CTA: 32 heads x 32 groups of rows.
__global__ void __launch_bounds__(1024) ssd_head_sums_kernel(const float* __restrict__ pA, const float* __restrict__ pD,
                                                             float* __restrict__ dA, float* __restrict__ dD, int rows, int H) {
  __shared__ float sums[32][33];
  const int l = threadIdx.x & 31, g = threadIdx.x >> 5, h = blockIdx.x * 32 + l;
  const float* src = blockIdx.y ? pD : pA;
  float s = 0.f;
  if (h < H) {
#pragma unroll 4
    for (int i = g; i < rows; i += 32) s += src[static_cast<long>(i) * H + h];
  }
  sums[g][l] = s;
  __syncthreads();
  s = sums[l][g];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const int hg = blockIdx.x * 32 + g;
  if (l == 0 && hg < H) (blockIdx.y ? dD : dA)[hg] = s;
}

// Launches of one CTA per (chunk, head, sequence).  Heads vary fastest: a head's row of a token is 128 bytes, so CTAs that run
// together read and write neighbouring pieces of the same rows, and share the chunk's B and C tiles in L2.  A grid's second
// dimension ends at 65535, so chunks go in slabs of that many (8.4 M tokens).
template <typename F>
void each_slab(SsdParams& p, F launch) {
  p.c0 = 0;
  do {                                             // no tokens: the launch reports an empty grid
    launch(dim3(p.H, p.nc - p.c0 < 65535 ? p.nc - p.c0 : 65535, p.B));
    nsa::count_launch();
    p.c0 += 65535;
  } while (p.c0 < p.nc);
}

// (chunk, head) items are dealt out in equal runs, one per SM (one CTA fills an SM)
int items_per_cta(int B, int T, int H) {
  const long total = static_cast<long>(B) * ((T + L - 1) / L) * H, sms = nsa::sm_count();
  return static_cast<int>((total + sms - 1) / sms);
}
// Sets the runs of a launch and returns its CTAs (0: nothing to do)
unsigned deal_items(SsdParams& p) {
  p.quota = items_per_cta(p.B, p.T, p.H);
  if (p.quota == 0) return 0;
  const long total = static_cast<long>(p.B) * p.nc * p.H;
  return static_cast<unsigned>((total + p.quota - 1) / p.quota);
}

int map_bc(CUtensorMap* m, const void* base, int B, int T, long ld) {
  uint64_t dims[3] = {(uint64_t)NS, (uint64_t)T, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)T * ld * 2};
  uint32_t box[3] = {64, (uint32_t)L, 1};
  return nsa::make_tmap_bf16(m, base, 3, dims, strides, box, 1);
}
int map_v(CUtensorMap* m, const void* base, int B, int T, int H, long ld) {
  uint64_t dims[4] = {(uint64_t)PD, (uint64_t)H, (uint64_t)T, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)PD * 2, (uint64_t)ld * 2, (uint64_t)T * ld * 2};
  uint32_t box[4] = {64, 1, (uint32_t)L, 1};
  return nsa::make_tmap_bf16(m, base, 4, dims, strides, box, 1);
}
int map_state(CUtensorMap* m, const void* base, long rows, int box_rows = NS) {
  return nsa::make_tmap_2d_bf16(m, base, PD, rows, PD, 64, box_rows);
}
template <typename K>
int smem_attr(K kern, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "ssd: shared memory attribute");
}
int check_dims(int N, int P, long ld_bc, long ld_v) {
  if (N != NS || P != PD) return nsa::fail(NSA_ERR_SHAPE, "ssd: native kernels need d_state 128 and headdim 64");
  if ((ld_bc & 7) || (ld_v & 7)) return nsa::fail(NSA_ERR_ALIGNMENT, "ssd: token strides must be multiples of 8 elements");
  return 0;
}
}  // namespace

extern "C" int nsa_ssd_state_fwd(const float* S, const float* gamma, float* Hprev, void* Hprev_bf16, float* Hlast, int B,
                                 int nc, int H, long E, cudaStream_t st) {
  return launch_state<false>(S, gamma, Hprev, Hprev_bf16, Hlast, B, nc, H, E, st);
}
extern "C" int nsa_ssd_state_bwd(const float* dHprev, const float* gamma, float* dS, void* dS_bf16, int B, int nc, int H,
                                 long E, cudaStream_t st) {
  return launch_state<true>(dHprev, gamma, dS, dS_bf16, nullptr, B, nc, H, E, st);
}

// Partial tiles of dB and dC per chunk that nsa_ssd_chunk_grad writes: the runs of (chunk, head) items that the heads of one
// chunk can fall into.
extern "C" int nsa_ssd_grad_slots(int B, int T, int H) {
  const int quota = items_per_cta(B, T, H);
  return H < 2 || quota == 0 ? 1 : (H - 2) / quota + 2;
}

// dB_part, dC_part [B, T, slots, 128] fp32 of nsa_ssd_chunk_grad -> dB, dC [B, T, 128] bf16; q, k, r (or null), dt [B, T, H], A [H]
// fp32 -> ddt [B, T, H], dA [H], dD [H] (or null).  scratch: 3 * B * ceil(T / 128) * H floats.
extern "C" int nsa_ssd_finish(const float* dB_part, const float* dC_part, const float* q, const float* k, const float* r,
                              const float* dt, const float* A, float* scratch, void* dB, void* dC, float* ddt, float* dA,
                              float* dD, int B, int T, int H, cudaStream_t st) {
  if (B <= 0 || T <= 0 || H <= 0 || (r == nullptr) != (dD == nullptr)) return nsa::fail(NSA_ERR_SHAPE, "ssd_finish: bad arguments");
  const long rows = static_cast<long>(B) * T;
  const int nc = (T + L - 1) / L;
  float *totals = scratch, *pA = totals + static_cast<long>(B) * nc * H, *pD = pA + static_cast<long>(B) * nc * H;
  // A long sequence has two or three partials per token and the kernel is bound by memory, a short one has up to one per head and
  // few tokens: 16384 tokens x 64 heads 9.0 us with four in flight, 17.7 with sixteen; 300 x 48 6.6, 4.7; 128 x 128 11.2, 7.7.
  const int slots = nsa_ssd_grad_slots(B, T, H);
  auto* sum_parts = slots > 4 ? ssd_sum_parts_kernel<16> : ssd_sum_parts_kernel<4>;
  sum_parts<<<dim3((unsigned)((rows + 7) / 8), 2), 256, 0, st>>>(dB_part, dC_part, (bf16*)dB, (bf16*)dC, rows, T, H, nc,
                                                                 items_per_cta(B, T, H), slots);
  ssd_totals_kernel<<<dim3(nc, B), 256, 0, st>>>(q, k, r, totals, pD, T, H, nc);
  ssd_ddt_kernel<<<dim3(nc, B), 256, 0, st>>>(q, k, dt, A, totals, ddt, pA, T, H, nc);
  ssd_head_sums_kernel<<<dim3((H + 31) / 32, dD ? 2 : 1), 1024, 0, st>>>(pA, pD, dA, dD, B * nc, H);
  nsa::count_launch(4);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_ssd_finish launch");
}

// One pass over the chunks (nsa_ssd_states) or chunk_state and the state pass.  The walk is counted with 3.2 us, and 1.13 a chunk for each head
// per SM: 0.2 more than a chunk has come to take, which decides nothing, as up to half as many heads as SMs have the halves below for
// where it would, and beyond that the walk is the faster form at every length.  The two kernels take 6.6 us and 0.095 a chunk (the pass is a
// chain), 5.1 and 0.0165 per (chunk, head), or 0.019 per (chunk, head), whichever is the most, and have a gap between them.  Walk and two
// kernels, us: 1300 tokens x 1 head 12.5, 7.3; 2000 x 24 17.2, 11.4; 4000 x 32 31, 20.5; 300 x 75 5.8, 9.3; 4000 x 75 31, 50; 1000 x 128 10.6,
// 20.8; 200 x 149 8.1, 11.2 (a head more than SMs: the start is not paid again); 3000 x 149 51, 72; 129 x 320 11.7, 18.2; 4000 x 320 105, 195.
extern "C" int nsa_ssd_states_in_one(int B, int T, int H) {
  const long heads = static_cast<long>(B) * H, chunks = (T + L - 1) / L, items = heads * chunks, sms = nsa::sm_count();
  const double walk = 3.2 + 1.13 * chunks * ((heads + sms - 1) / sms);
  return walk <= std::max({6.6 + 0.095 * chunks, 5.1 + 0.0165 * items, 0.019 * items}) + 0.5;
}

// How the states are best formed: 0 chunk_state and the state pass, 1 one walk over the chunks per head, 2 two walks with half of the
// state's rows each.  The halves take 3.0 us and 0.56 a chunk, and 0.0019 more a chunk for each head (memory); they are the better form as long
// as all of them run at once, except where heads are few and chunks many.  us of halves, one walk and two kernels: 300 tokens x 1 head
// 4.7, 5.9, 6.7; 1000 x 32 8.7, 10.5, 9.1; 1000 x 64 9.2, 10.9, 13.5; 4000 x 32 24.5, 32, 21; 4000 x 64 26, 34, 40; 16384 x 48 87, 120, 122; 16384 x 64
// 90, 121, 169; 16384 x 128 181, 127.
extern "C" int nsa_ssd_states_form(int B, int T, int H) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  const long heads = static_cast<long>(B) * H, chunks = (T + L - 1) / L, items = heads * chunks, sms = nsa::sm_count();
  const double two = std::max({6.6 + 0.095 * chunks, 5.1 + 0.0165 * items, 0.019 * items}) + 0.5;
  if (chunks > 1 && 2 * heads <= sms && 3.0 + (0.56 + 0.0019 * heads) * chunks <= two) return 2;
  return nsa_ssd_states_in_one(B, T, H) ? 1 : 0;
}

// back = 0: bc = B rows, v = x -> states entering the chunks; back = 1: bc = C rows, v = dy -> gradients of the states leaving them.
// out: bf16 [B, nc, H, N, P].
extern "C" int nsa_ssd_states(int back, const void* bc, long ld_bc, const void* v, long ld_v, const float* dt, const float* A,
                              void* out, int B, int T, int H, int N, int P, cudaStream_t st) {
  int rc = check_dims(N, P, ld_bc, ld_v);
  if (rc) return rc;
  SsdParams p{};
  p.dt = dt; p.A = A; p.B = B; p.T = T; p.H = H; p.nc = (T + L - 1) / L; p.status = nsa::status_ptr();
  CUtensorMap tb, tv, to;
  if ((rc = map_bc(&tb, bc, B, T, ld_bc))) return rc;
  if ((rc = map_v(&tv, v, B, T, H, ld_v))) return rc;
  const int parts = nsa_ssd_states_form(B, T, H) == 2 ? 2 : 1, bytes = walk_smem(parts);
  if ((rc = map_state(&to, out, static_cast<long>(B) * p.nc * H * NS, NS / parts))) return rc;
  auto* kernel = parts == 2 ? (back ? ssd_walk_kernel<true, 2> : ssd_walk_kernel<false, 2>) : back ? ssd_walk_kernel<true, 1> : ssd_walk_kernel<false, 1>;
  static bool cfg[4] = {};
  bool& ready = cfg[parts * 2 - 2 + (back != 0)];
  if (!ready) { if ((rc = smem_attr(kernel, bytes))) return rc; ready = true; }
  kernel<<<dim3(H * parts, B), parts == 1 ? 672 : 640, bytes, st>>>(tb, tv, to, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_ssd_states launch");
}

// mode 0: bc = B rows, v = x -> chunk end states and gamma.  mode 1: bc = C rows, v = dy -> G.
// bc: [B, T, N] with token stride ld_bc; v: [B, T, H, P] with token stride ld_v (elements).
extern "C" int nsa_ssd_chunk_state(int mode, const void* bc, long ld_bc, const void* v, long ld_v, const float* dt,
                                   const float* A, float* S_out, float* gamma_out, int B, int T, int H, int N, int P,
                                   cudaStream_t st) {
  int rc = check_dims(N, P, ld_bc, ld_v);
  if (rc) return rc;
  CUtensorMap tb, tv;
  if ((rc = map_bc(&tb, bc, B, T, ld_bc))) return rc;
  if ((rc = map_v(&tv, v, B, T, H, ld_v))) return rc;
  SsdParams p{};
  p.dt = dt; p.A = A; p.B = B; p.T = T; p.H = H; p.nc = (T + L - 1) / L;
  p.S_out = S_out; p.gamma_out = gamma_out; p.status = nsa::status_ptr();
  const int smem = 3 * BOXB + 1024 + 2048;
  if (mode == 0) {
    static bool cfg = false;
    if (!cfg) { if ((rc = smem_attr(ssd_chunk_state_kernel<0>, smem))) return rc; cfg = true; }
    each_slab(p, [&](dim3 grid) { ssd_chunk_state_kernel<0><<<grid, 128, smem, st>>>(tb, tv, p); });
  } else {
    static bool cfg = false;
    if (!cfg) { if ((rc = smem_attr(ssd_chunk_state_kernel<1>, smem))) return rc; cfg = true; }
    each_slab(p, [&](dim3 grid) { ssd_chunk_state_kernel<1><<<grid, 128, smem, st>>>(tb, tv, p); });
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_ssd_chunk_state launch");
}

// y [B, T, H, P] contiguous.  Hprev_bf16: [B, nc, H, N, P] bf16.
extern "C" int nsa_ssd_chunk_out(const void* Cm, long ld_c, const void* Bm, long ld_b, const void* x, long ld_x,
                                 const void* Hprev_bf16, const float* dt, const float* A, const float* Dskip, void* y,
                                 int B, int T, int H, int N, int P, cudaStream_t st) {
  int rc = check_dims(N, P, ld_c | ld_b, ld_x);
  if (rc) return rc;
  const int nc = (T + L - 1) / L;
  CUtensorMap tc, tb, tx, th, ty;
  if ((rc = map_bc(&tc, Cm, B, T, ld_c))) return rc;
  if ((rc = map_bc(&tb, Bm, B, T, ld_b))) return rc;
  if ((rc = map_v(&tx, x, B, T, H, ld_x))) return rc;
  if ((rc = map_state(&th, Hprev_bf16, static_cast<long>(B) * nc * H * NS))) return rc;
  SsdParams p{};
  p.dt = dt; p.A = A; p.Dskip = Dskip; p.B = B; p.T = T; p.H = H; p.nc = nc;
  p.status = nsa::status_ptr();
  static bool cfg = false;
  if (!cfg) { if ((rc = smem_attr(ssd_chunk_out_kernel, OUT_SMEM))) return rc; cfg = true; }
  if ((rc = map_v(&ty, y, B, T, H, static_cast<long>(H) * PD))) return rc;
  ssd_chunk_out_kernel<<<deal_items(p), 608, OUT_SMEM, st>>>(tc, tb, tx, th, ty, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_ssd_chunk_out launch");
}

// dx [B, T, H, P]; dB_part, dC_part [B, T, nsa_ssd_grad_slots, N] fp32; q_out, k_out and r_out (or null) fp32 [B, T, H]: dy . (y - D x),
// x . (dx - D dy) and dy . x per token and head.
extern "C" int nsa_ssd_chunk_grad(const void* Cm, long ld_c, const void* Bm, long ld_b, const void* x, long ld_x,
                                  const void* dy, const void* Hprev_bf16, const void* dHn_bf16, const float* dt, const float* A,
                                  const float* Dskip, void* dx, float* dB_part, float* dC_part, float* q_out, float* k_out,
                                  float* r_out, int B, int T, int H, int N, int P, cudaStream_t st) {
  int rc = check_dims(N, P, ld_c | ld_b, ld_x);
  if (rc) return rc;
  const int nc = (T + L - 1) / L;
  const long rows = static_cast<long>(B) * nc * H * NS;
  CUtensorMap tc, tb, tx, tdy, th, tdh, tdx;
  if ((rc = map_bc(&tc, Cm, B, T, ld_c))) return rc;
  if ((rc = map_bc(&tb, Bm, B, T, ld_b))) return rc;
  if ((rc = map_v(&tx, x, B, T, H, ld_x))) return rc;
  if ((rc = map_v(&tdy, dy, B, T, H, static_cast<long>(H) * PD))) return rc;
  if ((rc = map_state(&th, Hprev_bf16, rows))) return rc;
  if ((rc = map_state(&tdh, dHn_bf16, rows))) return rc;
  if ((rc = map_v(&tdx, dx, B, T, H, static_cast<long>(H) * PD))) return rc;
  SsdParams p{};
  p.dt = dt; p.A = A; p.Dskip = Dskip; p.B = B; p.T = T; p.H = H; p.nc = nc;
  p.dB_part = dB_part; p.dC_part = dC_part; p.q_out = q_out; p.k_out = k_out; p.r_out = r_out; p.status = nsa::status_ptr();
  p.slots = nsa_ssd_grad_slots(B, T, H);
  static bool cfg = false;
  if (!cfg) { if ((rc = smem_attr(ssd_chunk_grad_kernel, GRAD_SMEM))) return rc; cfg = true; }
  ssd_chunk_grad_kernel<<<deal_items(p), 544, GRAD_SMEM, st>>>(tc, tb, tx, tdy, th, tdh, tdx, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_ssd_chunk_grad launch");
}
