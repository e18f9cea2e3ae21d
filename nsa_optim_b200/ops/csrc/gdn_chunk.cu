// Gated DeltaNet: everything of the chunkwise gated delta rule that is local to a chunk of 64 tokens, one
// kernel in front of the sequential state kernels of gdn.cu and one behind their backward.
//
// With gc the cumulative log-decay inside the chunk, sq_i = scale e^gc_i, sk_i = e^(gc_last - gc_i):
//     A[i][j]  = beta_i (k_i . k_j) e^(gc_i - gc_j)   (j < i)         X = (I + A)^-1
//     Tu = X diag(beta), Tw = X diag(beta e^gc)                       u = Tu v, w = Tw k
//     qk[i][j] = scale (q_i . k_j) e^(gc_i - gc_j)    (j <= i)
// q, k, v and the gates are read token-major as the caller has them, gradients leave the same way.
#include "f32x2.cuh"
#include "host.cuh"
#include "mma16.cuh"
#include "tc5.cuh"

namespace {
using namespace mma16;
constexpr int CH = 64, KD = 128;
constexpr int PK = KD + 8, PC = CH + 8;          // tile pitches (elements)
constexpr int PX = 68;                           // pitch of the fp32 64 x 64 tiles: rows 16-byte aligned, spread over the banks

// Per-chunk gate quantities: the CTA's first warp does the work, two tokens a lane; the caller synchronises.
// gs: cumulative log-decay, bs: beta.
__device__ __forceinline__ void load_gates(const float* g, const float* beta, long tok0, int T, int t0, int H, float* gs, float* bs) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    const int ta = t0 + 2 * lane, tb = ta + 1;
    const float a = ta < T ? g[tok0 + static_cast<long>(ta) * H] : 0.f, b = tb < T ? g[tok0 + static_cast<long>(tb) * H] : 0.f;
    bs[2 * lane] = ta < T ? beta[tok0 + static_cast<long>(ta) * H] : 0.f;
    bs[2 * lane + 1] = tb < T ? beta[tok0 + static_cast<long>(tb) * H] : 0.f;
    float s = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += n;
    }
    gs[2 * lane] = s - b;
    gs[2 * lane + 1] = s;
  }
}

struct PrepParams {
  const bf16 *q, *k, *v;       // [B, T, H, .]
  const float *g, *beta;       // [B, T, H]
  bf16 *w, *u, *qk;            // [BH, NC, 64, 128 / V / 64]
  float *X, *gc;               // [BH, NC, 64, 64] or null, [BH, NC, 64]
  int T, H, NC, V;
  float scale;
};

// One CTA of eight warps per (chunk, head).  What bounds it is its chain of phases, not the memory traffic of q, k, v, u, w (2 KB
// per token and head, 87 us at the copy rate for 16384 tokens x 16 heads), so three CTAs share an SM (70 KB each, for every width of
// the values): v passes through in pieces of 128 columns, over q and X, which are through by then, and Tu and Tw
// take the place of A.  16384 tokens x 16 heads, values 256 wide: 283 us with one CTA per SM, 198 with two (101 KB, all of v at once), 170
// with three, 165 without asking for the next chunk's inputs in L2.  The triangular inverse is the longest dependent phase and runs as
// two 32-column substitutions side by side, joined by two 32 x 32 products over all threads.
__global__ void __launch_bounds__(256, 3) gdn_prep_kernel(const PrepParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int V = p.V;
  bf16* sK = reinterpret_cast<bf16*>(smem_raw);            // rows 0..63 k, 64..127 q
  float* As = reinterpret_cast<float*>(sK + 2 * CH * PK);  // [64][PX]
  bf16* sTu = reinterpret_cast<bf16*>(As);                 // Tu and Tw over A once its inverse is known
  bf16* sTw = sTu + CH * PC;
  float* Xs = reinterpret_cast<float*>(sTw + CH * PC);     // [64][PX]
  float* gs = Xs + CH * PX;
  float* bs = gs + CH;
  // 128 columns of v: over q once q k^T is done, over X once Tu and Tw are
  auto piece = [&](int i) { return i & 1 ? reinterpret_cast<bf16*>(Xs) : sK + CH * PK; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, h = bh % p.H, b = bh / p.H, c = blockIdx.z * gridDim.y + blockIdx.y;   // see chunk_grid
  if (c >= p.NC) return;
  const int t0 = c * CH;
  const long tok0 = static_cast<long>(b) * p.T * p.H + h;  // (b, t, h) = tok0 + t * H
  for (int i = tid; i < CH * (KD / 8); i += 256) {
    const int r = i / (KD / 8), cc = (i % (KD / 8)) * 8, t = t0 + r;
    const bool ok = t < p.T;
    const long off = (tok0 + static_cast<long>(ok ? t : 0) * p.H) * KD + cc;
    cp_async16(sK + r * PK + cc, p.k + off, ok);
    cp_async16(sK + (CH + r) * PK + cc, p.q + off, ok);
  }
  cp_async_commit();
  auto load_v = [&](int i) {                               // piece i
    const int c8 = min(16, (V - 128 * i) / 8), shift = c8 == 16 ? 4 : 3;   // 16-byte columns: 16 or 8
    for (int e = tid; e < CH * c8; e += 256) {
      const int r = e >> shift, cc = (e & (c8 - 1)) * 8, t = t0 + r;
      const bool ok = t < p.T;
      cp_async16(piece(i) + r * PK + cc, p.v + (tok0 + static_cast<long>(ok ? t : 0) * p.H) * V + 128 * i + cc, ok);
    }
    cp_async_commit();
  };
  load_gates(p.g, p.beta, tok0, p.T, t0, p.H, gs, bs);
  cp_async_wait<0>();
  __syncthreads();
  const long chunk = static_cast<long>(bh) * p.NC + c;
  if (tid < CH) p.gc[chunk * CH + tid] = gs[tid];
  // ---- [k ; q] k^T: warp w owns rows 16 w .. of the stacked 128
  {
    float acc[8][4] = {};
#pragma unroll
    for (int kk = 0; kk < KD; kk += 16) {
      uint32_t a[4];
      load_a(a, sK, PK, warp * 16, kk);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t bb[4];
        load_b(bb, sK, PK, n * 16, kk);
        mma2(acc[2 * n], acc[2 * n + 1], a, bb);
      }
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = (warp & 3) * 16 + (lane >> 2) + 8 * hh;
      const float gi = gs[i], bi = bs[i];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int j = n * 8 + 2 * (lane & 3);
        // the exponent is zero where the entry is masked, so nothing overflows (loads first: a load under a condition is a branch)
        const float2 gj = *reinterpret_cast<const float2*>(gs + j);
        const float e0 = __expf(j <= i ? gi - gj.x : 0.f), e1 = __expf(j + 1 <= i ? gi - gj.y : 0.f);
        const float x0 = acc[n][2 * hh] * e0, x1 = acc[n][2 * hh + 1] * e1;
        if (warp < 4) {
          *reinterpret_cast<float2*>(As + i * PX + j) = make_float2(j < i ? bi * x0 : 0.f, j + 1 < i ? bi * x1 : 0.f);
        } else {
          *reinterpret_cast<uint32_t*>(p.qk + (chunk * CH + i) * CH + j) =
              pack2(j <= i ? p.scale * x0 : 0.f, j + 1 <= i ? p.scale * x1 : 0.f);
        }
      }
    }
  }
  __syncthreads();
  load_v(0);
  // ---- X = (I + A)^-1.  Diagonal 32 x 32 blocks: thread (block, column) substitutes forward
  if (warp < 2) {
    const float* Ad = As + warp * 32 * PX + warp * 32;
    float x[32];
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      float s[4] = {r == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < r; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(Ad + r * PX + j);   // zero from column r on
        s[0] = fmaf(-a.x, x[j], s[0]);
        if (j + 1 < r) s[1] = fmaf(-a.y, x[j + 1], s[1]);
        if (j + 2 < r) s[2] = fmaf(-a.z, x[j + 2], s[2]);
        if (j + 3 < r) s[3] = fmaf(-a.w, x[j + 3], s[3]);
      }
      x[r] = (s[0] + s[1]) + (s[2] + s[3]);
    }
#pragma unroll
    for (int r = 0; r < 32; ++r) Xs[(warp * 32 + r) * PX + warp * 32 + lane] = x[r];
  } else if (warp < 4) {
    for (int r = (warp - 2) * 16; r < (warp - 2) * 16 + 16; ++r) Xs[r * PX + 32 + lane] = 0.f;
  }
  __syncthreads();
  // ---- X21 = -X22 (A21 X11); the product in the middle goes to the unused upper block of As
  {
    const int i = tid >> 3, c4 = (tid & 7) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
      const float a = As[(32 + i) * PX + j];
      const float4 x = *reinterpret_cast<const float4*>(Xs + j * PX + c4);
      s.x = fmaf(a, x.x, s.x); s.y = fmaf(a, x.y, s.y); s.z = fmaf(a, x.z, s.z); s.w = fmaf(a, x.w, s.w);
    }
    *reinterpret_cast<float4*>(As + i * PX + 32 + c4) = s;
    __syncthreads();
    s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
      const float a = Xs[(32 + i) * PX + 32 + j];
      const float4 m = *reinterpret_cast<const float4*>(As + j * PX + 32 + c4);
      s.x = fmaf(-a, m.x, s.x); s.y = fmaf(-a, m.y, s.y); s.z = fmaf(-a, m.z, s.z); s.w = fmaf(-a, m.w, s.w);
    }
    *reinterpret_cast<float4*>(Xs + (32 + i) * PX + c4) = s;
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int i = tid; i < CH * CH / 4; i += 256) {
    const int r = i / (CH / 4), j = (i % (CH / 4)) * 4;
    const float4 x = *reinterpret_cast<const float4*>(Xs + r * PX + j);
    if (p.X) *reinterpret_cast<float4*>(p.X + (chunk * CH + r) * CH + j) = x;
    const float u0 = x.x * bs[j], u1 = x.y * bs[j + 1], u2 = x.z * bs[j + 2], u3 = x.w * bs[j + 3];
    *reinterpret_cast<uint2*>(sTu + r * PC + j) = make_uint2(pack2(u0, u1), pack2(u2, u3));
    *reinterpret_cast<uint2*>(sTw + r * PC + j) = make_uint2(pack2(u0 * __expf(gs[j]), u1 * __expf(gs[j + 1])),
                                                             pack2(u2 * __expf(gs[j + 2]), u3 * __expf(gs[j + 3])));
  }
  __syncthreads();
  // ---- w = Tw k and u = Tu v, 128 columns at a time, 16 a warp, which is the only reader of its columns and puts the
  //      result in their place
  auto multiply = [&](const bf16* tm, bf16* src) {
    const int n0 = warp * 16;
    float acc[4][2][4] = {};
#pragma unroll
    for (int kk = 0; kk < CH; kk += 16) {
      uint32_t bb[4];
      load_b_t(bb, src, PK, n0, kk);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (kk > m * 16) continue;                 // the matrices are lower triangular
        uint32_t a[4];
        load_a(a, tm, PC, m * 16, kk);
        mma2(acc[m][0], acc[m][1], a, bb);
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          *reinterpret_cast<uint32_t*>(src + (m * 16 + (lane >> 2) + 8 * hh) * PK + n0 + n * 8 + 2 * (lane & 3)) =
              pack2(acc[m][n][2 * hh], acc[m][n][2 * hh + 1]);
  };
  const int pieces = (V + 127) / 128;
  if (pieces > 1) load_v(1);
  multiply(sTw, sK);
  for (int i = 0; i < pieces; ++i) {
    if (i > 0) {
      cp_async_wait<0>();
      __syncthreads();                             // the piece is there, and the one before has left
      if (i + 1 < pieces) load_v(i + 1);
    }
    const int c8 = min(16, (V - 128 * i) / 8), shift = c8 == 16 ? 4 : 3;
    bf16* src = piece(i);
    if (warp * 2 < c8) multiply(sTu, src);
    __syncthreads();
    for (int e = tid; e < CH * c8; e += 256) {
      const int r = e >> shift, cc = (e & (c8 - 1)) * 8;
      *reinterpret_cast<uint4*>(p.u + (chunk * CH + r) * V + 128 * i + cc) = *reinterpret_cast<const uint4*>(src + r * PK + cc);
    }
    if (i == 0)
      for (int e = tid; e < CH * (KD / 8); e += 256) {
        const int r = e / (KD / 8), cc = (e % (KD / 8)) * 8;
        *reinterpret_cast<uint4*>(p.w + (chunk * CH + r) * KD + cc) = *reinterpret_cast<const uint4*>(sK + r * PK + cc);
      }
  }
}

struct PostParams {
  const bf16 *q, *k;                    // [B, T, H, 128]
  const float* beta;                    // [B, T, H]
  const float *gc, *X;                  // [BH, NC, 64], [BH, NC, 64, 64]
  const float* dgamma;                  // [V / 64, BH, NC]: <state entering, gradient of the state leaving> per V tile
  bf16 *dq, *dk, *dv;                   // [B, T, H, .]
  float *dg, *dbeta;                    // [B, T, H]
  int B, T, H, NC, V;
  float scale;
  KernelStatus* status;
};

// Tiles of 64 value columns, 128-byte-swizzled as TMA writes them: [du ; do] and [v_new ; v] (128 rows each) in one of two
// places, S and dS in a third.
constexpr int TILE = 128 * 128;
constexpr int POST_A1 = 2 * TILE, POST_B = POST_A1 + 2 * CH * PK * 2;      // the tail's tiles of k and q fill the second place
constexpr int POST_TILES = POST_B + 2 * TILE;
constexpr int POST_RED = 16;                                               // rows of partial sums
constexpr int POST_SMEM = POST_TILES + CH * PC * 2 + (2 + POST_RED) * CH * 4 + 128 + 1024;
constexpr int FX = CH * CH * 4, FF = CH * KD * 4;                          // fp32 tiles of the tail, rows without padding
static_assert(POST_B % 1024 == 0 && 2 * TILE <= 2 * CH * PK * 2, "gdn post: swizzled tiles");
static_assert(2 * FX <= POST_A1 && CH * PC * 2 <= FX, "gdn post: X, dX and what takes their places");
static_assert(TILE + FX <= 2 * TILE && FF <= POST_A1 && FF <= 2 * TILE, "gdn post: dw, X^T dX, results");
static_assert(2 * (POST_SMEM + 1024) <= 228 * 1024, "gdn post: two CTAs per SM");

// Fragments of a swizzled tile.  A: rows m0.., reduction k0..; B: 16 columns n0.. from [n][k] or (_t) from [k][n].
__device__ __forceinline__ void ldsm4_swz(uint32_t (&r)[4], const uint8_t* tile, int row, int chunk) {
  ldsm4(r, reinterpret_cast<const bf16*>(tile + row * 128 + ((chunk ^ (row & 7)) << 4)));
}
__device__ __forceinline__ void load_a_swz(uint32_t (&r)[4], const uint8_t* tile, int m0, int k0) {
  const int l = threadIdx.x & 31;
  ldsm4_swz(r, tile, m0 + (l & 15), (k0 >> 3) + (l >> 4));
}
__device__ __forceinline__ void load_b_swz(uint32_t (&r)[4], const uint8_t* tile, int n0, int k0) {
  const int l = threadIdx.x & 31, i = l >> 3;
  ldsm4_swz(r, tile, n0 + (i >> 1) * 8 + (l & 7), (k0 >> 3) + (i & 1));
}
__device__ __forceinline__ void load_b_t_swz(uint32_t (&r)[4], const uint8_t* tile, int n0, int k0) {
  const int l = threadIdx.x & 31, i = l >> 3, row = k0 + (i & 1) * 8 + (l & 7), chunk = (n0 >> 3) + (i >> 1);
  ldsm4_t(r, reinterpret_cast<const bf16*>(tile + row * 128 + ((chunk ^ (row & 7)) << 4)));
}
// Element (r, c) of an fp32 tile of W columns: groups of four are spread over the banks by row.
template <int W>
__device__ __forceinline__ int spread(int r, int c) {
  return r * W + ((((c >> 2) ^ r) & 15) << 2) + (c & ~63) + (c & 3);
}
__device__ __forceinline__ float dot32(const float (&a)[32], const bf16* b) {
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 u = *reinterpret_cast<const uint4*>(b + 8 * j);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      s += a[8 * j + 2 * e] * f.x + a[8 * j + 2 * e + 1] * f.y;
    }
  }
  return s;
}
__device__ __forceinline__ void tmem_cols(uint32_t taddr, float (&out)[32]) {
  uint32_t a[32];
  tc5::tmem_ld_x32(taddr, a);
  tc5::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; ++j) out[j] = __uint_as_float(a[j]);
}

// One CTA of sixteen warps per (chunk, head), two per SM: every gradient of the chunk once du (of the sequential pass) and
// the two states are known.
//     dw = -du S^T, dqs = do S^T, dks = v_new dS^T, dqk = do v_new^T, dTu = du v^T, dTw = dw k^T
//     dX = (dTu + dTw e^gc) beta (columns), dA = -(X^T dX X^T), then through the definitions above.
// Of the products that sum over the value dimension, those with a state are two full tcgen05 tiles of the stacked operands,
// [du ; do] S^T and [v_new ; v] dS^T, accumulated in tensor memory (half of it per CTA) while slices of 64 value columns stream
// through; dqk and dTu, of which only the lower triangle counts, are warp products whose accumulators stay in the registers that
// the tail wants them in.  The rest are 64-row products in a chain of phases.  One CTA per SM left the SM idle in that chain (a
// chunk took 42000 cycles, a quarter of them issued an instruction), so two share it and each fills the other's waits: 112 KB
// hold three 32 KB places for the slices and every tile of the tail lies over them (fp32 tiles without padding, Tw^T as a row
// scaling of Tu^T), and 64-row products leave out the blocks above the diagonal.  What bounds it now is the shared-memory pipe, 70 %
// busy; asking for the next chunk's tiles in L2 ahead only delays this one's (462 us without, 485 with).  16384 tokens x 16 heads,
// values 256 wide: 637 us with one CTA per SM, 449 with two of sixteen warps at 64 registers, 455 with two of eight and one that copies and
// issues.  Per token and head 3.5 KB come in and 1 KB goes out, against 6 KB alone for the per-V-tile partials of dw, dq
// and dk that the sequential pass would otherwise write and re-read.
__global__ void __launch_bounds__(512, 2)
gdn_post_kernel(const __grid_constant__ CUtensorMap tm_du, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_vn, const __grid_constant__ CUtensorMap tm_v,
                const __grid_constant__ CUtensorMap tm_S, const __grid_constant__ CUtensorMap tm_dS, const PostParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  bf16* sTu = reinterpret_cast<bf16*>(tiles + POST_TILES);
  float* gs = reinterpret_cast<float*>(sTu + CH * PC);
  float* bs = gs + CH;
  float* red = bs + CH;                                    // [POST_RED][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(red + POST_RED * CH);
  uint64_t *full_a = bars, *used_a = bars + 2, *done = bars + 4, *full_b = bars + 6;   // [2] each, full_b one
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // the tail, over the slices: k and q over the second place while the last slice is in the first
  float* Xs = reinterpret_cast<float*>(tiles);
  float* sDX = reinterpret_cast<float*>(tiles + FX);
  bf16* sDQ = reinterpret_cast<bf16*>(tiles);              // d(q k^T), over X
  bf16* sDK = reinterpret_cast<bf16*>(tiles + FX);         // d(k k^T), over dX
  bf16* sK = reinterpret_cast<bf16*>(tiles + POST_A1);
  bf16* sQ = sK + CH * PK;
  uint8_t* sW = tiles + POST_B;                            // dw, two swizzled tiles of 64 columns
  float* sY = reinterpret_cast<float*>(tiles + POST_B + TILE);   // X^T dX, then dA
  float* sFQ = reinterpret_cast<float*>(tiles);            // [64][128] at the very end
  float* sFK = reinterpret_cast<float*>(tiles + POST_B);
  const int tid = threadIdx.x, warp = tc5::warp_index(), lane = tid & 31;
  const int bh = blockIdx.x, h = bh % p.H, b = bh / p.H, c = blockIdx.z * gridDim.y + blockIdx.y;   // see chunk_grid
  if (c >= p.NC) return;
  const int t0 = c * CH, V = p.V, nvt = V / CH;
  const long tok0 = static_cast<long>(b) * p.T * p.H + h;
  const long chunk = static_cast<long>(bh) * p.NC + c;
  auto place = [&](int s) { return (nvt - 1 - s) & 1; };   // the last slice is in the first place
  auto load_a_part = [&](int s) {                          // one thread
    uint8_t* d = tiles + place(s) * POST_A1;
    uint64_t* bar = full_a + place(s);
    const int row = static_cast<int>(chunk) * CH, x = s * CH;
    tc5::mbar_expect_tx(bar, 2 * TILE);
    tc5::tma_load_2d(d, &tm_du, bar, x, row);
    tc5::tma_load_4d(d + TILE / 2, &tm_do, bar, x, h, t0, b);
    tc5::tma_load_2d(d + TILE, &tm_vn, bar, x, row);
    tc5::tma_load_4d(d + TILE + TILE / 2, &tm_v, bar, x, h, t0, b);
  };
  auto load_b_part = [&](int s) {
    tc5::mbar_expect_tx(full_b, 2 * TILE);
    tc5::tma_load_2d(tiles + POST_B, &tm_S, full_b, s * CH, static_cast<int>(chunk) * KD);
    tc5::tma_load_2d(tiles + POST_B + TILE, &tm_dS, full_b, s * CH, static_cast<int>(chunk) * KD);
  };
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) { tc5::mbar_init(full_a + i, 1); tc5::mbar_init(used_a + i, 16); tc5::mbar_init(done + i, 1); }
    tc5::mbar_init(full_b, 1);
    tc5::fence_barrier_init();
    load_a_part(0);
    load_b_part(0);
    if (nvt > 1) load_a_part(1);
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 256); tc5::tmem_relinquish(); }
  const float4* xg = reinterpret_cast<const float4*>(p.X + chunk * CH * CH) + tid;
  const float4 x4[2] = {xg[0], xg[512]};                   // X, for Tu
  if (tid < CH) {
    gs[tid] = p.gc[chunk * CH + tid];
    bs[tid] = t0 + tid < p.T ? p.beta[tok0 + static_cast<long>(t0 + tid) * p.H] : 0.f;
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = (tid + i * 512) / (CH / 4), j = (tid & 15) * 4;
    *reinterpret_cast<uint2*>(sTu + r * PC + j) =
        make_uint2(pack2(x4[i].x * bs[j], x4[i].y * bs[j + 1]), pack2(x4[i].z * bs[j + 2], x4[i].w * bs[j + 3]));
  }
  __syncthreads();
  // fragment view of warp products: rows m0.., 32 (of 128) or 16 (of 64) columns
  const int m0 = (warp & 3) * 16, n32 = (warp >> 2) * 32, n16 = (warp >> 2) * 16;
  const int r0 = m0 + (lane >> 2), cl = 2 * (lane & 3);    // first row and column offset of this lane's accumulator elements
  const bool lower = n16 <= m0;                            // of a 64 x 64 product: not all above the diagonal
  // tensor-memory view: lane row (0..63 the upper operand of a stack, 64..127 the lower), 32 columns from n32
  const int row = (warp & 3) * 32 + lane, ri = row & 63;
  const bool upper = (warp & 3) < 2;
  const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + n32;
  constexpr uint32_t cWQ = 0, cKS = 128;                   // accumulator columns of the two products
  constexpr uint32_t idesc = tc5::make_idesc_bf16(128, 128, 0, 0);
  constexpr int ISSUER = 14;                               // copies and issues too: it has nothing of dTu and dqk
  auto wait = [&](uint64_t* bar, int use, int code) {
    return tc5::mbar_wait_warp(bar, use & 1, abort_flag, p.status, code);
  };
  float dtu[2][4] = {}, dqk[2][4] = {};                    // rows m0.., columns n16..
  {
    bf16* dv_row = p.dv + (tok0 + static_cast<long>(t0 + r0) * p.H) * V + n16 + cl;
    bool ok = true;
    for (int s = 0; s < nvt; ++s) {
      const uint8_t* st = tiles + place(s) * POST_A1;
      if (!(ok = wait(full_a + place(s), s >> 1, STATUS_TIMEOUT_SMEM_FULL))) break;
      if (warp == ISSUER) {
        if (!(ok = wait(full_b, s, STATUS_TIMEOUT_SMEM_FULL))) break;
        const bool lead = tc5::elect_one();                // converged warp, elected lane issues
        tc5::fence_after_sync();
        const uint32_t sa = tc5::smem_u32(st), sb = tc5::smem_u32(tiles + POST_B);
        const uint64_t uo = tc5::desc_kmajor(sa), nv = tc5::desc_kmajor(sa + TILE), S = tc5::desc_kmajor(sb), dS = tc5::desc_kmajor(sb + TILE);
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < CH / 16; ++kk) {
            const uint64_t off = static_cast<uint64_t>((kk * 32) >> 4);
            const uint32_t acc = s > 0 || kk > 0 ? 1u : 0u;
            tc5::mma_ss(tmem + cWQ, uo + off, S + off, idesc, acc);
            tc5::mma_ss(tmem + cKS, nv + off, dS + off, idesc, acc);
          }
          tc5::mma_commit(done + (s & 1));
        }
        __syncwarp();
        if (s + 1 < nvt) {                                 // the states' place is free once the MMAs are through
          if (!(ok = wait(done + (s & 1), s >> 1, STATUS_TIMEOUT_TMEM_FULL))) break;
          if (lead) load_b_part(s + 1);
          __syncwarp();
        }
      }
      // behind the MMAs: dTu += du v^T, dqk += do v_new^T
      if (lower) {
#pragma unroll
        for (int kk = 0; kk < CH; kk += 16) {
          uint32_t a[4], bb[4];
          load_a_swz(a, st, m0, kk);
          load_b_swz(bb, st + TILE + TILE / 2, n16, kk);
          mma2(dtu[0], dtu[1], a, bb);
          load_a_swz(a, st + TILE / 2, m0, kk);
          load_b_swz(bb, st + TILE, n16, kk);
          mma2(dqk[0], dqk[1], a, bb);
        }
      }
      if (s + 1 == nvt) {                                  // k and q into the place of the slice before
        if (s > 0 && !(ok = wait(used_a + 1, (s - 1) >> 1, STATUS_TIMEOUT_SMEM_EMPTY) &&
                            wait(done + ((s - 1) & 1), (s - 1) >> 1, STATUS_TIMEOUT_TMEM_FULL))) break;
#pragma unroll
        for (int i = tid; i < CH * (KD / 8); i += 512) {
          const int r = i / (KD / 8), cc = (i % (KD / 8)) * 8, t = t0 + r;
          const bool in = t < p.T;
          const long off = (tok0 + static_cast<long>(in ? t : 0) * p.H) * KD + cc;
          cp_async16(sK + r * PK + cc, p.k + off, in);
          cp_async16(sQ + r * PK + cc, p.q + off, in);
        }
        cp_async_commit();
      }
      // dv of this slice: Tu^T du (row j needs i >= j only)
      float dv[2][4] = {};
#pragma unroll
      for (int q = 0; q < CH / 16; ++q) {
        if (q * 16 < m0) continue;
        uint32_t a[4], bb[4];
        load_a_t(a, sTu, PC, m0, q * 16);
        load_b_t_swz(bb, st, n16, q * 16);
        mma2(dv[0], dv[1], a, bb);
      }
      if (s + 1 < nvt) tc5::arrive_warp(used_a + place(s));
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
        if (t0 + r0 + 8 * hh < p.T)
#pragma unroll
          for (int n = 0; n < 2; ++n)
            *reinterpret_cast<uint32_t*>(dv_row + static_cast<long>(8 * hh) * p.H * V + s * CH + n * 8) = pack2(dv[n][2 * hh], dv[n][2 * hh + 1]);
      if (warp == ISSUER && s + 2 < nvt) {                 // its MMAs are through, see above
        if (!(ok = wait(used_a + place(s), s >> 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
        if (tc5::elect_one()) load_a_part(s + 2);
        __syncwarp();
      }
    }
    // the last commit covers every product
    if (ok) ok = wait(done + ((nvt - 1) & 1), (nvt - 1) >> 1, STATUS_TIMEOUT_TMEM_FULL);
    cp_async_wait<0>();
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {                                      // slices may still be in flight
        tc5::mbar_drain(full_a);
        tc5::mbar_drain(full_a + 1);
        tc5::mbar_drain(full_b);
      }
      __syncthreads();
      if (warp == 0) tc5::tmem_dealloc(tmem, 256);
      return;
    }
  }
  tc5::fence_after_sync();
#pragma unroll
  for (int i = tid; i < CH * CH / 4; i += 512) {
    const int r = i / (CH / 4), j = (i % (CH / 4)) * 4;
    cp_async16(Xs + spread<CH>(r, j), p.X + (chunk * CH + r) * CH + j, true);
  }
  cp_async_commit();
  const float g_last = gs[CH - 1];
  // ---- out of tensor memory: dw as an operand and the row sums q . dqs and k . dks (gates that scale rows of q and k);
  //      dqs and dks stay where they are until the end
  {
    float a[32], dot;
    tmem_cols(trow + cWQ, a);
    if (upper) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(sW + (n32 >> 6) * (TILE / 2) + ri * 128 + ((((n32 & 63) / 8 + j) ^ (ri & 7)) << 4)) =
            make_uint4(pack2(-a[8 * j], -a[8 * j + 1]), pack2(-a[8 * j + 2], -a[8 * j + 3]), pack2(-a[8 * j + 4], -a[8 * j + 5]),
                       pack2(-a[8 * j + 6], -a[8 * j + 7]));
      tmem_cols(trow + cKS, a);
      dot = dot32(a, sK + ri * PK + n32);
    } else {
      dot = dot32(a, sQ + ri * PK + n32);
    }
    red[((upper ? 4 : 0) + (warp >> 2)) * CH + ri] = dot;
  }
  cp_async_wait<0>();
  __syncthreads();
  // gradient of gc_i and beta_i, collected by thread i < 64
  float dgc = 0.f, dbeta = 0.f, dlast = 0.f;
  if (tid < CH) {
    float a = 0.f, k_ = 0.f;
#pragma unroll
    for (int n = 0; n < 4; ++n) { a += red[n * CH + tid]; k_ += red[(4 + n) * CH + tid]; }
    dlast = __expf(g_last - gs[tid]) * k_;
    dgc = p.scale * __expf(gs[tid]) * a - dlast;
  }
  // ---- dTw = dw k^T, dX
  {
    float aw[2][4] = {};
    if (lower) {
#pragma unroll
      for (int kk = 0; kk < KD; kk += 16) {
        uint32_t a[4], bb[4];
        load_a_swz(a, sW + (kk >> 6) * (TILE / 2), m0, kk & 63);
        load_b(bb, sK, PK, n16, kk);
        mma2(aw[0], aw[1], a, bb);
      }
    }
    float* part = red + 8 * CH;                            // sums of beta and gc, per 16 rows
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = n16 + n * 8 + cl + e;
        const float eg = __expf(gs[j]), bj = bs[j];
        float cb = 0.f, cg = 0.f;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int i = r0 + 8 * hh;
          const float x = Xs[spread<CH>(i, j)], tw = aw[n][2 * hh + e] * eg, d = dtu[n][2 * hh + e] + tw;
          sDX[spread<CH>(i, j)] = j <= i ? d * bj : 0.f;
          cb += d * x;                                     // x is zero above the diagonal
          cg += tw * x;
        }
        cg *= bj;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          cb += __shfl_xor_sync(0xffffffffu, cb, o);
          cg += __shfl_xor_sync(0xffffffffu, cg, o);
        }
        if (lane < 4) {
          part[(warp & 3) * CH + j] = cb;
          part[(4 + (warp & 3)) * CH + j] = cg;
        }
      }
  }
  __syncthreads();
  if (tid < CH)
#pragma unroll
    for (int n = 0; n < 4; ++n) { dbeta += red[(8 + n) * CH + tid]; dgc += red[(12 + n) * CH + tid]; }
  // ---- dA = -(X^T dX X^T) below the diagonal, fp32.  Warp w owns rows a = 4 w .. 4 w + 3 of y = X^T dX and of dA, so there is
  //      no barrier in between.  y[a][c] is wanted for c < a only and its sum starts at i = a: the warps of the upper half, whose
  //      sums are long and rows short, give half of the sum to the lanes that would have the other columns.
  {
    const int a0 = warp * 4;
    {
      const bool split = warp < 8;
      const int cc = (split ? lane & 15 : lane) * 2;
      const int len = split ? (CH - a0) / 2 : CH - a0, from = a0 + (split ? (lane >> 4) * len : 0);
      float2 y[2][2] = {};                                 // rows a0, a0 + 1 and a0 + 2, a0 + 3; two columns
#pragma unroll 4
      for (int i = from; i < from + len; ++i) {            // X[i][a] is zero for i < a
        const float4 x = *reinterpret_cast<const float4*>(Xs + spread<CH>(i, a0));
        const float2 d = *reinterpret_cast<const float2*>(sDX + spread<CH>(i, cc));
        const float2 d0 = make_float2(d.x, d.x), d1 = make_float2(d.y, d.y);
        y[0][0] = fma2(make_float2(x.x, x.y), d0, y[0][0]);
        y[0][1] = fma2(make_float2(x.x, x.y), d1, y[0][1]);
        y[1][0] = fma2(make_float2(x.z, x.w), d0, y[1][0]);
        y[1][1] = fma2(make_float2(x.z, x.w), d1, y[1][1]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (split) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            y[e][k].x += __shfl_xor_sync(0xffffffffu, y[e][k].x, 16);
            y[e][k].y += __shfl_xor_sync(0xffffffffu, y[e][k].y, 16);
          }
        }
        if (!split || lane < 16) {
          *reinterpret_cast<float2*>(sY + spread<CH>(a0 + 2 * e, cc)) = make_float2(y[e][0].x, y[e][1].x);
          *reinterpret_cast<float2*>(sY + spread<CH>(a0 + 2 * e + 1, cc)) = make_float2(y[e][0].y, y[e][1].y);
        }
      }
    }
    __syncwarp();
    float2 s[4][2] = {};                                   // even and odd j; columns b = lane and lane + 32
#pragma unroll 2
    for (int j = 0; j < a0 + 4; j += 4) {                  // X[b][j] is zero for j > b, and b < a
      float4 ya[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) ya[e] = *reinterpret_cast<const float4*>(sY + spread<CH>(a0 + e, j));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (32 * k > a0) continue;
        const float4 x = *reinterpret_cast<const float4*>(Xs + spread<CH>(lane + 32 * k, j));
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[e][k] = fma2(make_float2(ya[e].x, ya[e].y), make_float2(x.x, x.y), s[e][k]);
          s[e][k] = fma2(make_float2(ya[e].z, ya[e].w), make_float2(x.z, x.w), s[e][k]);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (32 * k <= a0) sY[spread<CH>(a0 + e, lane + 32 * k)] = -(s[e][k].x + s[e][k].y);
  }
  __syncthreads();                                         // X and dX are read
  // ---- through the definitions of A and qk
  {
    float kk_[2][4] = {}, qk_[2][4] = {};
    if (lower) {
#pragma unroll
      for (int kk = 0; kk < KD; kk += 16) {
        uint32_t a[4], bb[4];
        load_b(bb, sK, PK, n16, kk);
        load_a(a, sK, PK, m0, kk);
        mma2(kk_[0], kk_[1], a, bb);
        load_a(a, sQ, PK, m0, kk);
        mma2(qk_[0], qk_[1], a, bb);
      }
    }
    float col[2][2] = {};
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = r0 + 8 * hh;
      const float gi = gs[i], bi = bs[i];
      float rb = 0.f, rg = 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        float ok[2], oq[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = n16 + n * 8 + cl + e;
          const float gj = gs[j], da = sY[spread<CH>(i, j)];                   // loads first: a load under a condition is a branch
          const float ex = __expf(j <= i ? gi - gj : 0.f);
          const float d = j < i ? da : 0.f;
          const float araw = kk_[n][2 * hh + e] * ex;
          ok[e] = d * bi * ex;
          oq[e] = j <= i ? dqk[n][2 * hh + e] * p.scale * ex : 0.f;
          const float t = d * bi * araw + oq[e] * qk_[n][2 * hh + e];
          rb += d * araw;
          rg += t;
          col[n][e] -= t;
        }
        *reinterpret_cast<uint32_t*>(sDK + i * PC + n16 + n * 8 + cl) = pack2(ok[0], ok[1]);
        *reinterpret_cast<uint32_t*>(sDQ + i * PC + n16 + n * 8 + cl) = pack2(oq[0], oq[1]);
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        rb += __shfl_xor_sync(0xffffffffu, rb, o);
        rg += __shfl_xor_sync(0xffffffffu, rg, o);
      }
      if ((lane & 3) == 0) {
        red[(warp >> 2) * CH + i] = rb;
        red[(4 + (warp >> 2)) * CH + i] = rg;
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float s = col[n][e];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < 4) red[(8 + (warp & 3)) * CH + n16 + n * 8 + cl + e] = s;
      }
  }
  __syncthreads();
  if (tid < CH) {
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      dbeta += red[n * CH + tid];
      dgc += red[(4 + n) * CH + tid] + red[(8 + n) * CH + tid];
    }
    red[12 * CH + tid] = dgc;
    red[13 * CH + tid] = dlast;
    if (t0 + tid < p.T) p.dbeta[tok0 + static_cast<long>(t0 + tid) * p.H] = dbeta;
  }
  // ---- dq = sq dqs + dqkr k;  dk = sk dks + dkk k + dkk^T k + dqkr^T q + Tw^T dw,  Tw^T = diag(e^gc) Tu^T
  {
    float aQ[4][4] = {}, aK[4][4] = {};
#pragma unroll
    for (int kk = 0; kk < CH; kk += 16) {
      if (kk < m0) continue;                               // Tu is lower triangular
      uint32_t a[4], bb[4];
      load_a_t(a, sTu, PC, m0, kk);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        load_b_t_swz(bb, sW + (n32 >> 6) * (TILE / 2), (n32 & 63) + n * 16, kk);
        mma2(aK[2 * n], aK[2 * n + 1], a, bb);
      }
    }
    const float e0 = __expf(gs[r0]), e1 = __expf(gs[r0 + 8]);
#pragma unroll
    for (int n = 0; n < 4; ++n) { aK[n][0] *= e0; aK[n][1] *= e0; aK[n][2] *= e1; aK[n][3] *= e1; }
#pragma unroll
    for (int kk = 0; kk < CH; kk += 16) {                  // so are dkk and dqkr
      uint32_t a1[4], a2[4], bb[4];
      if (kk <= m0) {
        load_a(a1, sDQ, PC, m0, kk);
        load_a(a2, sDK, PC, m0, kk);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          load_b_t(bb, sK, PK, n32 + n * 16, kk);
          mma2(aQ[2 * n], aQ[2 * n + 1], a1, bb);
          mma2(aK[2 * n], aK[2 * n + 1], a2, bb);
        }
      }
      if (kk >= m0) {
        load_a_t(a1, sDK, PC, m0, kk);
        load_a_t(a2, sDQ, PC, m0, kk);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          load_b_t(bb, sK, PK, n32 + n * 16, kk);
          mma2(aK[2 * n], aK[2 * n + 1], a1, bb);
          load_b_t(bb, sQ, PK, n32 + n * 16, kk);
          mma2(aK[2 * n], aK[2 * n + 1], a2, bb);
        }
      }
    }
    __syncthreads();                                       // the operands are read
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int o = spread<KD>(r0 + 8 * hh, n32 + n * 8 + cl);
        *reinterpret_cast<float2*>(sFQ + o) = make_float2(aQ[n][2 * hh], aQ[n][2 * hh + 1]);
        *reinterpret_cast<float2*>(sFK + o) = make_float2(aK[n][2 * hh], aK[n][2 * hh + 1]);
      }
  }
  __syncthreads();                                         // the tiles of q and k become those of dq and dk
  {
    const float sc = upper ? __expf(g_last - gs[ri]) : p.scale * __expf(gs[ri]);
    const float* add = upper ? sFK : sFQ;
    bf16* dst = (upper ? sK : sQ) + ri * PK + n32;
    float a[32];
    tmem_cols(trow + (upper ? cKS : cWQ), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 f = *reinterpret_cast<const float4*>(add + spread<KD>(ri, n32 + 4 * j));
      *reinterpret_cast<uint2*>(dst + 4 * j) = make_uint2(pack2(sc * a[4 * j] + f.x, sc * a[4 * j + 1] + f.y),
                                                          pack2(sc * a[4 * j + 2] + f.z, sc * a[4 * j + 3] + f.w));
    }
  }
  // ---- d g_t: sum of d gc_i over i >= t; the chunk's last gc also carries the decay of the state and of k
  if (warp == 0) {
    float l2 = red[13 * CH + 2 * lane] + red[13 * CH + 2 * lane + 1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l2 += __shfl_xor_sync(0xffffffffu, l2, o);
    float dgam = 0.f;
    for (int s = 0; s < nvt; ++s) dgam += p.dgamma[(static_cast<long>(s) * gridDim.x + bh) * p.NC + c];
    l2 += dgam * __expf(g_last);
    const float a = red[12 * CH + 2 * lane], bq = red[12 * CH + 2 * lane + 1] + (lane == 31 ? l2 : 0.f);
    float s = a + bq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_down_sync(0xffffffffu, s, o);
      if (lane + o < 32) s += n;
    }
    const int ta = t0 + 2 * lane;
    if (ta < p.T) p.dg[tok0 + static_cast<long>(ta) * p.H] = s;
    if (ta + 1 < p.T) p.dg[tok0 + static_cast<long>(ta + 1) * p.H] = s - a;
  }
  tc5::fence_before_sync();
  __syncthreads();
  for (int i = tid; i < CH * (KD / 8); i += 512) {
    const int r = i / (KD / 8), cc = (i % (KD / 8)) * 8, t = t0 + r;
    if (t >= p.T) continue;
    const long off = (tok0 + static_cast<long>(t) * p.H) * KD + cc;
    *reinterpret_cast<uint4*>(p.dq + off) = *reinterpret_cast<const uint4*>(sQ + r * PK + cc);
    *reinterpret_cast<uint4*>(p.dk + off) = *reinterpret_cast<const uint4*>(sK + r * PK + cc);
  }
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 256); }
}
// One CTA per (chunk, head), heads fastest so that CTAs that run together touch neighbouring pieces of the same token rows.
// y ends at 65535 chunks (4.2 M tokens); longer sequences go on in z, whose last layer may reach past the end.
dim3 chunk_grid(int BH, int NC) { return dim3(BH, NC < 65535 ? NC : 65535, (NC + 65534) / 65535); }
}  // namespace

// q, k [B, T, H, 128], v [B, T, H, V] bf16 contiguous, g (log-decay) and beta [B, T, H] fp32 -> w, u, qk, gc and, where
// X is not null, the fp32 inverse the backward needs.  NC = ceil(T / 64).
extern "C" int nsa_gdn_prep(const void* q, const void* k, const void* v, const float* g, const float* beta, void* w, void* u,
                            void* qk, float* X, float* gc, int B, int T, int H, int K, int V, float scale, cudaStream_t st) {
  if (K != KD || V % 64 || V > 512) return nsa::fail(NSA_ERR_SHAPE, "gdn: key width must be 128, value width a multiple of 64 up to 512");
  const int NC = (T + CH - 1) / CH;
  PrepParams p{(const bf16*)q, (const bf16*)k, (const bf16*)v, g, beta, (bf16*)w, (bf16*)u, (bf16*)qk, X, gc, T, H, NC, V, scale};
  constexpr int smem = 2 * CH * PK * 2 + 2 * CH * PC * 2 + CH * PX * 4 + 2 * CH * 4;
  static_assert(3 * (smem + 1024) <= 228 * 1024 && CH * PX * 4 <= 2 * CH * PC * 2 && CH * PK * 2 <= CH * PX * 4, "gdn prep: three CTAs per SM, tiles");
  cudaError_t e = cudaFuncSetAttribute(gdn_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return nsa::fail_cuda(e, "gdn prep smem attribute");
  gdn_prep_kernel<<<chunk_grid(B * H, NC), 256, smem, st>>>(p);
  nsa::count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gdn_prep launch");
}

// d_o [B, T, H, V] bf16; du, v_new [B*H, NC, 64, V]; S, dS [B*H, NC, 128, V]; dgamma [V / 64, B*H, NC] -> dq, dk, dv, dg, dbeta.
extern "C" int nsa_gdn_post(const void* q, const void* k, const void* v, const void* d_o, const float* beta, const float* gc,
                            const float* X, const void* v_new, const void* du, const void* S, const void* dS,
                            const float* dgamma, void* dq, void* dk, void* dv, float* dg, float* dbeta, int B, int T, int H,
                            int K, int V, float scale, cudaStream_t st) {
  if (K != KD || V % 64) return nsa::fail(NSA_ERR_SHAPE, "gdn: key width must be 128 and value width a multiple of 64");
  const int NC = (T + CH - 1) / CH;
  const long chunks = static_cast<long>(B) * H * NC;
  CUtensorMap tdu, tdo, tvn, tv, tS, tdS;
  int rc;
  auto token_map = [&](CUtensorMap* m, const void* base) {
    const uint64_t dims[4] = {(uint64_t)V, (uint64_t)H, (uint64_t)T, (uint64_t)B};
    const uint64_t strides[3] = {(uint64_t)V * 2, (uint64_t)H * V * 2, (uint64_t)T * H * V * 2};
    const uint32_t box[4] = {64, 1, (uint32_t)CH, 1};
    return nsa::make_tmap_bf16(m, base, 4, dims, strides, box, 1);
  };
  if ((rc = nsa::make_tmap_2d_bf16(&tdu, du, V, chunks * CH, V, 64, CH))) return rc;
  if ((rc = token_map(&tdo, d_o))) return rc;
  if ((rc = nsa::make_tmap_2d_bf16(&tvn, v_new, V, chunks * CH, V, 64, CH))) return rc;
  if ((rc = token_map(&tv, v))) return rc;
  if ((rc = nsa::make_tmap_2d_bf16(&tS, S, V, chunks * KD, V, 64, KD))) return rc;
  if ((rc = nsa::make_tmap_2d_bf16(&tdS, dS, V, chunks * KD, V, 64, KD))) return rc;
  PostParams p{(const bf16*)q, (const bf16*)k, beta, gc, X, dgamma, (bf16*)dq, (bf16*)dk, (bf16*)dv, dg, dbeta, B, T, H, NC, V, scale,
               nsa::status_ptr()};
  cudaError_t e = cudaFuncSetAttribute(gdn_post_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, POST_SMEM);
  if (e != cudaSuccess) return nsa::fail_cuda(e, "gdn post smem attribute");
  gdn_post_kernel<<<chunk_grid(B * H, NC), 512, POST_SMEM, st>>>(tdu, tdo, tvn, tv, tS, tdS, p);
  nsa::count_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gdn_post launch");
}
