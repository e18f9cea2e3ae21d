// Gated DeltaNet: the sequential (inter-chunk) part of the chunkwise gated delta rule,
// forward and backward, on tcgen05 tensor cores with the K x V state resident in tensor
// memory.  Chunk length 64, key width 128, value width a multiple of 64.
//
// Per head, with S the K x V state entering chunk c (fp32), w (64 x K), u (64 x V), qk (64 x 64) and the
// cumulative log-decay gc from gdn_chunk.cu, and q, k as the caller has them:
//     v_new   = u - w S                 o = sq (q S) + qk v_new            sq_i = scale e^gc_i
//     S_next  = e^gc_last S + k^T (sk v_new)                               sk_i = e^(gc_last - gc_i)
// One CTA owns one (head, 64-wide V tile) and walks the chunks in order, two threads per accumulator row
// (half the conversions in the chain: 256 instead of 128 threads).  The loop is one dependent
// chain and there are fewer CTAs than SMs at the usual head counts, so its length is what a call
// takes: row scalings are applied to accumulator rows in registers instead of to operands, the
// output's part of a chunk (its second product, the read-back, the store) runs behind the
// next chunk's first product, and o leaves token-major.
//
// Backward walks the chunks in reverse with dS (K x 64 tile, gradient of the state leaving the chunk) in TMEM:
//     du      = qk^T do + sk (k dS)     dgamma = <S, dS>  (partial per V tile)
//     dS_prev = e^gc_last dS + q^T (sq do) - w^T du
// It stores dS per chunk; what only needs S and dS of one chunk (dw, dq, dk) is left to gdn_post_kernel.
#include "host.cuh"
#include "tc5.cuh"

namespace {
typedef __nv_bfloat16 bf16;
constexpr int KD = 128;   // key width
constexpr int VT = 64;    // V tile per CTA
constexpr int CH = 64;    // chunk length
constexpr int BOX = 8192; // bytes of one [64 rows][64 bf16] swizzled box

// A thread handles half a row: HC columns from column half * HC on.
constexpr int HC = 32;
__device__ __forceinline__ void write_half(uint8_t* tile, int row, int half, const uint32_t (&packed)[HC / 2]) {
#pragma unroll
  for (int j = 0; j < HC / 8; ++j) {
    const uint4 v = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
    *reinterpret_cast<uint4*>(tile + row * 128 + (((half * (HC / 8) + j) ^ (row & 7)) << 4)) = v;
  }
}
__device__ __forceinline__ void read_half(const uint8_t* tile, int row, int half, float (&out)[HC]) {
#pragma unroll
  for (int j = 0; j < HC / 8; ++j) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + row * 128 + (((half * (HC / 8) + j) ^ (row & 7)) << 4));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 f = __bfloat1622float2(h[k]);
      out[8 * j + 2 * k] = f.x;
      out[8 * j + 2 * k + 1] = f.y;
    }
  }
}
__device__ __forceinline__ void load_global(const bf16* src, uint32_t (&packed)[HC / 2]) {
  const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
  for (int j = 0; j < HC / 8; ++j) {
    const uint4 v = s4[j];
    packed[4 * j] = v.x; packed[4 * j + 1] = v.y; packed[4 * j + 2] = v.z; packed[4 * j + 3] = v.w;
  }
}
__device__ __forceinline__ void unpack_half(const uint32_t (&packed)[HC / 2], float (&out)[HC]) {
#pragma unroll
  for (int j = 0; j < HC / 2; ++j) {
    float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&packed[j]));
    out[2 * j] = f.x;
    out[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ void tmem_ld_half(uint32_t taddr, float (&out)[HC]) {
  uint32_t a[HC];
  tc5::tmem_ld_x32(taddr, a);
  tc5::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < HC; ++j) out[j] = __uint_as_float(a[j]);
}
__device__ __forceinline__ void tmem_st_half(uint32_t taddr, const float (&in)[HC]) {
  uint32_t a[HC];
#pragma unroll
  for (int j = 0; j < HC; ++j) a[j] = __float_as_uint(in[j]);
  tc5::tmem_st_x32(taddr, a);
  tc5::tmem_st_wait();
}
__device__ __forceinline__ void pack_half(const float (&in)[HC], uint32_t (&packed)[HC / 2]) {
#pragma unroll
  for (int j = 0; j < HC / 2; ++j) packed[j] = tc5::pack_bf16(in[2 * j], in[2 * j + 1]);
}

struct FwdParams {
  const bf16* u;        // [BH, NC, 64, V]
  const float* gc;      // [BH, NC, 64]
  int store_states;     // also write v_new and S_all (the backward needs them)
  int NC, V, H;
  float scale;
  KernelStatus* status;
};

// stage: k-block kb of [w ; q] (2 x 16 KB), k (16 KB), [0 ; qk] (16 KB, first half zero)
constexpr int FWD_STAGE = 8 * BOX;
constexpr int FWD_TX = 7 * BOX;                                                       // bytes that arrive per chunk
constexpr int FWD_SMEM = 2 * FWD_STAGE + 2 * BOX /*Sb*/ + 2 * BOX /*Vb, Vs*/ + BOX /*Ob*/ + 1024 + 128;

__global__ void __launch_bounds__(256, 1)
gdn_seq_fwd_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_qk,
                   const __grid_constant__ CUtensorMap tm_vn, const __grid_constant__ CUtensorMap tm_o,
                   const __grid_constant__ CUtensorMap tm_sa, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* Sb = smem + 2 * FWD_STAGE;           // [KD rows][64] bf16 state, B operand
  uint8_t* Vb = Sb + 2 * BOX;                   // [64 rows][64] v_new
  uint8_t* Vs = Vb + BOX;                       // [64 rows][64] sk v_new
  uint8_t* Ob = Vs + BOX;                       // [64 rows][64] o on its way out
  uint64_t* bars = reinterpret_cast<uint64_t*>(Ob + BOX);
  uint64_t* full = bars;        // [2]
  uint64_t* m1 = bars + 2;
  uint64_t* m2 = bars + 3;
  uint64_t* m3 = bars + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int r = threadIdx.x & 127, half = threadIdx.x >> 7;   // TMEM lane / tile row, half of its columns
  const int warp = threadIdx.x >> 5;
  const bool boss = threadIdx.x == 0;
  const int vt = blockIdx.x, bh = blockIdx.y, h = bh % p.H, b = bh / p.H;
  const int NC = p.NC, V = p.V;

  if (boss) {
    *abort_flag = 0;
    tc5::mbar_init(&full[0], 1);
    tc5::mbar_init(&full[1], 1);
    tc5::mbar_init(m1, 1);
    tc5::mbar_init(m2, 1);
    tc5::mbar_init(m3, 1);
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 256); tc5::tmem_relinquish(); }
  // S = 0: bf16 mirror in shared memory; the constant zero half of both [0 ; qk] operands
  {
    uint32_t z[HC / 2];
#pragma unroll
    for (int j = 0; j < HC / 2; ++j) z[j] = 0u;
    write_half(Sb, r, half, z);
    write_half(smem + (r >> 6) * FWD_STAGE + 6 * BOX, r & 63, half, z);
  }
  tc5::fence_proxy_async();
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_off = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * HC;   // lanes and columns of this thread
  // TMEM columns: D1 = [w ; q] S [0, 64)   S [64, 128)   D2 = [0 ; qk] v_new [128, 192)
  const uint32_t cD1 = 0, cS = 64, cD2 = 128;
  {
    float z[HC];
#pragma unroll
    for (int j = 0; j < HC; ++j) z[j] = 0.f;
    tmem_st_half(tmem + lane_off + cS, z);
  }
  tc5::fence_before_sync();
  __syncthreads();
  // Outputs leave as TMA stores from the swizzled tiles they are in anyway.  Thread 0 stores v_new and the
  // state, thread 64 the output; each waits until its earlier store has read a tile before that tile is
  // rewritten.  Chunk 0 enters with the zero state that Sb holds now.
  if (boss && p.store_states) {
    tc5::tma_store_2d(&tm_sa, Sb, vt * VT, bh * NC * KD);
    tc5::tma_store_commit();
  }

  auto issue_loads = [&](int c) {
    const int s = c & 1;
    uint8_t* st = smem + s * FWD_STAGE;
    const int row0 = (bh * NC + c) * CH;
    tc5::mbar_expect_tx(&full[s], FWD_TX);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tc5::tma_load_2d(st + kb * 2 * BOX, &tm_w, &full[s], kb * 64, row0);
      tc5::tma_load_4d(st + kb * 2 * BOX + BOX, &tm_q, &full[s], kb * 64, h, c * CH, b);
      tc5::tma_load_4d(st + 4 * BOX + kb * BOX, &tm_k, &full[s], kb * 64, h, c * CH, b);
    }
    tc5::tma_load_2d(st + 7 * BOX, &tm_qk, &full[s], 0, row0);
  };
  if (boss) issue_loads(0);

  constexpr uint32_t idesc1 = tc5::make_idesc_bf16(128, VT, 0, 1);   // A K-major, B MN-major
  constexpr uint32_t idesc2 = tc5::make_idesc_bf16(128, VT, 1, 1);   // A MN-major (k^T), B MN-major
  bool ok = true;
  // Global loads of the chain (u row, gates) are fetched one chunk ahead.
  const float* gc = p.gc + static_cast<long>(bh) * NC * CH;
  uint32_t upk_next[HC / 2];
#pragma unroll
  for (int j = 0; j < HC / 2; ++j) upk_next[j] = 0u;
  if (r < CH) load_global(p.u + (static_cast<long>(bh * NC) * CH + r) * V + vt * VT + half * HC, upk_next);
  float gr_next = gc[r & 63], gl_next = gc[CH - 1];
  float oi[HC];                                    // sq (q S) of the chunk whose output is still open (rows 64..127)
  // Output of chunk c: D2 joins oi; runs while the tensor core works on chunk c + 1.
  auto finish_output = [&](int c) {
    if (!tc5::mbar_wait(m3, c & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) ok = false;
    __syncwarp();
    tc5::fence_after_sync();
    if (r < CH) return;                            // the other warps stay together, also after a wait that gave up
    float d2[HC];
    tmem_ld_half(tmem + lane_off + cD2, d2);
#pragma unroll
    for (int j = 0; j < HC; ++j) d2[j] += oi[j];
    uint32_t pk[HC / 2];
    pack_half(d2, pk);
    if (threadIdx.x == CH) tc5::tma_store_wait_read<0>();    // the previous output tile has been read
    asm volatile("bar.sync 1, 128;" ::: "memory");
    write_half(Ob, r - CH, half, pk);
    tc5::fence_proxy_async();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (threadIdx.x == CH && ok) {                           // rows past T are clipped by the copy engine
      tc5::tma_store_4d(&tm_o, Ob, vt * VT, h, c * CH, b);
      tc5::tma_store_commit();
    }
  };
  for (int c = 0; c < NC && ok; ++c) {
    const int s = c & 1;
    uint8_t* st = smem + s * FWD_STAGE;
    const long row0 = static_cast<long>(bh * NC + c) * CH;
    uint32_t upk[HC / 2];
#pragma unroll
    for (int j = 0; j < HC / 2; ++j) upk[j] = upk_next[j];
    const float g_row = gr_next, g_last = gl_next;
    if (warp == 0) {
      // The issuing warp stays converged and one elected lane issues: descriptors then live in
      // uniform registers and an MMA costs the issuing thread a few cycles instead of 70 to 100,
      // which matters in a loop that is one dependent chain.
      const bool lead = tc5::elect_one();
      if (__all_sync(0xffffffffu, tc5::mbar_wait(&full[s], (c >> 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_SMEM_FULL))) {
        tc5::fence_after_sync();
        const uint64_t a1 = tc5::desc_kmajor(tc5::smem_u32(st)), sb = tc5::desc_mnmajor(tc5::smem_u32(Sb), BOX);
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < KD / 16; ++kk)
            tc5::mma_ss(tmem + cD1, a1 + static_cast<uint64_t>(((kk >> 2) * 2 * BOX + (kk & 3) * 32) >> 4),
                        sb + static_cast<uint64_t>((kk * 2048) >> 4), idesc1, kk > 0 ? 1u : 0u);
          tc5::mma_commit(m1);
        }
      }
      __syncwarp();
    }
    // next chunk's u row (rows 0..63 only) and gates, in flight while this chunk computes
    if (c + 1 < NC) {
      if (r < CH) load_global(p.u + (row0 + CH + r) * V + vt * VT + half * HC, upk_next);
      gr_next = gc[(c + 1) * CH + (r & 63)];
      gl_next = gc[(c + 1) * CH + CH - 1];
    }
    if (c > 0) finish_output(c - 1);
    // the stage of chunk c + 1 was last read by chunk c - 1's second group of MMAs, complete since finish_output
    if (boss && ok && c + 1 < NC) issue_loads(c + 1);
    if (boss) tc5::tma_store_wait_read<1>();     // the previous v_new tile has been read
    if (ok && !tc5::mbar_wait(m1, c & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) { ok = false; }
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc5::fence_after_sync();
    {
      float d1[HC];
      tmem_ld_half(tmem + lane_off + cD1, d1);
      if (r < CH) {
        float uf[HC];
        unpack_half(upk, uf);
        const float sk = __expf(g_last - g_row);
        uint32_t pk[HC / 2], ps[HC / 2];
#pragma unroll
        for (int j = 0; j < HC; ++j) d1[j] = uf[j] - d1[j];
        pack_half(d1, pk);
#pragma unroll
        for (int j = 0; j < HC; ++j) d1[j] *= sk;
        pack_half(d1, ps);
        write_half(Vb, r, half, pk);
        write_half(Vs, r, half, ps);
      } else {
        const float sq = p.scale * __expf(g_row);
#pragma unroll
        for (int j = 0; j < HC; ++j) oi[j] = sq * d1[j];
      }
    }
    tc5::fence_proxy_async();
    tc5::fence_before_sync();
    __syncthreads();
    if (boss && p.store_states) {
      tc5::tma_store_2d(&tm_vn, Vb, vt * VT, static_cast<int>(row0));
      tc5::tma_store_commit();
    }
    if (warp == 0) {
      const bool lead = tc5::elect_one();
      tc5::fence_after_sync();
      const uint64_t kt = tc5::desc_mnmajor(tc5::smem_u32(st + 4 * BOX), BOX), vs = tc5::desc_mnmajor(tc5::smem_u32(Vs), BOX);
      const uint64_t qk = tc5::desc_kmajor(tc5::smem_u32(st + 6 * BOX)), vb = tc5::desc_mnmajor(tc5::smem_u32(Vb), BOX);
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)       // S += k^T (sk v_new)
          tc5::mma_ss(tmem + cS, kt + static_cast<uint64_t>((kk * 2048) >> 4), vs + static_cast<uint64_t>((kk * 2048) >> 4), idesc2, 1u);
        tc5::mma_commit(m2);
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)       // D2 = [0 ; qk] v_new
          tc5::mma_ss(tmem + cD2, qk + static_cast<uint64_t>((kk * 32) >> 4), vb + static_cast<uint64_t>((kk * 2048) >> 4), idesc1, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m3);
      }
      __syncwarp();
    }
    if (boss) tc5::tma_store_wait_read<1>();     // the previous state tile has been read
    if (!tc5::mbar_wait(m2, c & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) { ok = false; }
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc5::fence_after_sync();
    if (c + 1 < NC) {
      float sv[HC];
      tmem_ld_half(tmem + lane_off + cS, sv);     // S entering chunk c+1, row r
      uint32_t pk[HC / 2];
      pack_half(sv, pk);
      write_half(Sb, r, half, pk);
      const float g = __expf(gl_next);             // its decay through chunk c + 1
#pragma unroll
      for (int j = 0; j < HC; ++j) sv[j] *= g;
      tmem_st_half(tmem + lane_off + cS, sv);
      tc5::fence_proxy_async();
    }
    tc5::fence_before_sync();
    __syncthreads();
    if (boss && c + 1 < NC && p.store_states) {
      tc5::tma_store_2d(&tm_sa, Sb, vt * VT, (bh * NC + c + 1) * KD);
      tc5::tma_store_commit();
    }
  }
  if (ok) finish_output(NC - 1);
  if (boss || threadIdx.x == CH) tc5::tma_store_wait_read<0>();
  if (!ok && boss) {                               // a load for the next chunk may still be in flight
    tc5::mbar_drain(&full[0]);
    tc5::mbar_drain(&full[1]);
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 256); }
}

struct BwdParams {
  const bf16* d_o;       // [B, T, H, V]
  const float* gc;       // [BH, NC, 64]
  float* dgamma_part;    // [VTILES, BH, NC]
  int NC, V, BH, H, T;
  float scale;
  KernelStatus* status;
};

// stage: k-block kb of [k ; w] (2 x 16 KB), q (16 KB), S_prev [KD][64] (16 KB), [qk | 0] (16 KB, second half zero)
constexpr int BWD_STAGE = 10 * BOX;                                        // 80 KB
constexpr int BWD_TX = 9 * BOX;
constexpr int BWD_SMEM = 2 * BWD_STAGE + BOX /*du*/ + 2 * BOX /*do, sq do*/ + 2 * BOX /*dSb*/ + 1024 + 128;

__global__ void __launch_bounds__(256, 1)
gdn_seq_bwd_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_S,
                   const __grid_constant__ CUtensorMap tm_qk, const __grid_constant__ CUtensorMap tm_du,
                   const __grid_constant__ CUtensorMap tm_ds, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sDU = smem + 2 * BWD_STAGE;    // [64][64] du
  uint8_t* sDO = sDU + BOX;               // [64][64] do
  uint8_t* sDOs = sDO + BOX;              // [64][64] sq do
  uint8_t* dSb = sDOs + BOX;              // [KD rows][64] bf16 mirror of dS
  uint64_t* bars = reinterpret_cast<uint64_t*>(dSb + 2 * BOX);
  uint64_t* full = bars;
  uint64_t* m1 = bars + 2;
  uint64_t* m2 = bars + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* red = reinterpret_cast<float*>(tmem_slot + 2);     // [8]

  const int r = threadIdx.x & 127, half = threadIdx.x >> 7;
  const int warp = threadIdx.x >> 5;
  const bool boss = threadIdx.x == 0;
  const int vt = blockIdx.x, bh = blockIdx.y, h = bh % p.H, b = bh / p.H;
  const int NC = p.NC, V = p.V;

  if (boss) {
    *abort_flag = 0;
    tc5::mbar_init(&full[0], 1);
    tc5::mbar_init(&full[1], 1);
    tc5::mbar_init(m1, 1);
    tc5::mbar_init(m2, 1);
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 256); tc5::tmem_relinquish(); }
  {
    uint32_t z[HC / 2];
#pragma unroll
    for (int j = 0; j < HC / 2; ++j) z[j] = 0u;
    write_half(dSb, r, half, z);
    write_half(smem + (r >> 6) * BWD_STAGE + 9 * BOX, r & 63, half, z);
  }
  tc5::fence_proxy_async();
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_off = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * HC;   // lanes and columns of this thread
  // TMEM columns: Da = [k ; w] dS [0,64)   Dd = [qk^T ; 0] do [64,128)   dS [128,192)
  const uint32_t cDa = 0, cDd = 64, cDs = 128;
  {
    float z[HC];
#pragma unroll
    for (int j = 0; j < HC; ++j) z[j] = 0.f;
    tmem_st_half(tmem + lane_off + cDs, z);
  }
  tc5::fence_before_sync();
  __syncthreads();
  // outputs leave as TMA stores from swizzled tiles (see the forward kernel); the last chunk's state has no gradient
  if (boss) {
    tc5::tma_store_2d(&tm_ds, dSb, vt * VT, (bh * NC + NC - 1) * KD);
    tc5::tma_store_commit();
  }

  auto issue_loads = [&](int c, int it) {
    const int s = it & 1;
    uint8_t* st = smem + s * BWD_STAGE;
    const int row0 = (bh * NC + c) * CH;
    tc5::mbar_expect_tx(&full[s], BWD_TX);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tc5::tma_load_4d(st + kb * 2 * BOX, &tm_k, &full[s], kb * 64, h, c * CH, b);
      tc5::tma_load_2d(st + kb * 2 * BOX + BOX, &tm_w, &full[s], kb * 64, row0);
      tc5::tma_load_4d(st + 4 * BOX + kb * BOX, &tm_q, &full[s], kb * 64, h, c * CH, b);
    }
    tc5::tma_load_2d(st + 6 * BOX, &tm_S, &full[s], vt * VT, (bh * NC + c) * KD);
    tc5::tma_load_2d(st + 8 * BOX, &tm_qk, &full[s], 0, row0);
  };
  if (boss) issue_loads(NC - 1, 0);

  constexpr uint32_t id_a = tc5::make_idesc_bf16(128, VT, 0, 1);        // [k;w] (K-major) x dS (MN-major)
  constexpr uint32_t id_d = tc5::make_idesc_bf16(128, VT, 1, 1);        // q^T x (sq do), [qk^T ; 0] x do
  constexpr uint32_t id_dn = tc5::make_idesc_bf16(128, VT, 1, 1, 1);    // (-w)^T x du
  bool ok = true;
  // The chunk loop is one dependent chain: the do rows (threads 64..127) and the gates are fetched one chunk ahead.
  const float* gc = p.gc + static_cast<long>(bh) * NC * CH;
  const bf16* d_o = p.d_o + (static_cast<long>(b) * p.T * p.H + h) * V + vt * VT + half * HC;
  uint32_t row_next[HC / 2];
#pragma unroll
  for (int j = 0; j < HC / 2; ++j) row_next[j] = 0u;
  float gr_next, gl_next;
  auto fetch_rows = [&](int cc) {
    const int t = cc * CH + r - CH;
    if (r >= CH) {
      if (t < p.T) load_global(d_o + static_cast<long>(t) * p.H * V, row_next);
      else {
#pragma unroll
        for (int j = 0; j < HC / 2; ++j) row_next[j] = 0u;
      }
    }
    gr_next = gc[cc * CH + (r & 63)];
    gl_next = gc[cc * CH + CH - 1];
  };
  fetch_rows(NC - 1);
  for (int it = 0; it < NC && ok; ++it) {
    const int c = NC - 1 - it;
    const int s = it & 1;
    uint8_t* st = smem + s * BWD_STAGE;
    const long row0 = static_cast<long>(bh * NC + c) * CH;
    const float g_row = gr_next, g_last = gl_next;
    // stage this chunk's do rows (already in registers) and start the next chunk's loads
    if (r >= CH) {
      write_half(sDO, r - CH, half, row_next);
      float f[HC];
      unpack_half(row_next, f);
      const float sq = p.scale * __expf(g_row);
#pragma unroll
      for (int j = 0; j < HC; ++j) f[j] *= sq;
      uint32_t pk[HC / 2];
      pack_half(f, pk);
      write_half(sDOs, r - CH, half, pk);
    }
    if (c > 0) fetch_rows(c - 1);
    tc5::fence_proxy_async();
    tc5::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      // converged issuing warp, one elected lane issues (see the forward kernel)
      const bool lead = tc5::elect_one();
      if (__all_sync(0xffffffffu, tc5::mbar_wait(&full[s], (it >> 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_SMEM_FULL))) {
        tc5::fence_after_sync();
        const uint64_t a = tc5::desc_kmajor(tc5::smem_u32(st)), dsbm = tc5::desc_mnmajor(tc5::smem_u32(dSb), BOX);
        const uint64_t qk = tc5::desc_mnmajor(tc5::smem_u32(st + 8 * BOX), BOX), dom = tc5::desc_mnmajor(tc5::smem_u32(sDO), BOX);
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < KD / 16; ++kk)      // Da = [k ; w] dS
            tc5::mma_ss(tmem + cDa, a + static_cast<uint64_t>(((kk >> 2) * 2 * BOX + (kk & 3) * 32) >> 4),
                        dsbm + static_cast<uint64_t>((kk * 2048) >> 4), id_a, kk > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < CH / 16; ++kk)      // Dd = [qk^T ; 0] do
            tc5::mma_ss(tmem + cDd, qk + static_cast<uint64_t>((kk * 2048) >> 4), dom + static_cast<uint64_t>((kk * 2048) >> 4), id_d, kk > 0 ? 1u : 0u);
          tc5::mma_commit(m1);
          if (it + 1 < NC) issue_loads(c - 1, it + 1);
        }
      }
      __syncwarp();
    }
    if (!tc5::mbar_wait(m1, it & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) { ok = false; }
    if (boss) tc5::tma_store_wait_read<1>();     // the previous du tile has been read (one newer store: the dS tile)
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc5::fence_after_sync();
    if (r < CH) {
      float da[HC], dd[HC];
      tmem_ld_half(tmem + lane_off + cDa, da);
      tmem_ld_half(tmem + lane_off + cDd, dd);
      const float sk = __expf(g_last - g_row);
#pragma unroll
      for (int j = 0; j < HC; ++j) da[j] = dd[j] + sk * da[j];
      uint32_t pk[HC / 2];
      pack_half(da, pk);
      write_half(sDU, r, half, pk);
    }
    float part_dg = 0.f;
    {
      // dS: dgamma partial with S_prev, then scaled by gamma in place
      float ds[HC], sp[HC];
      tmem_ld_half(tmem + lane_off + cDs, ds);
      read_half(st + 6 * BOX, r, half, sp);
      const float g = __expf(g_last);
#pragma unroll
      for (int j = 0; j < HC; ++j) { part_dg += ds[j] * sp[j]; ds[j] *= g; }
      tmem_st_half(tmem + lane_off + cDs, ds);
    }
    tc5::fence_proxy_async();
    tc5::fence_before_sync();
    __syncthreads();
    if (boss) {
      tc5::tma_store_2d(&tm_du, sDU, vt * VT, static_cast<int>(row0));
      tc5::tma_store_commit();
    }
    if (warp == 0) {
      const bool lead = tc5::elect_one();
      tc5::fence_after_sync();
      const uint64_t qdm = tc5::desc_mnmajor(tc5::smem_u32(st + 4 * BOX), BOX), dom = tc5::desc_mnmajor(tc5::smem_u32(sDOs), BOX);
      const uint64_t wm = tc5::desc_mnmajor(tc5::smem_u32(st + BOX), 2 * BOX), dum = tc5::desc_mnmajor(tc5::smem_u32(sDU), BOX);
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)        // dS += q^T (sq do)
          tc5::mma_ss(tmem + cDs, qdm + static_cast<uint64_t>((kk * 2048) >> 4), dom + static_cast<uint64_t>((kk * 2048) >> 4), id_d, 1u);
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)        // dS -= w^T du      (w = second half of each k-block)
          tc5::mma_ss(tmem + cDs, wm + static_cast<uint64_t>((kk * 2048) >> 4), dum + static_cast<uint64_t>((kk * 2048) >> 4), id_dn, 1u);
        tc5::mma_commit(m2);
      }
      __syncwarp();
    }
    // block reduction of the dgamma partial, behind the MMAs
    for (int o = 16; o > 0; o >>= 1) part_dg += __shfl_xor_sync(0xffffffffu, part_dg, o);
    if ((threadIdx.x & 31) == 0) red[warp] = part_dg;
    if (boss) tc5::tma_store_wait_read<1>();     // the previous dS tile has been read
    if (!tc5::mbar_wait(m2, it & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) { ok = false; }
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc5::fence_after_sync();
    if (boss) p.dgamma_part[(static_cast<long>(vt) * p.BH + bh) * NC + c] =
        ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
    if (c > 0) {
      float ds[HC];
      tmem_ld_half(tmem + lane_off + cDs, ds);
      uint32_t pk[HC / 2];
      pack_half(ds, pk);
      write_half(dSb, r, half, pk);
    }
    tc5::fence_proxy_async();
    tc5::fence_before_sync();
    __syncthreads();
    if (boss && c > 0) {
      tc5::tma_store_2d(&tm_ds, dSb, vt * VT, (bh * NC + c - 1) * KD);
      tc5::tma_store_commit();
    }
  }
  if (boss) tc5::tma_store_wait_read<0>();
  if (!ok && boss) {                               // a load for the next chunk may still be in flight
    tc5::mbar_drain(&full[0]);
    tc5::mbar_drain(&full[1]);
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 256); }
}

int make_rows_map(CUtensorMap* m, const void* base, long rows, int cols, int box_rows) {
  return nsa::make_tmap_2d_bf16(m, base, cols, rows, cols, 64, box_rows);
}
// [B, T, H, D] token-major; box: 64 tokens of one head, 64 columns
int make_token_map(CUtensorMap* m, const void* base, int B, int T, int H, int D) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)T, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)D * 2, (uint64_t)H * D * 2, (uint64_t)T * H * D * 2};
  uint32_t box[4] = {64, 1, (uint32_t)CH, 1};
  return nsa::make_tmap_bf16(m, base, 4, dims, strides, box, 1);
}
template <typename F>
int set_smem(F* kernel, int bytes, const char* what) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, what);
}
}  // namespace

// q, k [B, T, H, 128] bf16; w [B*H, NC, 64, 128], u [.., 64, V], qk [.., 64, 64] bf16 and gc [B*H, NC, 64] fp32 from
// nsa_gdn_prep.  o [B, T, H, V]; v_new [B*H, NC, 64, V] and S_all [B*H, NC, 128, V] (states entering the chunks) are
// written for the backward, or null.
extern "C" int nsa_gdn_seq_fwd(const void* q, const void* k, const void* w, const void* u, const void* qk, const float* gc,
                               void* o, void* v_new, void* S_all, int B, int T, int H, int K, int V, float scale,
                               cudaStream_t st) {
  if (K != KD || V % VT) return nsa::fail(NSA_ERR_SHAPE, "gdn: key width must be 128 and value width a multiple of 64");
  const int NC = (T + CH - 1) / CH, BH = B * H;
  const long rows = static_cast<long>(BH) * NC * CH;
  const bool states = v_new != nullptr && S_all != nullptr;
  CUtensorMap tw, tq, tk, tqk, tvn, to, tsa;
  int rc;
  if ((rc = make_rows_map(&tw, w, rows, KD, CH))) return rc;
  if ((rc = make_token_map(&tq, q, B, T, H, KD))) return rc;
  if ((rc = make_token_map(&tk, k, B, T, H, KD))) return rc;
  if ((rc = make_rows_map(&tqk, qk, rows, CH, CH))) return rc;
  if ((rc = make_token_map(&to, o, B, T, H, V))) return rc;
  tvn = tw; tsa = tw;                              // never used without the states
  if (states && (rc = make_rows_map(&tvn, v_new, rows, V, CH))) return rc;
  if (states && (rc = make_rows_map(&tsa, S_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  FwdParams p{(const bf16*)u, gc, states, NC, V, H, scale, nsa::status_ptr()};
  if ((rc = set_smem(gdn_seq_fwd_kernel, FWD_SMEM, "gdn fwd smem attribute"))) return rc;
  gdn_seq_fwd_kernel<<<dim3(V / VT, BH), 256, FWD_SMEM, st>>>(tw, tq, tk, tqk, tvn, to, tsa, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gdn_seq_fwd launch");
}

// d_o [B, T, H, V] bf16.  Outputs: du [B*H, NC, 64, V], dS_all [B*H, NC, 128, V] (gradients of the states leaving the
// chunks) bf16, dgamma_part [V/64, B*H, NC] fp32.
extern "C" int nsa_gdn_seq_bwd(const void* q, const void* k, const void* w, const void* qk, const void* S_all, const void* d_o,
                               const float* gc, void* du, void* dS_all, float* dgamma_part, int B, int T, int H, int K, int V,
                               float scale, cudaStream_t st) {
  if (K != KD || V % VT) return nsa::fail(NSA_ERR_SHAPE, "gdn: key width must be 128 and value width a multiple of 64");
  const int NC = (T + CH - 1) / CH, BH = B * H;
  const long rows = static_cast<long>(BH) * NC * CH;
  CUtensorMap tw, tq, tk, tqk, ts, tdu, tds;
  int rc;
  if ((rc = make_rows_map(&tw, w, rows, KD, CH))) return rc;
  if ((rc = make_token_map(&tq, q, B, T, H, KD))) return rc;
  if ((rc = make_token_map(&tk, k, B, T, H, KD))) return rc;
  if ((rc = make_rows_map(&tqk, qk, rows, CH, CH))) return rc;
  if ((rc = make_rows_map(&ts, S_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  if ((rc = make_rows_map(&tdu, du, rows, V, CH))) return rc;
  if ((rc = make_rows_map(&tds, dS_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  BwdParams p{(const bf16*)d_o, gc, dgamma_part, NC, V, BH, H, T, scale, nsa::status_ptr()};
  if ((rc = set_smem(gdn_seq_bwd_kernel, BWD_SMEM, "gdn bwd smem attribute"))) return rc;
  gdn_seq_bwd_kernel<<<dim3(V / VT, BH), 256, BWD_SMEM, st>>>(tw, tq, tk, ts, tqk, tdu, tds, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gdn_seq_bwd launch");
}
