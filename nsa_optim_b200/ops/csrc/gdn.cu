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
  const float* gc;      // [BH, NC, 64]
  int store_states;     // also write v_new and S_all (the backward needs them)
  int NC, H;
  float scale;
  KernelStatus* status;
};

// Roles of both kernels: warps 0..7 compute, warp 8 issues the products, warp 9 loads, the last one stores.  The chunk loop is one
// dependent chain (product, accumulator rows, product, state rows), so everything that is not on it is kept off the
// warps that are: a thread that also copies and issues costs its whole CTA 1400 of 3500 cycles a chunk at the barriers.
constexpr int WARP_MMA = 8, WARP_LOAD = 9;
// A chunk's tiles are asked for into L2 this many chunks ahead: two stages alone leave a load from memory one chunk's time,
// and the chain then waits for it.  256 chunks x 64 CTAs, forward and backward: 472 and 526 us with one thread for copies,
// stores and products, 455 and 597 with warps for each, 395 and 492 with the prefetch and operands released where their last
// product is issued, 356 and 365 with u and do as tiles too (rows of their own per thread are 32 lines an instruction),
// 336 and 361 with the wait for a tile's last stores in front of the one for the state, 316 and 321 with waits that vote and, backward,
// qk^T do issued in front of the wait for the state (that alone: 354 to 346).
constexpr int AHEAD = 6;

// stage: k-block kb of [w ; q] (2 x 16 KB), k (16 KB), [0 ; qk] (16 KB, first half zero)
constexpr int FWD_STAGE = 8 * BOX;
constexpr int FWD_TX_A = 4 * BOX, FWD_TX_B = 3 * BOX;    // bytes that arrive per chunk: [w ; q], free after the first product, and the rest
constexpr int FWD_SMEM = 2 * FWD_STAGE + 2 * BOX /*u*/ + 4 * BOX /*Sb*/ + 3 * BOX /*Vb, Vs*/ + 2 * BOX /*Ob*/ + 1024 + 256;

__global__ void __launch_bounds__(352, 1)
gdn_seq_fwd_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_qk,
                   const __grid_constant__ CUtensorMap tm_vn, const __grid_constant__ CUtensorMap tm_o,
                   const __grid_constant__ CUtensorMap tm_sa, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* Sb = smem + 2 * FWD_STAGE;           // 2 x [KD rows][64] bf16 state, B operand
  uint8_t* Vb = Sb + 4 * BOX;                   // 2 x [64 rows][64] v_new
  uint8_t* Ob = Vb + 2 * BOX;                   // 2 x [64 rows][64] o on its way out
  uint8_t* Vs = Ob + 2 * BOX;                   // [64 rows][64] sk v_new
  uint8_t* Us = Vs + BOX;                       // 2 x [64 rows][64] u
  uint64_t* bars = reinterpret_cast<uint64_t*>(Us + 2 * BOX);
  uint64_t *full_a = bars, *empty_a = bars + 2, *full_b = bars + 4, *empty_b = bars + 6;     // [2] each: the stages
  uint64_t *full_u = bars + 8, *empty_u = bars + 10;                  // [2] each
  uint64_t *m1 = bars + 12, *m2 = bars + 13, *m3 = bars + 14;         // products complete: D1, S, D2
  uint64_t *sready = bars + 15, *scaled = bars + 16, *vready = bars + 17, *oready = bars + 18;   // rows written: Sb, S, Vb and Vs, Ob
  uint64_t* freed = bars + 19;                  // stores of the chunk before have read their tiles
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int r = threadIdx.x & 127, half = (threadIdx.x >> 7) & 1;   // TMEM lane / tile row, half of its columns
  const int warp = threadIdx.x >> 5;
  const int vt = blockIdx.x, bh = blockIdx.y, h = bh % p.H, b = bh / p.H;
  const int NC = p.NC;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 10; ++i) tc5::mbar_init(bars + i, 1);
    tc5::mbar_init(empty_u, 4);
    tc5::mbar_init(empty_u + 1, 4);
    tc5::mbar_init(m1, 1);
    tc5::mbar_init(m2, 1);
    tc5::mbar_init(m3, 1);
    tc5::mbar_init(sready, 8);
    tc5::mbar_init(scaled, 8);
    tc5::mbar_init(vready, 4);
    tc5::mbar_init(oready, 4);
    tc5::mbar_init(freed, 1);
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 256); tc5::tmem_relinquish(); }
  if (warp < 8) {
    // S = 0: bf16 mirror in shared memory; the constant zero half of both [0 ; qk] operands
    uint32_t z[HC / 2];
#pragma unroll
    for (int j = 0; j < HC / 2; ++j) z[j] = 0u;
    write_half(Sb, r, half, z);
    write_half(smem + (r >> 6) * FWD_STAGE + 6 * BOX, r & 63, half, z);
    tc5::fence_proxy_async();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // TMEM columns: D1 = [w ; q] S [0, 64)   S [64, 128)   D2 = [0 ; qk] v_new [128, 192)
  const uint32_t cD1 = 0, cS = 64, cD2 = 128;
  auto wait = [&](uint64_t* bar, int phase, int code) {
    return tc5::mbar_wait_warp(bar, phase & 1, abort_flag, p.status, code);
  };
  const float* gc = p.gc + static_cast<long>(bh) * NC * CH;
  if (warp < 8) {
    const uint32_t lane_off = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * HC;   // lanes and columns of this thread
    {
      float z[HC];
#pragma unroll
      for (int j = 0; j < HC; ++j) z[j] = 0.f;
      tmem_st_half(tmem + lane_off + cS, z);
    }
    tc5::fence_before_sync();
    tc5::arrive_warp(sready);
    tc5::arrive_warp(scaled);
    const bool upper = r < CH;                     // rows of w S and v_new; the others hold q S and the output
    // The gates are in flight for a whole chunk.
    float g_row = gc[r & 63], g_last = gc[CH - 1];
    for (int c = 0; c < NC; ++c) {
      float g_row_next = 0.f, g_last_next = 0.f;
      if (c + 1 < NC) {
        g_row_next = gc[(c + 1) * CH + (r & 63)];
        g_last_next = gc[(c + 1) * CH + CH - 1];
      }
      const float sk = __expf(g_last - g_row), sq = p.scale * __expf(g_row);
      float uf[HC];
      if (upper) {
        if (!wait(full_u + (c & 1), c >> 1, STATUS_TIMEOUT_SMEM_FULL)) break;
        read_half(Us + (c & 1) * BOX, r, half, uf);
        tc5::arrive_warp(empty_u + (c & 1));
      }
      if (!wait(m1, c, STATUS_TIMEOUT_TMEM_FULL)) break;
      tc5::fence_after_sync();
      float d1[HC];
      tmem_ld_half(tmem + lane_off + cD1, d1);
      if (upper) {
        uint32_t pk[HC / 2], ps[HC / 2];
#pragma unroll
        for (int j = 0; j < HC; ++j) d1[j] = uf[j] - d1[j];
        pack_half(d1, pk);
#pragma unroll
        for (int j = 0; j < HC; ++j) d1[j] *= sk;
        pack_half(d1, ps);
        write_half(Vs, r, half, ps);               // read by the products of chunk c - 1, complete since m2
        write_half(Vb + (c & 1) * BOX, r, half, pk);
        tc5::fence_proxy_async();
        tc5::arrive_warp(vready);
      } else {
#pragma unroll
        for (int j = 0; j < HC; ++j) d1[j] *= sq;
      }
      if (c + 1 < NC) {
        const float g = __expf(g_last_next);       // decay of the state through chunk c + 1
        // the wait for the stores, which are through by now, goes first and is off the chain
        if (!wait(freed, c, STATUS_TIMEOUT_SMEM_EMPTY) || !wait(m2, c, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        float sv[HC];
        tmem_ld_half(tmem + lane_off + cS, sv);    // S entering chunk c + 1, row r
        uint32_t pk[HC / 2];
        pack_half(sv, pk);
        write_half(Sb + ((c + 1) & 1) * 2 * BOX, r, half, pk);
        tc5::fence_proxy_async();
        tc5::fence_before_sync();
        tc5::arrive_warp(sready);
#pragma unroll
        for (int j = 0; j < HC; ++j) sv[j] *= g;
        tmem_st_half(tmem + lane_off + cS, sv);
        tc5::fence_before_sync();
        tc5::arrive_warp(scaled);
      } else if (!wait(freed, c, STATUS_TIMEOUT_SMEM_EMPTY)) {
        break;
      }
      if (!upper) {                                // output rows, behind the next chunk's first product
        if (!wait(m3, c, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        float d2[HC];
        tmem_ld_half(tmem + lane_off + cD2, d2);
#pragma unroll
        for (int j = 0; j < HC; ++j) d2[j] += d1[j];
        uint32_t pk[HC / 2];
        pack_half(d2, pk);
        write_half(Ob + (c & 1) * BOX, r - CH, half, pk);
        tc5::fence_proxy_async();
        tc5::fence_before_sync();
        tc5::arrive_warp(oready);
      }
      g_row = g_row_next;
      g_last = g_last_next;
    }
  } else if (warp == WARP_MMA) {
    constexpr uint32_t idesc1 = tc5::make_idesc_bf16(128, VT, 0, 1);   // A K-major, B MN-major
    constexpr uint32_t idesc2 = tc5::make_idesc_bf16(128, VT, 1, 1);   // A MN-major (k^T), B MN-major
    // The issuing warp stays converged and one elected lane issues: descriptors then live in uniform
    // registers and an MMA costs the issuing thread a few cycles instead of 70 to 100.
    const bool lead = tc5::elect_one();
    const uint64_t vs = tc5::desc_mnmajor(tc5::smem_u32(Vs), BOX);
    for (int c = 0; c < NC; ++c) {
      const int s = c & 1;
      const uint32_t st = tc5::smem_u32(smem + s * FWD_STAGE);
      const uint64_t a1 = tc5::desc_kmajor(st), sb = tc5::desc_mnmajor(tc5::smem_u32(Sb + s * 2 * BOX), BOX);
      const uint64_t kt = tc5::desc_mnmajor(st + 4 * BOX, BOX), qk = tc5::desc_kmajor(st + 6 * BOX);
      const uint64_t vb = tc5::desc_mnmajor(tc5::smem_u32(Vb + s * BOX), BOX);
      if (!wait(full_a + s, c >> 1, STATUS_TIMEOUT_SMEM_FULL) || !wait(sready, c, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < KD / 16; ++kk)
          tc5::mma_ss(tmem + cD1, a1 + static_cast<uint64_t>(((kk >> 2) * 2 * BOX + (kk & 3) * 32) >> 4),
                      sb + static_cast<uint64_t>((kk * 2048) >> 4), idesc1, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m1);
        tc5::mma_commit(empty_a + s);
      }
      __syncwarp();
      if (!wait(full_b + s, c >> 1, STATUS_TIMEOUT_SMEM_FULL) || !wait(scaled, c, STATUS_TIMEOUT_TMEM_EMPTY) || (c > 0 && !wait(oready, c - 1, STATUS_TIMEOUT_TMEM_EMPTY)) ||
          !wait(vready, c, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)       // S += k^T (sk v_new)
          tc5::mma_ss(tmem + cS, kt + static_cast<uint64_t>((kk * 2048) >> 4), vs + static_cast<uint64_t>((kk * 2048) >> 4), idesc2, 1u);
        tc5::mma_commit(m2);
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)       // D2 = [0 ; qk] v_new
          tc5::mma_ss(tmem + cD2, qk + static_cast<uint64_t>((kk * 32) >> 4), vb + static_cast<uint64_t>((kk * 2048) >> 4), idesc1, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m3);
        tc5::mma_commit(empty_b + s);
      }
      __syncwarp();
    }
  } else if (warp == WARP_LOAD) {
    const bool lead = tc5::elect_one();
    bool ok = true;
    // The CTAs of a head's V tiles share the chunk's tiles; each asks for those of every nvt-th chunk.
    const int nvt = gridDim.x;
    auto prefetch = [&](int c) {
      if (c >= NC || !lead) return;
      const int row0 = (bh * NC + c) * CH;
      tc5::tma_prefetch_2d(&tm_u, vt * VT, row0);
      if (c % nvt != vt) return;
#pragma unroll
      for (int kb = 0; kb < 2; ++kb) {
        tc5::tma_prefetch_2d(&tm_w, kb * 64, row0);
        tc5::tma_prefetch_4d(&tm_q, kb * 64, h, c * CH, b);
        tc5::tma_prefetch_4d(&tm_k, kb * 64, h, c * CH, b);
      }
      tc5::tma_prefetch_2d(&tm_qk, 0, row0);
    };
    for (int c = 2; c < AHEAD; ++c) prefetch(c);
    for (int c = 0; c < NC; ++c) {
      const int s = c & 1, row0 = (bh * NC + c) * CH;
      uint8_t* st = smem + s * FWD_STAGE;
      if (c >= 2 && !(ok = wait(empty_a + s, (c >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full_a + s, FWD_TX_A);
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          tc5::tma_load_2d(st + kb * 2 * BOX, &tm_w, full_a + s, kb * 64, row0);
          tc5::tma_load_4d(st + kb * 2 * BOX + BOX, &tm_q, full_a + s, kb * 64, h, c * CH, b);
        }
      }
      __syncwarp();
      if (c >= 2 && !(ok = wait(empty_u + s, (c >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full_u + s, BOX);
        tc5::tma_load_2d(Us + s * BOX, &tm_u, full_u + s, vt * VT, row0);
      }
      __syncwarp();
      if (c >= 2 && !(ok = wait(empty_b + s, (c >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full_b + s, FWD_TX_B);
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) tc5::tma_load_4d(st + 4 * BOX + kb * BOX, &tm_k, full_b + s, kb * 64, h, c * CH, b);
        tc5::tma_load_2d(st + 7 * BOX, &tm_qk, full_b + s, 0, row0);
      }
      prefetch(c + AHEAD);
      __syncwarp();
    }
    for (int c = NC > 2 ? NC - 2 : 0; c < NC && ok; ++c)
      ok = wait(empty_a + (c & 1), c >> 1, STATUS_TIMEOUT_SMEM_EMPTY) && wait(empty_b + (c & 1), c >> 1, STATUS_TIMEOUT_SMEM_EMPTY);
    if (!ok && lead) {                             // loads may still be in flight
      for (int i = 0; i < 2; ++i) {
        tc5::mbar_drain(full_a + i);
        tc5::mbar_drain(full_b + i);
        tc5::mbar_drain(full_u + i);
      }
    }
    __syncwarp();
  } else {
    // Outputs leave as TMA stores from the swizzled tiles they are in anyway; chunk 0 enters with the zero state.
    const bool lead = tc5::elect_one();
    auto store_o = [&](int c) {                    // rows past T are clipped by the copy engine
      if (lead) tc5::tma_store_4d(&tm_o, Ob + (c & 1) * BOX, vt * VT, h, c * CH, b);
    };
    bool ok = true;
    for (int c = 0; c < NC; ++c) {
      if (!(ok = wait(sready, c, STATUS_TIMEOUT_TMEM_EMPTY))) break;
      if (lead && p.store_states) tc5::tma_store_2d(&tm_sa, Sb + (c & 1) * 2 * BOX, vt * VT, (bh * NC + c) * KD);
      if (c > 0) {
        if (!(ok = wait(oready, c - 1, STATUS_TIMEOUT_TMEM_EMPTY))) break;
        store_o(c - 1);
      }
      if (!(ok = wait(vready, c, STATUS_TIMEOUT_TMEM_EMPTY))) break;
      if (lead) {
        if (p.store_states) tc5::tma_store_2d(&tm_vn, Vb + (c & 1) * BOX, vt * VT, (bh * NC + c) * CH);
        tc5::tma_store_commit();
        tc5::tma_store_wait_read<1>();
      }
      tc5::arrive_warp(freed);
    }
    if (ok && wait(oready, NC - 1, STATUS_TIMEOUT_TMEM_EMPTY)) store_o(NC - 1);
    if (lead) {
      tc5::tma_store_commit();
      tc5::tma_store_wait_read<0>();
    }
    __syncwarp();
  }
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc5::fence_after_sync(); tc5::tmem_dealloc(tmem, 256); }
}

struct BwdParams {
  const float* gc;       // [BH, NC, 64]
  float* dgamma_part;    // [VTILES, BH, NC]
  int NC, BH, H;
  float scale;
  KernelStatus* status;
};

// stage: k-block kb of [k ; w] (2 x 16 KB), q (16 KB), S_prev [KD][64] (16 KB), [qk | 0] (16 KB, second half zero)
constexpr int BWD_STAGE = 10 * BOX;                                        // 80 KB
constexpr int BWD_TX = 8 * BOX, BWD_TX_S = 2 * BOX;                        // with do; S_prev is free much earlier than the others
constexpr int BWD_SMEM = 2 * BWD_STAGE + 2 * BOX /*du*/ + 3 * BOX /*do, sq do*/ + 2 * BOX /*dSb*/ + 1024 + 256;

__global__ void __launch_bounds__(352, 1)
gdn_seq_bwd_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_S,
                   const __grid_constant__ CUtensorMap tm_qk, const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_du,
                   const __grid_constant__ CUtensorMap tm_ds, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sDU = smem + 2 * BWD_STAGE;    // 2 x [64][64] du
  uint8_t* sDO = sDU + 2 * BOX;           // 2 x [64][64] do, of the stages
  uint8_t* sDOs = sDO + 2 * BOX;          // [64][64] sq do
  uint8_t* dSb = sDOs + BOX;              // [KD rows][64] bf16 mirror of dS
  uint64_t* bars = reinterpret_cast<uint64_t*>(dSb + 2 * BOX);
  uint64_t *full = bars, *empty = bars + 2;     // [2] each: the stages without S_prev
  uint64_t *full_s = bars + 4, *empty_s = bars + 6;   // [2] each: S_prev
  uint64_t *m1 = bars + 8, *m2 = bars + 9;      // products complete: Da and Dd, dS
  uint64_t *sready = bars + 10, *scaled = bars + 11, *uready = bars + 12, *oready = bars + 13;    // rows written: dSb, dS, du, do and sq do
  uint64_t *gready = bars + 14, *freed = bars + 15;   // sums of dgamma are there; dSb and the other tile of du have been read by their stores
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* red = reinterpret_cast<float*>(tmem_slot + 2);     // [2][8]

  const int r = threadIdx.x & 127, half = (threadIdx.x >> 7) & 1;
  const int warp = tc5::warp_index();
  const int vt = blockIdx.x, bh = blockIdx.y, h = bh % p.H, b = bh / p.H;
  const int NC = p.NC;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 6; ++i) tc5::mbar_init(bars + i, 1);
    tc5::mbar_init(empty_s, 8);
    tc5::mbar_init(empty_s + 1, 8);
    tc5::mbar_init(m1, 1);
    tc5::mbar_init(m2, 1);
    tc5::mbar_init(sready, 8);
    tc5::mbar_init(scaled, 8);
    tc5::mbar_init(uready, 4);
    tc5::mbar_init(oready, 4);
    tc5::mbar_init(gready, 8);
    tc5::mbar_init(freed, 1);
    tc5::fence_barrier_init();
  }
  if (warp == 0) { tc5::tmem_alloc(tmem_slot, 256); tc5::tmem_relinquish(); }
  if (warp < 8) {
    uint32_t z[HC / 2];
#pragma unroll
    for (int j = 0; j < HC / 2; ++j) z[j] = 0u;
    write_half(dSb, r, half, z);
    write_half(smem + (r >> 6) * BWD_STAGE + 9 * BOX, r & 63, half, z);
    tc5::fence_proxy_async();
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // TMEM columns: Da = [k ; w] dS [0,64)   Dd = [qk^T ; 0] do [64,128)   dS [128,192)
  const uint32_t cDa = 0, cDd = 64, cDs = 128;
  auto wait = [&](uint64_t* bar, int phase, int code) {
    return tc5::mbar_wait_warp(bar, phase & 1, abort_flag, p.status, code);
  };
  const float* gc = p.gc + static_cast<long>(bh) * NC * CH;
  if (warp < 8) {
    const uint32_t lane_off = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * HC;   // lanes and columns of this thread
    const bool upper = (warp & 3) < 2;                     // rows of k dS and du; the others bring do
    {
      float z[HC];
#pragma unroll
      for (int j = 0; j < HC; ++j) z[j] = 0.f;
      tmem_st_half(tmem + lane_off + cDs, z);
    }
    tc5::fence_before_sync();
    tc5::arrive_warp(sready);
    tc5::arrive_warp(scaled);
    auto stage_row = [&](int it, float g_row) {    // sq do of step `it`
      if (!wait(full + (it & 1), it >> 1, STATUS_TIMEOUT_SMEM_FULL)) return false;
      float f[HC];
      read_half(sDO + (it & 1) * BOX, r - CH, half, f);
      const float sq = p.scale * __expf(g_row);
#pragma unroll
      for (int j = 0; j < HC; ++j) f[j] *= sq;
      uint32_t pk[HC / 2];
      pack_half(f, pk);
      write_half(sDOs, r - CH, half, pk);
      tc5::fence_proxy_async();
      tc5::arrive_warp(oready);
      return true;
    };
    // dgamma of step `it`, whose leaving gradient is ds: partial per warp; the last use of the entering state in the stage
    auto gamma_part = [&](int it, const float (&ds)[HC]) {
      const int s = it & 1;
      if (!wait(full_s + s, it >> 1, STATUS_TIMEOUT_SMEM_FULL)) return false;
      float sp[HC], part = 0.f;
      read_half(smem + s * BWD_STAGE + 6 * BOX, r, half, sp);
#pragma unroll
      for (int j = 0; j < HC; ++j) part += ds[j] * sp[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if ((threadIdx.x & 31) == 0) red[s * 8 + warp] = part;
      tc5::arrive_warp(gready);
      tc5::arrive_warp(empty_s + s);
      return true;
    };
    float g_row = gc[(NC - 1) * CH + (r & 63)], g_last = gc[(NC - 1) * CH + CH - 1];
    bool ok = upper || stage_row(0, g_row);
    if (ok) {
      float z[HC];
#pragma unroll
      for (int j = 0; j < HC; ++j) z[j] = 0.f;
      ok = gamma_part(0, z);                       // nothing follows the last chunk
    }
    for (int it = 0; it < NC && ok; ++it) {
      const int c = NC - 1 - it;
      float g_row_next = 0.f, g_last_next = 0.f;
      if (c > 0) {
        g_row_next = gc[(c - 1) * CH + (r & 63)];
        g_last_next = gc[(c - 1) * CH + CH - 1];
      }
      const float sk = __expf(g_last - g_row);
      if (upper) {
        if (!wait(m1, it, STATUS_TIMEOUT_TMEM_FULL)) break;
        tc5::fence_after_sync();
        float da[HC], dd[HC];
        tmem_ld_half(tmem + lane_off + cDa, da);
        tmem_ld_half(tmem + lane_off + cDd, dd);
#pragma unroll
        for (int j = 0; j < HC; ++j) da[j] = dd[j] + sk * da[j];
        uint32_t pk[HC / 2];
        pack_half(da, pk);
        write_half(sDU + (it & 1) * BOX, r, half, pk);
        tc5::fence_proxy_async();
        tc5::fence_before_sync();
        tc5::arrive_warp(uready);
      }
      if (c == 0) break;
      const float g = __expf(g_last_next);
      if (!wait(freed, it, STATUS_TIMEOUT_SMEM_EMPTY) || !wait(m2, it, STATUS_TIMEOUT_TMEM_FULL)) break;
      tc5::fence_after_sync();
      float ds[HC];
      tmem_ld_half(tmem + lane_off + cDs, ds);     // gradient of the state leaving chunk c - 1
      uint32_t pk[HC / 2];
      pack_half(ds, pk);
      write_half(dSb, r, half, pk);
      tc5::fence_proxy_async();
      tc5::fence_before_sync();
      tc5::arrive_warp(sready);
      if (!upper && !stage_row(it + 1, g_row_next)) break;
      {
        float sv[HC];
#pragma unroll
        for (int j = 0; j < HC; ++j) sv[j] = g * ds[j];
        tmem_st_half(tmem + lane_off + cDs, sv);
      }
      tc5::fence_before_sync();
      tc5::arrive_warp(scaled);
      ok = gamma_part(it + 1, ds);
      g_row = g_row_next;
      g_last = g_last_next;
    }
  } else if (warp == WARP_MMA) {
    constexpr uint32_t id_a = tc5::make_idesc_bf16(128, VT, 0, 1);        // [k;w] (K-major) x dS (MN-major)
    constexpr uint32_t id_d = tc5::make_idesc_bf16(128, VT, 1, 1);        // q^T x (sq do), [qk^T ; 0] x do
    constexpr uint32_t id_dn = tc5::make_idesc_bf16(128, VT, 1, 1, 1);    // (-w)^T x du
    const bool lead = tc5::elect_one();            // converged issuing warp, one elected lane issues (see the forward kernel)
    const uint64_t dsbm = tc5::desc_mnmajor(tc5::smem_u32(dSb), BOX), dos = tc5::desc_mnmajor(tc5::smem_u32(sDOs), BOX);
    for (int it = 0; it < NC; ++it) {
      const int s = it & 1;
      const uint32_t st = tc5::smem_u32(smem + s * BWD_STAGE);
      const uint64_t a = tc5::desc_kmajor(st), dom = tc5::desc_mnmajor(tc5::smem_u32(sDO + s * BOX), BOX);
      const uint64_t qk = tc5::desc_mnmajor(st + 8 * BOX, BOX), qdm = tc5::desc_mnmajor(st + 4 * BOX, BOX);
      const uint64_t wm = tc5::desc_mnmajor(st + BOX, 2 * BOX), dum = tc5::desc_mnmajor(tc5::smem_u32(sDU + s * BOX), BOX);
      // Dd waits for nothing but its tiles (its last rows were read before the du that the products of step it - 1 waited for)
      if (!wait(full + s, it >> 1, STATUS_TIMEOUT_SMEM_FULL)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)      // Dd = [qk^T ; 0] do
          tc5::mma_ss(tmem + cDd, qk + static_cast<uint64_t>((kk * 2048) >> 4), dom + static_cast<uint64_t>((kk * 2048) >> 4), id_d, kk > 0 ? 1u : 0u);
      }
      __syncwarp();
      if (!wait(sready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < KD / 16; ++kk)      // Da = [k ; w] dS
          tc5::mma_ss(tmem + cDa, a + static_cast<uint64_t>(((kk >> 2) * 2 * BOX + (kk & 3) * 32) >> 4),
                      dsbm + static_cast<uint64_t>((kk * 2048) >> 4), id_a, kk > 0 ? 1u : 0u);
        tc5::mma_commit(m1);
      }
      __syncwarp();
      if (!wait(oready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      if (!wait(scaled, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)        // dS += q^T (sq do)
          tc5::mma_ss(tmem + cDs, qdm + static_cast<uint64_t>((kk * 2048) >> 4), dos + static_cast<uint64_t>((kk * 2048) >> 4), id_d, 1u);
      }
      __syncwarp();
      if (!wait(uready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      tc5::fence_after_sync();
      if (lead) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk)        // dS -= w^T du      (w = second half of each k-block)
          tc5::mma_ss(tmem + cDs, wm + static_cast<uint64_t>((kk * 2048) >> 4), dum + static_cast<uint64_t>((kk * 2048) >> 4), id_dn, 1u);
        tc5::mma_commit(m2);
        tc5::mma_commit(empty + s);
      }
      __syncwarp();
    }
  } else if (warp == WARP_LOAD) {
    const bool lead = tc5::elect_one();
    bool ok = true;
    const int nvt = gridDim.x;
    auto prefetch = [&](int it) {                    // see the forward kernel; S_prev is this CTA's own
      const int c = NC - 1 - it, row0 = (bh * NC + c) * CH;
      if (c < 0 || !lead) return;
      tc5::tma_prefetch_2d(&tm_S, vt * VT, (bh * NC + c) * KD);
      tc5::tma_prefetch_4d(&tm_do, vt * VT, h, c * CH, b);
      if (c % nvt != vt) return;
#pragma unroll
      for (int kb = 0; kb < 2; ++kb) {
        tc5::tma_prefetch_4d(&tm_k, kb * 64, h, c * CH, b);
        tc5::tma_prefetch_2d(&tm_w, kb * 64, row0);
        tc5::tma_prefetch_4d(&tm_q, kb * 64, h, c * CH, b);
      }
      tc5::tma_prefetch_2d(&tm_qk, 0, row0);
    };
    for (int it = 2; it < AHEAD; ++it) prefetch(it);
    for (int it = 0; it < NC; ++it) {
      const int s = it & 1, c = NC - 1 - it, row0 = (bh * NC + c) * CH;
      uint8_t* st = smem + s * BWD_STAGE;
      if (it >= 2 && !(ok = wait(empty_s + s, (it >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full_s + s, BWD_TX_S);
        tc5::tma_load_2d(st + 6 * BOX, &tm_S, full_s + s, vt * VT, (bh * NC + c) * KD);
      }
      __syncwarp();
      if (it >= 2 && !(ok = wait(empty + s, (it >> 1) - 1, STATUS_TIMEOUT_SMEM_EMPTY))) break;
      if (lead) {
        tc5::mbar_expect_tx(full + s, BWD_TX);
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          tc5::tma_load_4d(st + kb * 2 * BOX, &tm_k, full + s, kb * 64, h, c * CH, b);
          tc5::tma_load_2d(st + kb * 2 * BOX + BOX, &tm_w, full + s, kb * 64, row0);
          tc5::tma_load_4d(st + 4 * BOX + kb * BOX, &tm_q, full + s, kb * 64, h, c * CH, b);
        }
        tc5::tma_load_2d(st + 8 * BOX, &tm_qk, full + s, 0, row0);
        tc5::tma_load_4d(sDO + s * BOX, &tm_do, full + s, vt * VT, h, c * CH, b);
      }
      prefetch(it + AHEAD);
      __syncwarp();
    }
    for (int it = NC > 2 ? NC - 2 : 0; it < NC && ok; ++it)
      ok = wait(empty + (it & 1), it >> 1, STATUS_TIMEOUT_SMEM_EMPTY) && wait(empty_s + (it & 1), it >> 1, STATUS_TIMEOUT_SMEM_EMPTY);
    if (!ok && lead) {                               // loads may still be in flight
      for (int i = 0; i < 2; ++i) {
        tc5::mbar_drain(full + i);
        tc5::mbar_drain(full_s + i);
      }
    }
    __syncwarp();
  } else {
    // outputs leave as TMA stores from swizzled tiles; the last chunk's state has no gradient
    const bool lead = tc5::elect_one();
    for (int it = 0; it < NC; ++it) {
      const int s = it & 1, c = NC - 1 - it;
      if (!wait(sready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      if (lead) {
        tc5::tma_store_2d(&tm_ds, dSb, vt * VT, (bh * NC + c) * KD);
        tc5::tma_store_commit();
      }
      if (!wait(gready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      if (lead) {
        const float* g = red + s * 8;
        p.dgamma_part[(static_cast<long>(vt) * p.BH + bh) * NC + c] = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7]));
      }
      if (!wait(uready, it, STATUS_TIMEOUT_TMEM_EMPTY)) break;
      if (lead) {
        tc5::tma_store_2d(&tm_du, sDU + s * BOX, vt * VT, (bh * NC + c) * CH);
        tc5::tma_store_commit();
        tc5::tma_store_wait_read<1>();             // dS of this chunk and du of the one before have been read
      }
      tc5::arrive_warp(freed);
    }
    if (lead) tc5::tma_store_wait_read<0>();
    __syncwarp();
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
  CUtensorMap tw, tu, tq, tk, tqk, tvn, to, tsa;
  int rc;
  if ((rc = make_rows_map(&tw, w, rows, KD, CH))) return rc;
  if ((rc = make_rows_map(&tu, u, rows, V, CH))) return rc;
  if ((rc = make_token_map(&tq, q, B, T, H, KD))) return rc;
  if ((rc = make_token_map(&tk, k, B, T, H, KD))) return rc;
  if ((rc = make_rows_map(&tqk, qk, rows, CH, CH))) return rc;
  if ((rc = make_token_map(&to, o, B, T, H, V))) return rc;
  tvn = tw; tsa = tw;                              // never used without the states
  if (states && (rc = make_rows_map(&tvn, v_new, rows, V, CH))) return rc;
  if (states && (rc = make_rows_map(&tsa, S_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  FwdParams p{gc, states, NC, H, scale, nsa::status_ptr()};
  if ((rc = set_smem(gdn_seq_fwd_kernel, FWD_SMEM, "gdn fwd smem attribute"))) return rc;
  gdn_seq_fwd_kernel<<<dim3(V / VT, BH), 352, FWD_SMEM, st>>>(tw, tu, tq, tk, tqk, tvn, to, tsa, p);
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
  CUtensorMap tw, tq, tk, tqk, ts, tdo, tdu, tds;
  int rc;
  if ((rc = make_rows_map(&tw, w, rows, KD, CH))) return rc;
  if ((rc = make_token_map(&tq, q, B, T, H, KD))) return rc;
  if ((rc = make_token_map(&tk, k, B, T, H, KD))) return rc;
  if ((rc = make_rows_map(&tqk, qk, rows, CH, CH))) return rc;
  if ((rc = make_rows_map(&ts, S_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  if ((rc = make_token_map(&tdo, d_o, B, T, H, V))) return rc;
  if ((rc = make_rows_map(&tdu, du, rows, V, CH))) return rc;
  if ((rc = make_rows_map(&tds, dS_all, static_cast<long>(BH) * NC * KD, V, KD))) return rc;
  BwdParams p{gc, dgamma_part, NC, BH, H, scale, nsa::status_ptr()};
  if ((rc = set_smem(gdn_seq_bwd_kernel, BWD_SMEM, "gdn bwd smem attribute"))) return rc;
  gdn_seq_bwd_kernel<<<dim3(V / VT, BH), 352, BWD_SMEM, st>>>(tw, tq, tk, ts, tqk, tdo, tdu, tds, p);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gdn_seq_bwd launch");
}
