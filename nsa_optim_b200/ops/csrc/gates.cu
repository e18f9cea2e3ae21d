// Step sizes and gates of the recurrent mixers where nothing is recorded: what PyTorch computes in seven to ten launches of two
// microseconds, five with the host's part, on a few thousand values (1000 tokens, three blocks: 743 -> 619 us for the whole call).  Same
// functions and roundings as its kernels, which is why this file is compiled without fast math: a block recomputed for its
// backward gives the values it gave.
#include <cuda_bf16.h>

#include "host.cuh"

namespace {
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float param(const void* p, int i, int fp32) {
  return fp32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const bf16*>(p)[i]);
}
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// DELTA: g = -exp(A_log) softplus(a + bias) and beta = sigmoid(b) -> out0, out1 [rows, H];
// else:  dt = softplus(a + bias) -> out0 [rows, H], -exp(A_log) -> out1 [H].
template <bool DELTA>
__global__ void __launch_bounds__(256) gates_kernel(const bf16* __restrict__ a, long lda, const bf16* __restrict__ b, long ldb,
                                                    const void* __restrict__ bias, int bias_fp32, const void* __restrict__ A_log, int A_fp32,
                                                    float* __restrict__ out0, float* __restrict__ out1, long rows, int H) {
  for (long i = static_cast<long>(blockIdx.x) * 256 + threadIdx.x; i < rows * H; i += static_cast<long>(gridDim.x) * 256) {
    const long row = i / H;
    const int h = static_cast<int>(i - row * H);
    const float sp = softplus(__bfloat162float(a[row * lda + h]) + param(bias, h, bias_fp32));
    if (DELTA) {
      out0[i] = -expf(param(A_log, h, A_fp32)) * sp;
      out1[i] = 1.f / (1.f + expf(-__bfloat162float(b[row * ldb + h])));
    } else {
      out0[i] = sp;
    }
    if (!DELTA && row == 0) out1[h] = -expf(param(A_log, h, A_fp32));
  }
}
}  // namespace

extern "C" int nsa_gates(const void* a, long lda, const void* b, long ldb, const void* bias, int bias_fp32, const void* A_log, int A_fp32,
                         float* out0, float* out1, long rows, int H, cudaStream_t st) {
  if (rows <= 0 || H <= 0) return nsa::fail(NSA_ERR_SHAPE, "gates: empty problem");
  const long blocks = (rows * H + 255) / 256, most = 16l * nsa::sm_count();
  auto* kernel = b ? gates_kernel<true> : gates_kernel<false>;
  kernel<<<static_cast<unsigned>(blocks < most ? blocks : most), 256, 0, st>>>((const bf16*)a, lda, (const bf16*)b, ldb, bias, bias_fp32, A_log, A_fp32,
                                                                               out0, out1, rows, H);
  nsa::count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : nsa::fail_cuda(e, "nsa_gates launch");
}
