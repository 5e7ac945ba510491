// Projections with at most 16 output columns (the router gate of a mixture-of-experts block): out[t, n] = x[t, :] . w[n, :].
//
// Bound: latency, then one read of x (8 MB for 1024 tokens of 4096: about 1.3 us).  A tensor-core tile would be mostly
// padding and its few CTAs would walk all of K one k-block after the other, so this is a dot-product kernel: a CTA takes
// ROWS tokens and all columns, its eight warps cut K into interleaved slices of 256 elements, a lane keeps
// ROWS x 8 fp32 sums of its 16-byte pieces (every loaded weight is used for ROWS tokens, every loaded activation for
// eight columns), and the sums meet in registers and shared memory in a fixed order.
#include "gemm_host.cuh"

namespace sb200 {

constexpr int kNarrowMaxCols = 16, kNarrowWarps = 8;

template <typename T, int ROWS>
__global__ void __launch_bounds__(kNarrowWarps * 32)
gemm_narrow_kernel(const T* x, int64_t ldx, const T* w, int64_t ldw, const GemmArgs g) {
  __shared__ float part[kNarrowWarps][ROWS * 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * ROWS, n0 = blockIdx.y * 8;
  grid_dependency_begin();
  float acc[ROWS][8];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int n = 0; n < 8; ++n) acc[r][n] = 0.f;
  for (int k = (warp * 32 + lane) * 8; k < g.K; k += kNarrowWarps * 256) {  // (K is a multiple of 8)
    Vec16<T> xv[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      xv[r].raw = make_uint4(0, 0, 0, 0);
      if (t0 + r < g.M) xv[r] = ld16(x + (int64_t)(t0 + r) * ldx + k);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      Vec16<T> wv;
      wv.raw = make_uint4(0, 0, 0, 0);
      if (n0 + n < g.N) wv = ld16(w + (int64_t)(n0 + n) * ldw + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float wf = DT<T>::to_f(wv.v[j]);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r][n] = fmaf(DT<T>::to_f(xv[r].v[j]), wf, acc[r][n]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const float s = warp_sum(acc[r][n]);
      if (lane == 0) part[warp][r * 8 + n] = s;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS * 8; i += kNarrowWarps * 32) {
    const int t = t0 + i / 8, n = n0 + i % 8;
    if (t >= g.M || n >= g.N) continue;
    float a = 0.f;
#pragma unroll
    for (int v = 0; v < kNarrowWarps; ++v) a += part[v][i];
    if (g.bias) a += DT<T>::to_f(reinterpret_cast<const T*>(g.bias)[n]);
    if (g.residual) a = DT<T>::to_f(reinterpret_cast<const T*>(g.residual)[(int64_t)t * g.ldr + n]) + rt<T>(a);
    reinterpret_cast<T*>(g.out)[(int64_t)t * g.ldo + n] = DT<T>::from_f(a);
  }
}

// Tokens of a CTA: eight reuse the weights most; two while that still leaves SMs without a CTA.
static int narrow_rows(int64_t M) { return M <= 2 * sm_count() ? 2 : 8; }

template <typename T>
static cudaError_t launch_narrow(const void* x, int64_t ldx, const void* w, int64_t ldw, const GemmArgs& g, cudaStream_t s) {
  const int rows = narrow_rows(g.M);
  const dim3 grid((unsigned)((g.M + rows - 1) / rows), (unsigned)((g.N + 7) / 8)), block(kNarrowWarps * 32);
  return launch_dependent(rows == 2 ? gemm_narrow_kernel<T, 2> : gemm_narrow_kernel<T, 8>, grid, block, 0, s, (const T*)x, ldx,
                          (const T*)w, ldw, g);
}

// An SM holds one CTA of eight tokens, so the time goes in rounds of 148 of them (8 columns, K = 4096: 1184 tokens 6.1 us, 1200
// 10.8, 2400 15.8, 4096 21 us), while the tensor-core kernels take 10 to 12 us for all of these: one round, and a second where
// K is long enough to make theirs slow and short enough to keep this one fast (1200 tokens, K = 512: 5.7 us against 5.2,
// 1024: 5.9 / 10.4, 4096: 10.8 / 11.5, 6144: 13.8 / 12.3 us).
bool narrow_fits(int epi, int64_t M, int64_t N, int64_t K) {
  // (K beyond 16384: 200 tokens x 16 x 28672 took 39 us here, 28 on the tensor cores; x 14336 20.6 and 20.1)
  if (epi != EPI_STORE || N > kNarrowMaxCols || K % 8 || K > 16384) return false;
  const int rows = narrow_rows(M);
  const int64_t ctas = (M + rows - 1) / rows * ((N + 7) / 8), sms = sm_count();
  return rows == 2 || ctas <= sms || (ctas <= 2 * sms && K >= 1024 && K <= 4096);
}

int run_gemm_narrow(int dtype, int epi, const void* x, int64_t ldx, const void* w, int64_t ldw, const GemmArgs& g,
                    cudaStream_t s, bool* done) {
  // rows that the 16-byte loads can read; anything else is left to the tensor-core kernel, which also words the errors
  *done = narrow_fits(epi, g.M, g.N, g.K) && (dtype == SB200_BF16 || dtype == SB200_F16) && ldx >= g.K && ldw >= g.K &&
          ldx % 8 == 0 && ldw % 8 == 0 && aligned16(x) && aligned16(w);
  if (!*done) return SB200_OK;
  SB_CUDA(dtype == SB200_BF16 ? launch_narrow<__nv_bfloat16>(x, ldx, w, ldw, g, s) : launch_narrow<__half>(x, ldx, w, ldw, g, s));
  return SB200_OK;
}

}  // namespace sb200
