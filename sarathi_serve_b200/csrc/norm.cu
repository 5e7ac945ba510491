// RMSNorm and residual-add + RMSNorm for [T, H] rows (HBM-bound row kernels).
//
// One CTA per token row.  The row is read once with 16-byte loads, held in
// registers across the block reduction and written once, so the kernel moves
// the algorithmic (2*T*H + H) * sizeof(T) bytes (4*T*H + H for the add variant).
// Semantics follow the reference kernel (csrc/layernorm_kernels.cu:10-35):
// sum of squares in fp32, inv = rsqrtf(var / H + eps), and the product
// x * inv is rounded to T BEFORE the multiply by the weight.
#include "common.cuh"

namespace sb200 {

constexpr int kNormMaxVec = 4;  // most 16-byte vectors cached per thread

// VEC: 16-byte vectors a thread holds, or 0 for the generic path.  Bound by memory, and by how many rows an SM has in flight.
// EARLY: the weights are loaded with the row, so that their latency hides behind its own; they then stay in registers over the
// reduction.  Good for up to two vectors and for a batch of at most a row per SM (64 rows of 24576: 4.5 -> 3.6 us); with
// more of both it costs the SM a resident row (8192 rows of 16384: 139 us against 96).
// early_next: let the next kernel start under this one.
template <typename T, bool ADD, int VEC, bool EARLY>
__global__ void __launch_bounds__(1024)
rms_norm_kernel(T* out, T* resid_out, const T* x, const T* resid,
                const T* w, float eps, int H, int early_next) {
  if (early_next) ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();
  __shared__ float red[33];
  constexpr int N = Vec16<T>::N;
  const int64_t row = blockIdx.x;
  const T* xr = x + row * H;
  const T* rr = ADD ? resid + row * H : nullptr;
  T* orow = out + row * H;
  T* zrow = ADD ? resid_out + row * H : nullptr;
  float ss = 0.f;

  if constexpr (VEC > 0) {
    Vec16<T> cache[VEC], wv[EARLY ? VEC : 1];
    const int nvec = H / N;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int v = i * blockDim.x + threadIdx.x;
      if (v < nvec) {
        cache[i] = ld16(xr + v * N);
        if constexpr (EARLY) wv[i] = ld16(w + v * N);
        if constexpr (ADD) {
          Vec16<T> r = ld16(rr + v * N);
#pragma unroll
          for (int j = 0; j < N; ++j)
            cache[i].v[j] = DT<T>::from_f(DT<T>::to_f(cache[i].v[j]) + DT<T>::to_f(r.v[j]));
          st16(zrow + v * N, cache[i]);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float f = DT<T>::to_f(cache[i].v[j]);
          ss += f * f;
        }
      }
    }
    ss = block_sum_once(ss, red);
    const float inv = rsqrtf(ss / (float)H + eps);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int v = i * blockDim.x + threadIdx.x;
      if (v < nvec) {
        Vec16<T> o, wi;
        if constexpr (EARLY) wi = wv[i];
        else wi = ld16(w + v * N);
#pragma unroll
        for (int j = 0; j < N; ++j)
          o.v[j] = DT<T>::from_f(rt<T>(DT<T>::to_f(cache[i].v[j]) * inv) * DT<T>::to_f(wi.v[j]));
        st16(orow + v * N, o);
      }
    }
  } else {
    // Generic path: any H / alignment; the row is re-read from L1/L2.
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
      float f = DT<T>::to_f(xr[i]);
      if constexpr (ADD) {
        f = rt<T>(f + DT<T>::to_f(rr[i]));
        zrow[i] = DT<T>::from_f(f);
      }
      ss += f * f;
    }
    ss = block_sum(ss, red);  // also orders the zrow writes before the re-read below
    const float inv = rsqrtf(ss / (float)H + eps);
    const T* src = ADD ? zrow : xr;
    for (int i = threadIdx.x; i < H; i += blockDim.x)
      orow[i] = DT<T>::from_f(rt<T>(DT<T>::to_f(src[i]) * inv) * DT<T>::to_f(w[i]));
  }
}

template <typename T, bool ADD>
static int launch_norm(void* out, void* resid_out, const void* x, const void* resid, const void* w,
                       float eps, int64_t T_, int64_t H, cudaStream_t s) {
  constexpr int N = Vec16<T>::N;
  bool vec = (H % N == 0) && aligned16(out) && aligned16(x) && aligned16(w) &&
             (!ADD || (aligned16(resid) && aligned16(resid_out)));
  int threads = 0, per = 1;
  if (vec) {
    const int64_t nvec = H / N;
    // fewest vectors per thread that keep the CTA at >= 128 threads when possible
    while (per < kNormMaxVec && (nvec + per - 1) / per > 512) ++per;
    int64_t t = (nvec + per - 1) / per;
    t = (t + 31) / 32 * 32;
    if (t > 1024) vec = false;
    threads = (int)t;
  }
  if (!vec) threads = (int)((H < 1024 ? (H + 31) / 32 * 32 : 1024));
  const bool few = T_ <= sm_count();
  // Signalling the next kernel takes 1.1 ns per CTA of the grid, whatever the CTA does (8192 rows of 64: 9.0 us against 6.0 without),
  // and CTAs that wait in the slots a row or two leave free unbalance the launch they belong to (512 rows of 5120 after one
  // another: 4.9 us against 4.4).  So only where a row is large enough to hide the first and fills the SM's threads, or the
  // batch is small.
  const int early_next = few || (vec && per <= 2 && threads >= 448) ? 1 : 0;
  auto kern = !vec ? rms_norm_kernel<T, ADD, 0, false> : per == 1 ? rms_norm_kernel<T, ADD, 1, true>
              : per == 2 ? rms_norm_kernel<T, ADD, 2, true>
              : per == 3 ? (few ? rms_norm_kernel<T, ADD, 3, true> : rms_norm_kernel<T, ADD, 3, false>)
                         : (few ? rms_norm_kernel<T, ADD, kNormMaxVec, true> : rms_norm_kernel<T, ADD, kNormMaxVec, false>);
  launch_dependent(kern, dim3((unsigned)T_), dim3((unsigned)threads), 0, s, (T*)out, (T*)resid_out, (const T*)x, (const T*)resid,
                   (const T*)w, eps, (int)H, early_next);
  SB_CHECK_LAUNCH("rms_norm_kernel");
  return SB200_OK;
}

}  // namespace sb200

using namespace sb200;

extern "C" int sb200_rms_norm(void* out, const void* x, const void* w, float eps, int64_t T, int64_t H,
                              int dtype, sb200_stream_t stream) {
  SB_CHECK_ARG(T >= 0 && H > 0 && H <= INT32_MAX && T <= INT32_MAX, "rms_norm: bad shape T=%lld H=%lld",
               (long long)T, (long long)H);
  if (T == 0) return SB200_OK;
  SB_CHECK_ARG(out && x && w, "rms_norm: null pointer");
  SB_DISPATCH_FLOAT(dtype, return (launch_norm<scalar_t, false>(out, nullptr, x, nullptr, w, eps, T, H,
                                                               (cudaStream_t)stream)));
  return SB200_OK;
}

extern "C" int sb200_fused_add_rms_norm(void* out, void* residual_out, const void* x, const void* residual,
                                        const void* w, float eps, int64_t T, int64_t H, int dtype,
                                        sb200_stream_t stream) {
  SB_CHECK_ARG(T >= 0 && H > 0 && H <= INT32_MAX && T <= INT32_MAX,
               "fused_add_rms_norm: bad shape T=%lld H=%lld", (long long)T, (long long)H);
  if (T == 0) return SB200_OK;
  SB_CHECK_ARG(out && residual_out && x && residual && w, "fused_add_rms_norm: null pointer");
  SB_CHECK_ARG(out != x && out != residual, "fused_add_rms_norm: out must not alias an input");
  SB_DISPATCH_FLOAT(dtype, return (launch_norm<scalar_t, true>(out, residual_out, x, residual, w, eps, T, H,
                                                              (cudaStream_t)stream)));
  return SB200_OK;
}
