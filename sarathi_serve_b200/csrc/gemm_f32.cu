// fp32 projections: C[M,N] = A[M,K] * B[N,K]^T (+bias) on the FMA pipes, fp32 products and sums.
//
// Bound: the FMA pipes (128 lanes per SM and clock; about 70 TFLOP/s).  Everything else is arranged so that they
// stay fed: a thread owns 8 x 8 outputs (4 x 8 in the 32-row tile), so one k-step costs a warp 64 FMA issue slots
// against four 16-byte shared-memory loads; products are issued as packed fma.rn.f32x2 (two IEEE fp32 FMAs per
// instruction, which leaves issue slots for those loads); the next k-tile travels global -> registers while the
// current one is multiplied, and lands in the other half of a double-buffered, k-major shared-memory tile.
// K is cut across the CTAs of a cluster when the output tiles alone do not fill the SMs evenly; the partial tiles
// meet in distributed shared memory and are added in the order of their k-ranges, so nothing leaves the chip, no
// workspace is shared between streams and the result does not depend on timing.
// Measured (B200, graph timeline): 288 x 5632 x 1024 in 91 us (36 TFLOP/s), 288 x 1536 x 1024 in 34 us; a whole fp32
// decoder layer of 288 tokens (hidden 1024, intermediate 2816) went from 971 to 247 us against 64 x 64 tiles of
// scalar 4 x 4 FMAs whose loads waited for one another.
#include "gemm_host.cuh"

namespace sb200 {

constexpr int kF32BN = 128, kF32BK = 16, kF32Threads = 128, kF32MaxSplit = 8;

__device__ __forceinline__ unsigned long long f32x2_dup(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ void f32x2_fma(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 f32x2_split(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// Four consecutive k of one row (zeros outside the matrix).  VEC: rows are 16-byte aligned and K is a multiple of 4.
template <bool VEC>
__device__ __forceinline__ float4 f32_load4(const float* p, int64_t ld, int row, int rows, int k, int K) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row < rows && k < K) {
    const float* q = p + (int64_t)row * ld + k;
    if (VEC) {
      v = *reinterpret_cast<const float4*>(q);
    } else {
      v.x = q[0];
      if (k + 1 < K) v.y = q[1];
      if (k + 2 < K) v.z = q[2];
      if (k + 3 < K) v.w = q[3];
    }
  }
  return v;
}

// Four consecutive output columns of one row.
__device__ __forceinline__ void f32_store4(float* C, int64_t ldc, const float* bias, int m, int n,
                                           int M, int N, float4 v, bool vec) {
  if (m >= M || n >= N) return;
  float* c = C + (int64_t)m * ldc + n;
  const float f[4] = {v.x, v.y, v.z, v.w};
  if (vec && n + 4 <= N) {
    float4 o = v;
    if (bias) { o.x += bias[n]; o.y += bias[n + 1]; o.z += bias[n + 2]; o.w += bias[n + 3]; }
    *reinterpret_cast<float4*>(c) = o;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) c[j] = f[j] + (bias ? bias[n + j] : 0.f);
  }
}

// Grid (n tiles, m tiles, k parts); the k parts of a tile are one cluster.
// Warps: 2 x 2 over the BM x 128 tile; in a warp, lane = 8 * ty + tx covers rows ty*4 (+ 16) and columns tx*4 (+ 32).
template <int BM, bool VEC>
__global__ void __launch_bounds__(kF32Threads, 3)
gemm_f32_kernel(float* C, int64_t ldc, const float* A, int64_t lda,
                const float* B, int64_t ldb, const float* bias, int M, int N, int K, int vec_c) {
  constexpr int TM = BM / 8, LDA = BM + 4, LDB = kF32BN + 4;  // (+4: the transposing stores conflict two ways at most)
  constexpr int A_LD = BM / 32, B_LD = kF32BN / 32;           // 16-byte loads per thread and k-tile
  constexpr int kTile = kF32BK * (LDA + LDB);
  constexpr int kSmem = 2 * kTile > BM * kF32BN ? 2 * kTile : BM * kF32BN;
  __shared__ __align__(16) float sm[kSmem];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane & 7, ty = lane >> 3;
  const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * 64;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * kF32BN;
  const int S = gridDim.z, part = blockIdx.z;
  const int kt_all = (K + kF32BK - 1) / kF32BK;
  const int kt0 = (int)((unsigned)kt_all * (unsigned)part / (unsigned)S), kt1 = (int)((unsigned)kt_all * (unsigned)(part + 1) / (unsigned)S);
  const int lrow = tid >> 2, lk = (tid & 3) * 4;
  grid_dependency_begin();

  unsigned long long acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  float4 ra[A_LD], rb[B_LD];
  auto fetch = [&](int kt) {
    const int k = kt * kF32BK + lk;
#pragma unroll
    for (int i = 0; i < A_LD; ++i) ra[i] = f32_load4<VEC>(A, lda, m0 + lrow + 32 * i, M, k, K);
#pragma unroll
    for (int i = 0; i < B_LD; ++i) rb[i] = f32_load4<VEC>(B, ldb, n0 + lrow + 32 * i, N, k, K);
  };
  auto park = [&](int buf) {
    float* sa = sm + buf * kTile;
    float* sb = sa + kF32BK * LDA;
#pragma unroll
    for (int i = 0; i < A_LD; ++i) {
      const int r = lrow + 32 * i;
      sa[(lk + 0) * LDA + r] = ra[i].x; sa[(lk + 1) * LDA + r] = ra[i].y;
      sa[(lk + 2) * LDA + r] = ra[i].z; sa[(lk + 3) * LDA + r] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < B_LD; ++i) {
      const int r = lrow + 32 * i;
      sb[(lk + 0) * LDB + r] = rb[i].x; sb[(lk + 1) * LDB + r] = rb[i].y;
      sb[(lk + 2) * LDB + r] = rb[i].z; sb[(lk + 3) * LDB + r] = rb[i].w;
    }
  };
  if (kt0 < kt1) {
    fetch(kt0);
    park(0);
  }
  __syncthreads();
  for (int kt = kt0; kt < kt1; ++kt) {
    const int buf = (kt - kt0) & 1;
    if (kt + 1 < kt1) fetch(kt + 1);
    const float* sa = sm + buf * kTile + wm + ty * 4;
    const float* sb = sm + buf * kTile + kF32BK * LDA + wn + tx * 4;
#pragma unroll
    for (int k = 0; k < kF32BK; ++k) {
      float a[TM];
#pragma unroll
      for (int h = 0; h < TM / 4; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(sa + k * LDA + h * 16);
        a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
      }
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(sb + k * LDB);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(sb + k * LDB + 32);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned long long ai = f32x2_dup(a[i]);
        f32x2_fma(acc[i][0], ai, b0.x);
        f32x2_fma(acc[i][1], ai, b0.y);
        f32x2_fma(acc[i][2], ai, b1.x);
        f32x2_fma(acc[i][3], ai, b1.y);
      }
    }
    if (kt + 1 < kt1) park(buf ^ 1);
    __syncthreads();
  }

  if (S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + wm + ty * 4 + (i >> 2) * 16 + (i & 3);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 lo = f32x2_split(acc[i][2 * h]), hi = f32x2_split(acc[i][2 * h + 1]);
        f32_store4(C, ldc, bias, m, n0 + wn + tx * 4 + h * 32, M, N, make_float4(lo.x, lo.y, hi.x, hi.y), vec_c != 0);
      }
    }
    return;
  }
  // the k-parts meet: every CTA parks its partial tile (the last __syncthreads above freed the buffers), then sums
  // its share of the tile's 16-byte groups over all parts, in part order
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = wm + ty * 4 + (i >> 2) * 16 + (i & 3);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 lo = f32x2_split(acc[i][2 * h]), hi = f32x2_split(acc[i][2 * h + 1]);
      *reinterpret_cast<float4*>(sm + r * kF32BN + wn + tx * 4 + h * 32) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  }
  ptx::cluster_sync_all();
  const int groups = BM * kF32BN / 4, share = (groups + S - 1) / S;
  const int g1 = min(groups, (part + 1) * share);
  for (int g = part * share + tid; g < g1; g += kF32Threads) {
    const uint32_t addr = ptx::smem_u32(sm + 4 * g);
    float4 v[kF32MaxSplit];
#pragma unroll
    for (int p = 0; p < kF32MaxSplit; ++p)
      if (p < S)
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[p].x), "=f"(v[p].y), "=f"(v[p].z), "=f"(v[p].w) : "r"(ptx::map_to_cta(addr, (uint32_t)p)) : "memory");
    float4 s = v[0];
#pragma unroll
    for (int p = 1; p < kF32MaxSplit; ++p)
      if (p < S) { s.x += v[p].x; s.y += v[p].y; s.z += v[p].z; s.w += v[p].w; }
    f32_store4(C, ldc, bias, m0 + g / (kF32BN / 4), n0 + (g % (kF32BN / 4)) * 4, M, N, s, vec_c != 0);
  }
  ptx::cluster_sync_all();  // no CTA leaves while another still reads its partial tile
}

// K parts per tile: the split whose busiest SM has the least to do.  One block alone on an SM (one warp per
// scheduler) keeps the FMA pipes about 70 % busy, two or more about 90 %.
static int f32_split(int64_t tiles, int k_tiles, int bm) {
  const double sms = sm_count();
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= kF32MaxSplit && s <= k_tiles; ++s) {
    if (s > 1 && k_tiles / s < 4) break;  // a part shorter than the prologue and the exchange
    const int64_t per_sm = (int64_t)((tiles * s + (int64_t)sms - 1) / (int64_t)sms);
    const double work = (double)((k_tiles + s - 1) / s) * kF32BK * bm + 1200.0 + (s > 1 ? 1500.0 : 0.0);
    const double cost = (double)per_sm * work / (per_sm == 1 ? 0.7 : 0.9);
    if (cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

template <int BM>
static int launch_f32(float* C, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb, const float* bias,
                      int M, int N, int K, cudaStream_t s) {
  const int64_t nt = ((int64_t)N + kF32BN - 1) / kF32BN, mt = ((int64_t)M + BM - 1) / BM;
  SB_CHECK_ARG(mt <= 65535, "fp32 projection: %d rows are more than one launch covers", M);
  const int split = f32_split(nt * mt, (K + kF32BK - 1) / kF32BK, BM);
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldb % 4 == 0 && aligned16(A) && aligned16(B);
  const int vec_c = ldc % 4 == 0 && aligned16(C) ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nt, (unsigned)mt, (unsigned)split);
  cfg.blockDim = dim3(kF32Threads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)split;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (vec) SB_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BM, true>, C, ldc, A, lda, B, ldb, bias, M, N, K, vec_c));
  else SB_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BM, false>, C, ldc, A, lda, B, ldb, bias, M, N, K, vec_c));
  return SB200_OK;
}

int run_gemm_f32(float* C, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb, const float* bias,
                 int M, int N, int K, cudaStream_t s) {
  // rows of a tile: 32 for the small batches a 64-row tile would pad by half or more
  if (M <= 32) return launch_f32<32>(C, ldc, A, lda, B, ldb, bias, M, N, K, s);
  return launch_f32<64>(C, ldc, A, lda, B, ldb, bias, M, N, K, s);
}

}  // namespace sb200
