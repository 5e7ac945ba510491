// Projections with the roles of the operands swapped against gemm_sm100.cuh: out[t, n] = x[t, :] . w[n, :] with 128 weight
// rows as the M side of an MMA (the A operand) and up to 256 tokens as its N side, which goes in steps of 16.
//
// What that is good for:
//   * Small batches are bound by the weights, each read from HBM once.  A stage of the ring is almost all weights (16 KiB
//     per accumulator against 128 bytes per token; on the M side the tokens would take a 128-row box), an accumulator
//     column is one token, and all epilogue warps have outputs to finish instead of the one with rows to store.
//   * Ragged batches pay for the tokens they have, not for multiples of 128 or 256 rows, and the number of tiles can be
//     chosen to fill whole rounds of the 148 SMs.
// How:
//   * NACC = 2 accumulators per CTA share the tokens of a stage: gate and up rows (EPI_SILU_MUL), the first and the second
//     halves of 128 / (head_size / 2) heads (EPI_ROTARY), so that the two values a thread combines sit in the same
//     lane.  EPI_STORE has one accumulator; two (256 columns) only by explicit configuration, for the autotuner.
//   * Few tiles: K is cut over a cluster of `split` CTAs.  Every CTA sends the others the tokens they finish through
//     distributed shared memory and sums its own tokens in the order of the k-ranges: no workspace, nothing that two
//     streams could share, and a result that does not depend on timing.
//   * Many tiles: CTAs walk the tiles round-robin and the loads run on across tile boundaries; two sets of accumulators
//     when they fit TMEM, so that a tile is finished under the next one's main loop.
//   * EW = 4 epilogue warps and half an SM's shared memory for small batches: under programmatic dependent launch the
//     next projection's CTAs are resident while this one drains, and before they wait for its results they ask for
//     their first weights -- into the L2 only, where a late write to the weights by an earlier kernel is still seen.
//     EW = 8 and the whole SM otherwise.
#include <atomic>

#include "gemm_host.cuh"

namespace sb200 {

constexpr int kSwapStages = 8;
constexpr int kSwapTileBytes = 128 * kBK * 2;  // one accumulator's weights of a stage

// 32 lanes x 16 consecutive TMEM columns.
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, float* f) {
  uint32_t r[16];
  __syncwarp();  // .aligned
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(r[j]);
}

// First weight row of box j of accumulator `acc` in a tile (g.N or more: nothing to load).
template <int EPI, int NACC>
__device__ __forceinline__ int swap_w_row(const GemmArgs& g, int tile, int acc, int j) {
  if (EPI == EPI_SILU_MUL) return acc * (g.N / 2) + tile * 128;
  if (EPI == EPI_ROTARY) {
    const int row = tile * 256 + j * g.head_size;
    return row < g.N ? row + acc * (g.head_size / 2) : g.N;
  }
  return (tile * NACC + acc) * 128;
}

// Finish tokens t0 .. t0 + n - 1 (n <= 16) of this thread's column(s): a[j] (and b[j]) are their fp32 sums.  The
// arithmetic and its roundings are those of finish_unit in gemm_sm100.cuh.  Called by all lanes of a warp; everything a
// token needs from memory is requested for all of them before the first store (token by token, the two dependent loads
// of a rotation alone cost 1200 clocks each time).
template <typename T, int EPI>
__device__ __forceinline__ void swap_finish(const GemmArgs& g, int t0, int n, int col, const float* a, const float* b) {
  const int lane = threadIdx.x & 31;
  T* out = reinterpret_cast<T*>(g.out) + (int64_t)t0 * g.ldo + col;
  if constexpr (EPI == EPI_STORE) {
    const bool ok = col < g.N;
    const float bias = g.bias && ok ? DT<T>::to_f(reinterpret_cast<const T*>(g.bias)[col]) : 0.f;
    if (g.residual) {
      const T* res = reinterpret_cast<const T*>(g.residual) + (int64_t)t0 * g.ldr + col;
      float r[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = j < n && ok ? DT<T>::to_f(res[(int64_t)j * g.ldr]) : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < n && ok) out[(int64_t)j * g.ldo] = DT<T>::from_f(r[j] + rt<T>(g.bias ? a[j] + bias : a[j]));
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < n && ok) out[(int64_t)j * g.ldo] = DT<T>::from_f(g.bias ? a[j] + bias : a[j]);
    }
  } else if constexpr (EPI == EPI_SILU_MUL) {
    const bool ok = col < g.N / 2;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (j < n) {
        const float gte = rt<T>(a[j]), up = rt<T>(b[j]);
        const float v = rt<T>(gte / (1.0f + expf(-gte))) * up;
        if (ok) out[(int64_t)j * g.ldo] = DT<T>::from_f(v);
      }
    }
  } else {
    const bool ok = col < g.N;
    const int half = g.head_size / 2, in_head = col & (g.head_size - 1);  // (head sizes are powers of two)
    const bool rotate = col - in_head < g.rot_cols;                       // the same for the lanes of a warp
    float co[16], si[16];
    if (rotate) {
      const long long pos = lane < n ? g.positions[t0 + lane] : 0;
      const T* cs = reinterpret_cast<const T*>(g.cos_sin) + in_head;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const T* p = cs + __shfl_sync(0xffffffffu, pos, j) * g.head_size;
        co[j] = j < n ? DT<T>::to_f(p[0]) : 0.f;
        si[j] = j < n ? DT<T>::to_f(p[half]) : 0.f;
      }
    }
    const int c = col - g.q_cols;
    const bool kv = g.kv_cache && c >= 0 && c < 2 * g.kv_cols;  // k and v heads: see store_kv32
    long long slot = -1;
    if (kv && lane < n) slot = g.kv_slots[t0 + lane];
    T* cache = reinterpret_cast<T*>(g.kv_cache) + (c < g.kv_cols ? c : (int64_t)g.kv_page_size * g.kv_cols + (c - g.kv_cols));
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float x = rt<T>(a[j]), y = rt<T>(b[j]);
      const T xo = DT<T>::from_f(rotate ? rt<T>(x * co[j]) - rt<T>(y * si[j]) : x);
      const T yo = DT<T>::from_f(rotate ? rt<T>(y * co[j]) + rt<T>(x * si[j]) : y);
      const long long s = kv ? __shfl_sync(0xffffffffu, slot, j) : -1;
      if (j < n && ok) {
        out[(int64_t)j * g.ldo] = xo;
        out[(int64_t)j * g.ldo + half] = yo;
        if (s >= 0) {
          cache[s * (int64_t)g.kv_cols] = xo;
          cache[s * (int64_t)g.kv_cols + half] = yo;
        }
      }
    }
  }
}

template <typename T, int EPI, int NACC, int EW>
__global__ void __launch_bounds__(64 + 32 * EW)
gemm_swap_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                 const __grid_constant__ CUtensorMap tmap_xt, const __grid_constant__ GemmArgs g,
                 const __grid_constant__ SwapPlan p) {
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp-uniform
  const int S = p.split, stages = p.stages, tiles = p.w_tiles * p.t_tiles;
  const int part = S > 1 ? (int)ptx::cluster_ctarank() : 0;
  const int first_tile = S > 1 ? (int)blockIdx.x / S : (int)blockIdx.x;
  const int tile_step = S > 1 ? tiles : (int)gridDim.x;
  const int kb0 = (int)((unsigned)p.k_blocks * (unsigned)part / (unsigned)S);  // (K < 2^31: at most 2^25 k-blocks, times 8)
  const int kb1 = (int)((unsigned)p.k_blocks * (unsigned)(part + 1) / (unsigned)S);
  const int stage_bytes = NACC * kSwapTileBytes + p.act_rows * kBK * 2;
  const bool dbuf = 2 * NACC * p.nt <= p.tmem_cols;
  const int box_rows = EPI == EPI_ROTARY ? g.head_size / 2 : 128, boxes = EPI == EPI_ROTARY ? 128 >> p.half_shift : 1;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[kSwapStages], empty_bar[kSwapStages], tmem_full[2], tmem_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { ptx::mbar_init(&full_bar[s], 1); ptx::mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { ptx::mbar_init(&tmem_full[b], 1); ptx::mbar_init(&tmem_empty[b], EW); }
    abort_word = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
    ptx::prefetch_tensormap(&tmap_xt);
  }
  if (warp == 1) { ptx::tmem_alloc(&tmem_slot, (uint32_t)p.tmem_cols); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  // TMEM is ours: kernels that start from here on cannot take it from a CTA this kernel still has to start
  ptx::grid_launch_dependents();

  __syncwarp();  // the roles start from converged warps
  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    const int pf1 = min(kb1, kb0 + p.prefetch);
    if (ptx::elect_one()) {
      for (int kb = kb0; kb < pf1; ++kb)
#pragma unroll
        for (int a = 0; a < NACC; ++a)
          for (int j = 0; j < boxes; ++j) {
            const int row = swap_w_row<EPI, NACC>(g, first_tile / p.t_tiles, a, j);
            if (row < g.N) ptx::tma_prefetch_l2_2d(&tmap_w, kb * kBK, row);
          }
    }
    __syncwarp();
    ptx::grid_dependency_wait();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < tiles; tile += tile_step) {
      const int wt = tile / p.t_tiles, t_first = (tile - wt * p.t_tiles) * p.nt;
      // the last token tile has a box of its own: box rows outside the tensor cost more time than rows inside it
      const bool last = t_first + p.nt >= g.M;
      uint32_t bytes = (uint32_t)((last ? (g.M - t_first + 7) & ~7 : p.act_rows) * kBK * 2);
#pragma unroll
      for (int a = 0; a < NACC; ++a)
        for (int j = 0; j < boxes; ++j)
          if (swap_w_row<EPI, NACC>(g, wt, a, j) < g.N) bytes += (uint32_t)(box_rows * kBK * 2);
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = ptx::mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag) && ok;
        if (ptx::elect_one() && ok) {
          uint8_t* sw = smem + (size_t)stage * stage_bytes;
          ptx::mbar_expect_tx(&full_bar[stage], bytes);
#pragma unroll
          for (int a = 0; a < NACC; ++a)
            for (int j = 0; j < boxes; ++j) {
              const int row = swap_w_row<EPI, NACC>(g, wt, a, j);
              uint8_t* dst = sw + a * kSwapTileBytes + j * box_rows * (kBK * 2);
              if (row >= g.N) continue;
              if (p.t_tiles == 1) ptx::tma_load_2d_once(dst, &tmap_w, &full_bar[stage], kb * kBK, row);
              else ptx::tma_load_2d(dst, &tmap_w, &full_bar[stage], kb * kBK, row);
            }
          ptx::tma_load_2d(sw + NACC * kSwapTileBytes, last ? &tmap_xt : &tmap_x, &full_bar[stage], kb * kBK, t_first);
        }
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
      ok = __all_sync(0xffffffffu, ok ? 1 : 0) != 0;
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    ptx::grid_dependency_wait();  // (nothing it reads needs this: the time limits of its waits start here)
    const uint32_t idesc = ptx::make_idesc(DT<T>::id == SB200_BF16 ? 1 : 0, p.nt, 128);
    int stage = 0, used = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < tiles; tile += tile_step, ++used) {
      const int buf = dbuf ? (used & 1) : 0;
      const uint32_t use = (uint32_t)(dbuf ? (used >> 1) : used);
      if (!ptx::mbar_wait_warp(&tmem_empty[buf], (use & 1u) ^ 1u, abort_flag)) break;
      ptx::tc_fence_after();
      const uint32_t d_tmem = tmem_base + (uint32_t)(buf * NACC * p.nt);
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = ptx::mbar_wait(&full_bar[stage], phase, abort_flag) && ok;
        ptx::tc_fence_after();
        if (ptx::elect_one() && ok) {
          const uint32_t sw = ptx::smem_u32(smem + (size_t)stage * stage_bytes);
          const uint64_t dx = ptx::make_smem_desc_sw128(sw + NACC * kSwapTileBytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
#pragma unroll
            for (int a = 0; a < NACC; ++a)
              ptx::umma_f16(d_tmem + (uint32_t)(a * p.nt), ptx::make_smem_desc_sw128(sw + a * kSwapTileBytes) + (uint64_t)(k * 2),
                            dx + (uint64_t)(k * 2), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          ptx::umma_commit(&empty_bar[stage]);
        }
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
      ok = __all_sync(0xffffffffu, ok ? 1 : 0) != 0;
      if (ok && ptx::elect_one()) ptx::umma_commit(&tmem_full[buf]);
      __syncwarp();
    }
  }
  __syncwarp();

  // ---------------------------------------------------------------- epilogue
  const int q = warp & 3;                // TMEM lane quarter this warp may read
  const int hsel = EW == 8 ? (warp - 2) >> 2 : 0;  // two warps of a quarter take the 16-token chunks in turn
  constexpr int kChunkStep = 16 * (EW / 4);
  const int l = q * 32 + lane;           // accumulator lane = weight row inside the tile
  const uint32_t tmem_row = tmem_base + ((uint32_t)(q * 32) << 16);
  auto column = [&](int wt) {            // this thread's (first) output column
    if (EPI == EPI_ROTARY) return wt * 256 + (l >> p.half_shift) * g.head_size + (l & (box_rows - 1));
    return wt * 128 * (EPI == EPI_STORE ? NACC : 1) + l;
  };
  auto finish = [&](int t, int n, int col, const float* a, const float* b) {
    swap_finish<T, EPI>(g, t, n, col, a, b);
    if constexpr (EPI == EPI_STORE && NACC == 2) swap_finish<T, EPI>(g, t, n, col + 128, b, b);
  };
  if (S == 1) {
    if (warp >= 2) {
      ptx::grid_dependency_wait();
      int used = 0;
      for (int tile = first_tile; tile < tiles; tile += tile_step, ++used) {
        const int buf = dbuf ? (used & 1) : 0;
        const uint32_t use = (uint32_t)(dbuf ? (used >> 1) : used);
        if (!ptx::mbar_wait_warp(&tmem_full[buf], use & 1u, abort_flag)) break;
        ptx::tc_fence_after();
        const int wt = tile / p.t_tiles, t_first = (tile - wt * p.t_tiles) * p.nt, m = min(p.nt, g.M - t_first);
        const int col = column(wt);
        const uint32_t src = tmem_row + (uint32_t)(buf * NACC * p.nt);
        for (int t0 = hsel * 16; t0 < m; t0 += kChunkStep) {
          float a[16], b[16];
          tmem_ld_32x16(src + (uint32_t)t0, a);
          if (NACC == 2) tmem_ld_32x16(src + (uint32_t)(p.nt + t0), b);
          finish(t_first + t0, min(16, m - t0), col, a, b);
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&tmem_empty[buf]);
      }
    }
  } else {
    // K split over the cluster: of the tile's m tokens CTA r finishes [m r / S, m (r + 1) / S).  The rings are free once
    // every CTA's MMAs are complete (first cluster barrier) and take [source][token][accumulator][128] fp32 partials.
    bool ok = true;
    if (warp >= 2) {
      ptx::grid_dependency_wait();
      ok = ptx::mbar_wait_warp(&tmem_full[0], 0u, abort_flag);
      ptx::tc_fence_after();
    }
    __syncthreads();
    ptx::cluster_sync_all();
    const int wt = first_tile / p.t_tiles, t_first = (first_tile - wt * p.t_tiles) * p.nt, m = min(p.nt, g.M - t_first);
    const int my0 = m * part / S, my1 = m * (part + 1) / S, cap = (m + S - 1) / S;
    if (warp >= 2 && ok) {
      const uint32_t mine = ptx::smem_u32(smem) + (uint32_t)(part * cap * NACC * 512 + l * 4);
      int owner = 0, o0 = 0, o1 = m / S;  // tokens [o0, o1) of the tile belong to `owner`
      for (int t0 = hsel * 16; t0 < m; t0 += kChunkStep) {
        float a[16], b[16];
        tmem_ld_32x16(tmem_row + (uint32_t)t0, a);
        if (NACC == 2) tmem_ld_32x16(tmem_row + (uint32_t)(p.nt + t0), b);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int t = t0 + j;
          if (t < m) {
            while (t >= o1) { ++owner; o0 = o1; o1 = m * (owner + 1) / S; }
            const uint32_t dst = ptx::map_to_cta(mine + (uint32_t)((t - o0) * NACC * 512), (uint32_t)owner);
            ptx::st_shared_cluster_f32(dst, a[j]);
            if (NACC == 2) ptx::st_shared_cluster_f32(dst + 512, b[j]);
          }
        }
      }
    }
    __syncwarp();
    ptx::cluster_sync_all();  // the partials have landed; from here on a CTA touches only its own shared memory
    if (warp >= 2 && ok) {
      const int col = column(wt);
      const float* in = reinterpret_cast<const float*>(smem) + l;
      for (int t0 = my0 + hsel * 16; t0 < my1; t0 += kChunkStep) {
        const int n = min(16, my1 - t0);
        float a[16], b[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] = b[j] = 0.f;
        for (int s = 0; s < S; ++s) {
          const float* v = in + (size_t)((s * cap + (t0 - my0)) * NACC) * 128;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < n) {
              a[j] += v[j * NACC * 128];
              if (NACC == 2) b[j] += v[j * NACC * 128 + 128];
            }
        }
        finish(t_first + t0, n, col, a, b);
      }
    }
  }

  // -------------------------------------------------------------- common exit
  __syncwarp();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
  if (abort_word && threadIdx.x == 0 && g.status) atomicCAS(g.status, 0u, (uint32_t)CS_TIMEOUT_MBARRIER);
}

// ------------------------------------------------------------------- planning
// Clusters of `split` CTAs that run at once, as the runtime reports them.  A cluster has to fit inside one GPC, so these
// are fewer CTAs than there are SMs, and the tiles beyond them wait for a second round that costs as much as the first
// (18 clusters of eight, 24 of six: qkv of a TP=8 rank, 512 tokens, took 30 us against 21 in the general kernel).
static int swap_clusters(int split, int ew) {
  static std::atomic<int> cache[16][2][9];  // [device][ew][split]; 0 = not asked yet
  int dev = 0;
  if (split < 2 || split > 8) return sm_count();
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) {  // planning without a device: as max_coresident_clusters
    (void)cudaGetLastError();
    return sm_count() / split * 3 / 4;
  }
  std::atomic<int>& c = cache[dev][ew == 4 ? 0 : 1][split];
  int n = c.load(std::memory_order_relaxed);
  if (n > 0) return n;
  // (the dynamic shared memory decides; the other epilogues' kernels differ in registers only)
  const void* kern = ew == 4 ? (const void*)gemm_swap_kernel<__nv_bfloat16, EPI_STORE, 1, 4> : (const void*)gemm_swap_kernel<__nv_bfloat16, EPI_STORE, 1, 8>;
  const int smem = (ew == 4 ? kSwapHalfRing : kSwapRing) + 2048;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sm_count() / split * split));
  cfg.blockDim = dim3((unsigned)(64 + 32 * ew));
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = 1;  // not answered: no tile is cut
  }
  c.store(n, std::memory_order_relaxed);
  return n;
}

// A plan for `nacc` accumulators, t_tiles token tiles and `split` CTAs per tile; false when it does not fit.
static bool swap_plan(int64_t M, int64_t N, int64_t K, int head_size, int nacc, int t_tiles, int split, SwapPlan* p) {
  const int sms = sm_count();
  const int64_t per = (M + t_tiles - 1) / t_tiles;
  const int64_t nt = (per + 15) / 16 * 16;
  if (nt > 256 || nacc * nt > 512 || (int64_t)(t_tiles - 1) * nt >= M) return false;
  p->nacc = nacc;
  p->nt = (int)nt;
  p->t_tiles = t_tiles;
  p->w_tiles = (int)((N + 128 * nacc - 1) / (128 * nacc));
  p->k_blocks = (int)((K + kBK - 1) / kBK);
  p->split = split;
  const int64_t tiles = (int64_t)p->w_tiles * t_tiles;
  if (tiles * split > INT32_MAX || split < 1 || split > 8 || split > p->k_blocks) return false;
  p->grid = (int)(split > 1 ? tiles * split : tiles < sms ? tiles : sms);
  p->act_rows = t_tiles == 1 ? (int)((M + 7) / 8 * 8) : (int)nt;
  p->half_shift = head_size == 64 ? 5 : head_size == 128 ? 6 : 7;
  const int stage = nacc * kSwapTileBytes + p->act_rows * kBK * 2;
  // Half an SM (and four epilogue warps) where that still holds three stages and two launches' accumulators, so that the
  // next launch finds room; otherwise the whole SM.
  p->ew = kSwapHalfRing / stage >= 3 && M <= 64 ? 4 : 8;
  p->stages = (p->ew == 4 ? kSwapHalfRing : kSwapRing) / stage;
  if (p->stages > kSwapStages) p->stages = kSwapStages;
  if (p->stages < 2) return false;
  // the exchange of a split tile lives in the ring
  if (split > 1 && (int64_t)split * ((nt + split - 1) / split) * nacc * 512 > (int64_t)p->stages * stage) return false;
  int cols = nacc * p->nt;
  if (split == 1 && tiles > p->grid && 2 * cols <= (p->ew == 4 ? 256 : 512)) cols *= 2;
  p->tmem_cols = 32;
  while (p->tmem_cols < cols) p->tmem_cols *= 2;
  // requested ahead: what HBM delivers while the kernels before this one end
  const int64_t pf = kSwapPrefetchBytes / ((int64_t)p->grid * nacc * kSwapTileBytes);
  p->prefetch = p->ew == 4 ? (int)(pf < 1 ? 1 : pf > 64 ? 64 : pf) : 0;
  return true;
}

// Estimated SM clocks.  The constants are fitted to the kernel's times over 8 .. 2048 tokens of the projections of 8B and
// 70B layers, whole and at 1/8 of the width (most within 15 %).
static double swap_per_kb(int epi, const SwapPlan& p) {
  const int sms = sm_count();
  const double stage = p.nacc * kSwapTileBytes + p.act_rows * kBK * 2;
  double per_kb = 4.0 * p.nacc * (p.nt / 2 > 46 ? p.nt / 2 : 46);  // tensor pipe
  double feed = gemm_feed_rate(p.grid < sms ? p.grid : sms);
  if (p.nacc == 2 && feed > 60.0) feed = 60.0;                     // three to five boxes a stage
  if (stage / feed > per_kb) per_kb = stage / feed;
  if (per_kb < 430.0) per_kb = 430.0;                              // issue
  if (epi == EPI_ROTARY) per_kb += 1.5 * p.nt;                     // measured: 16 k-blocks of 160 tokens 27 us, 64 of 176 52
  return per_kb;
}

static double swap_cost(int epi, int64_t N, int64_t K, const SwapPlan& p) {
  double per_kb = swap_per_kb(epi, p);
  if (p.stages <= 3) per_kb *= 1.2;                                // too shallow to hide a load
  const double chunks = p.nt / 16, warps = p.ew / 4;
  const double finish = 600.0 + chunks / warps * (epi == EPI_SILU_MUL ? 900.0 : epi == EPI_ROTARY ? 3000.0 : 350.0 * p.nacc);
  const int64_t tiles = (int64_t)p.w_tiles * p.t_tiles;
  double c = 6000.0;
  if (p.split > 1) {  // cluster launch, two cluster barriers, the exchange
    const int clusters = swap_clusters(p.split, p.ew);
    const int64_t rounds = (tiles + clusters - 1) / clusters;
    c += (double)rounds * ((p.k_blocks + p.split - 1) / p.split) * per_kb + 8000.0 + p.nt * p.nacc * (epi == EPI_ROTARY ? 60.0 : 30.0) / warps +
         (epi == EPI_ROTARY ? 3000.0 : 0.0) + finish / p.split;
  } else {
    const int64_t rounds = (tiles + p.grid - 1) / p.grid;
    const double main = p.k_blocks * per_kb;
    if (2 * p.nacc * p.nt <= p.tmem_cols && rounds > 1) c += rounds * (main > finish ? main : finish) + finish;
    else c += rounds * (main + finish);
  }
  // the weights at HBM's rate (3500 B/clk), as far as the rings hold enough of them for its latency (3000 clocks loaded)
  const double in_flight = (double)p.grid * p.stages * p.nacc * kSwapTileBytes / 3000.0;
  const double hbm = (double)N * K * 2 / (in_flight < 3500.0 ? in_flight : 3500.0) + 8000.0;
  return c > hbm ? c : hbm;
}

// Small batches are bound by the weights, and a round of tiles by its share of them or by the k-blocks of one tile: the last
// round costs as much with one tile as with many.  (8 tokens x 19072 x 4096: 40 us, estimated 41; x 128256 x 4096: 164, 161;
// SiLU, 8 x 38144 x 8192: 138, 137.)
double swap_walk_clocks(int epi, int64_t K, const SwapPlan& p) {
  const int64_t tiles = (int64_t)p.w_tiles * p.t_tiles, rounds = tiles / p.grid, left = tiles % p.grid;
  const double chunks = p.nt / 16, warps = p.ew / 4, main = p.k_blocks * swap_per_kb(epi, p);
  const double finish = epi == EPI_STORE ? 300.0 + chunks * 950.0 : 600.0 + chunks / warps * (epi == EPI_SILU_MUL ? 900.0 : 3000.0);
  const double tile = main > finish ? main : finish, bytes = 2.0 * 128 * p.nacc * (double)K / p.t_tiles;
  const double in_flight = (double)p.grid * p.stages * p.nacc * kSwapTileBytes / 3000.0, hbm = in_flight < 3500.0 ? in_flight : 3500.0;
  double c = 6000.0 + finish + (double)rounds * (p.grid * bytes / hbm > tile ? p.grid * bytes / hbm : tile);
  if (left) c += left * bytes / hbm > tile ? left * bytes / hbm : tile;
  return c;
}

static bool swap_fits(int epi, int64_t M, int64_t N, int head_size, int neox) {
  if (M < 1 || N < 1) return false;
  // rotary: the pairs of a NeoX head, whole heads of 64 / 128 / 256 columns
  if (epi == EPI_ROTARY) return neox && (head_size == 64 || head_size == 128 || head_size == 256) && N % head_size == 0;
  return epi == EPI_STORE || epi == EPI_SILU_MUL;
}

// tile_cfg 0: the cheapest plan; else nt + 6000 (two accumulators) or + 7000 (one) + 100000 * split.
static bool search_swap(int epi, int64_t M, int64_t N, int64_t K, int head_size, int tile_cfg, SwapPlan* best, double* cost) {
  *cost = 1e30;
  if (tile_cfg > 0) {
    const int nt = tile_cfg % 1000, mode = (tile_cfg / 1000) % 100, split = tile_cfg / 100000 > 1 ? tile_cfg / 100000 : 1;
    if (nt < 16 || nt > 256 || (mode == 7 && epi != EPI_STORE)) return false;
    *cost = 0.0;
    return swap_plan(M, N, K, head_size, mode == 7 ? 1 : 2, (int)((M + nt - 1) / nt), split, best);
  }
  const int64_t t_min = (M + 255) / 256, t_max = (M + 15) / 16 < t_min + 12 ? (M + 15) / 16 : t_min + 12;
  // one accumulator for EPI_STORE, always: with two no shape below 1300 tokens was faster, and 777 x 4096 x 4096 took 35 us
  // against 24; beyond that the general kernel has most shapes
  const int nacc = epi == EPI_STORE ? 1 : 2;
  for (int64_t t = t_min; t <= t_max; ++t)
    for (int s = 1; s <= 8; ++s) {
      SwapPlan p;
      if (!swap_plan(M, N, K, head_size, nacc, (int)t, s, &p)) continue;
      if (s > 1 && ((int64_t)p.w_tiles * t * s > sm_count() || p.k_blocks / s < 4)) break;
      if (s > 1 && (int64_t)p.w_tiles * t > swap_clusters(s, p.ew)) continue;  // one round of clusters
      const double c = swap_cost(epi, N, K, p);
      if (c < *cost) { *cost = c; *best = p; }
    }
  return *cost < 1e30;
}

bool plan_swap(int epi, int64_t M, int64_t N, int64_t K, int head_size, int neox, int tile_cfg, SwapPlan* plan, double* clocks) {
  return swap_fits(epi, M, N, head_size, neox) && search_swap(epi, M, N, K, head_size, tile_cfg, plan, clocks);
}

template <typename T, int EPI, int NACC, int EW>
static int launch_swap(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& txt, const GemmArgs& g, const SwapPlan& p,
                       cudaStream_t s) {
  auto kern = gemm_swap_kernel<T, EPI, NACC, EW>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  SB_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    SB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (EW == 4 ? kSwapHalfRing : kSwapRing) + 2048));
    configured_dev = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.grid);
  cfg.blockDim = dim3(64 + 32 * EW);
  // + 1 KiB for the alignment of the ring, + 1 KiB: an x box may be one swizzle atom shorter than the MMA's N
  cfg.dynamicSmemBytes = (size_t)p.stages * (NACC * kSwapTileBytes + p.act_rows * kBK * 2) + 2048;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SB_CUDA(cudaLaunchKernelEx(&cfg, kern, tw, tx, txt, g, p));
  return SB200_OK;
}

template <typename T>
static int dispatch_swap(int epi, const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& txt, const GemmArgs& g,
                         const SwapPlan& p, cudaStream_t s) {
#define SB_SWAP(E, A) (p.ew == 4 ? launch_swap<T, E, A, 4>(tw, tx, txt, g, p, s) : launch_swap<T, E, A, 8>(tw, tx, txt, g, p, s))
  if (epi == EPI_ROTARY) return SB_SWAP(EPI_ROTARY, 2);
  if (epi == EPI_SILU_MUL) return SB_SWAP(EPI_SILU_MUL, 2);
  return p.nacc == 1 ? SB_SWAP(EPI_STORE, 1) : SB_SWAP(EPI_STORE, 2);
#undef SB_SWAP
}

int run_gemm_swap(int dtype, int epi, const SwapPlan& p, const void* x, int64_t ldx, const void* w, int64_t ldw,
                  const GemmArgs& g, cudaStream_t s) {
  if (dtype != SB200_BF16 && dtype != SB200_F16) {
    set_error("tcgen05 GEMM supports bf16/fp16 only");
    return SB200_ERR_UNSUPPORTED;
  }
  CUtensorMap tw, tx, txt;
  int rc = make_tmap_2d(&tx, dtype, x, g.M, g.K, ldx, p.act_rows, kBK);
  if (rc) return rc;
  txt = tx;
  const int64_t left = g.M - (int64_t)(p.t_tiles - 1) * p.nt;  // tokens of the last tile
  if ((left + 7) / 8 * 8 != p.act_rows) {
    rc = make_tmap_2d(&txt, dtype, x, g.M, g.K, ldx, (int)((left + 7) / 8 * 8), kBK);
    if (rc) return rc;
  }
  rc = make_tmap_2d(&tw, dtype, w, g.N, g.K, ldw, epi == EPI_ROTARY ? g.head_size / 2 : 128, kBK);
  if (rc) return rc;
  return dtype == SB200_BF16 ? dispatch_swap<__nv_bfloat16>(epi, tw, tx, txt, g, p, s) : dispatch_swap<__half>(epi, tw, tx, txt, g, p, s);
}

}  // namespace sb200
