// Host-side declarations shared by gemm.cu (launch logic) and comm.cu (the
// row-parallel entry point builds its GemmArgs/ReduceArgs and calls in here).
#pragma once

#include "gemm_sm100.cuh"

namespace sb200 {

int make_tmap_2d(CUtensorMap* map, int dtype, const void* ptr, int64_t rows, int64_t cols, int64_t ld_elems,
                 int box_rows, int box_cols);
// First bytes of a split-K workspace hold the per-(tile, slot) arrival counters (zero between launches).
constexpr size_t kWsCounterBytes = 64 * 1024;

struct GemmPlan {
  int cta2, mi, bn, units, tiles_full;
  int rem_splits;  // S of the tile configuration: about S units share a tile of the last partial round
  int rem_units;   // units the k-blocks of that round are spread over (= its tiles when nothing is cut)
  int stages, m_tiles, n_tiles, k_blocks;
  int cluster_split;  // > 1: one tile per cluster of that many CTA pairs, K split between the pairs (MODE 5)
  double est_clocks;
};
// tile_cfg: 0 = choose; else BN + 1000*MODE + 100000*S (MODE 1|2: one CTA, 3|4: CTA pairs; S >= 2: the tiles of the last partial round are cut along K so that about S units share one; MODE 5: CTA pairs, every tile computed by a cluster of S = 2 or 4 pairs that split its k-blocks and combine their accumulators through distributed shared memory -- for problems with at most #SMs / (2 S) tiles).  ws_bytes: split-K workspace available (0 = none).
GemmPlan plan_gemm(int epi, int64_t M, int64_t N, int64_t K, int head_size, int tile_cfg, size_t ws_bytes, int neox = 1);
uint32_t gemm_push_increments(const GemmPlan& p, int64_t M, int64_t lo, int64_t hi);
int run_gemm_sm100(int dtype, int epi, const GemmPlan& plan, const void* x, int64_t ldx, const void* w, int64_t ldw,
                   GemmArgs g, void* workspace, const CommView& cv, const ReduceArgs& ra, cudaStream_t s,
                   int64_t b_rows = 0);  // b_rows: rows of the B matrix when it is taller than g.N (stacked experts)
// Operand roles swapped, tokens as the MMA's N (gemm_swap.cu).
constexpr int kSwapHalfRing = 104 * 1024;             // ring of one CTA: two of them fit an SM
constexpr int kSwapRing = 216 * 1024;
constexpr int64_t kSwapPrefetchBytes = 24ll << 20;    // weights of a launch requested before its dependency wait
// Clocks a gemm_sm100.cuh launch of this plan takes, fitted like the estimate of gemm_swap.cu it is compared with.
double gemm_plan_clocks(int epi, int64_t N, int64_t K, const GemmPlan& p);
// Bytes a clock that the L2 delivers to the shared memory of one SM while `ctas` SMs load.
inline double gemm_feed_rate(int ctas) { return 8600.0 / ctas < 90.0 ? 8600.0 / ctas : 90.0; }
struct SwapPlan {
  int w_tiles, t_tiles;  // tiles of 128 * nacc weight rows, and of `nt` tokens
  int nt;         // tokens of a tile: the MMA's N
  int split;      // CTAs of the cluster that shares a tile's K (1: whole tiles, walked round-robin)
  int grid;       // CTAs
  int stages;
  int act_rows;   // rows of the x box of a full tile (the last tile may have a shorter one)
  int prefetch;   // k-blocks of weights requested into the L2 before the dependency wait
  int tmem_cols;
  int k_blocks;
  int half_shift; // EPI_ROTARY: log2(head_size / 2)
  int nacc, ew;   // accumulators and epilogue warps: which kernel
};
// tile_cfg 0: the cheapest plan and its estimated clocks; else the plan of that configuration (MODE 6|7).  False: none.
bool plan_swap(int epi, int64_t M, int64_t N, int64_t K, int head_size, int neox, int tile_cfg, SwapPlan* plan, double* clocks);
// Clocks of a projection of up to 64 tokens whose CTAs walk several rounds of whole tiles.
double swap_walk_clocks(int epi, int64_t K, const SwapPlan& plan);
int run_gemm_swap(int dtype, int epi, const SwapPlan& plan, const void* x, int64_t ldx, const void* w, int64_t ldw,
                  const GemmArgs& g, cudaStream_t s);
// At most 16 output columns and not too many tokens (gemm_narrow.cu).  `fits`: the shape; `*done` = false: the operands' rows cannot be read in 16-byte
// pieces, nothing was launched.
bool narrow_fits(int epi, int64_t M, int64_t N, int64_t K);
int run_gemm_narrow(int dtype, int epi, const void* x, int64_t ldx, const void* w, int64_t ldw, const GemmArgs& g,
                    cudaStream_t s, bool* done);
// Which tensor-core kernel runs a problem, with its schedule.
enum { GEMM_NONE = 0, GEMM_GENERAL = 1, GEMM_SWAPPED = 2 };
struct GemmChoice {
  int kernel;
  GemmPlan general;
  SwapPlan swapped;
};
GemmChoice choose_gemm(int epi, int64_t M, int64_t N, int64_t K, int head_size, int neox, int tile_cfg, size_t ws_bytes);
int run_gemm_f32(float* C, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb, const float* bias,
                 int M, int N, int K, cudaStream_t s);

}  // namespace sb200
