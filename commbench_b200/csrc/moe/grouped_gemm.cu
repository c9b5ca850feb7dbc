// Grouped (per-expert) tcgen05 GEMMs over the expert-major receive buffer.
//
//   up:    H1[rows, 2I] = A[rows, H] * W1[e][2I, H]^T          (TMA-store epilogue, local)
//          or, gated: S[rows, I] = silu(A * Wgate^T) * (A * Wup^T) in the same epilogue
//   down:  O[rows, H]   = S[rows, I] * W2[e][H, I]^T, each output row written straight
//          into the combine buffer of the rank that owns the token (fused combine send)
//
// Rows are grouped by local expert, every group padded to a multiple of 128, so
// one 128-row block belongs to exactly one expert: `mblk_expert[m_blk]` picks the
// weight slab, the number of row blocks is read from device memory (it depends
// on the routing), and the tile list is simply (row block, column block).
//
// A decode step (early): each product starts as a programmatic dependent and fetches weights - which no kernel of
// the layer writes - while the kernel before ends.  That saves 3 to 8 us of a layer, calls in a row, three layers'
// weights in turn: 16 tokens, top-8 of 8 experts, hidden 7168, intermediate 2048 (16 rows per expert) 174 -> 168;
// 52, top-4 of 8, 4096 / 1024 (26) 86 -> 81; 200, top-8 of 32, 2048 / 1024 (50) 143 -> 136; 380 of the same (95)
// 143 -> 136; 1500, top-4 of 32 (188) 182 -> 178.  Layers of 300 us and more do not show it: 100, top-8 of 32,
// 7168 / 2048 514 to 529 without, 517 to 539 with; 740, top-8 of 64, 2048 / 2048 (93) 341, 348 to 354; 3096,
// top-8 of 64, 2048 / 1024 (387) 455 to 510, 505 to 513.  Two waves of tiles or less run 128 columns
// wide (narrow_tiles in ops/moe.py).  Loading only the rows that a block has, in boxes of 32, cost the producer
// more than it saved (511 -> 521).  What bounds a large layer is the power cap: a CTA pair per two row blocks,
// which draws a third less out of L2, takes 2450 us instead of 2540 in a burst (4096 tokens, top-8 of 32) and as
// long as this, 2960, when calls follow each other.
//
// The reference's grouped GEMM for the same layer is a scalar-FMA kernel
// (datasets/example056_thunderkitten_moe_dispatch_gemm_easy/nv/
// empty_thunderkitten_moe_dispatch_gemm.cu:227-293); its combine sends expert
// outputs back in a separate kernel (datasets/example082_deepep_jit_combine/nv/
// empty_deepep_jit_combine.cu:15-67).
#include "../gemm/gemm_sm100.cuh"

#include <string>

#include "../gemm/launch.h"
#include "../gemm/tmap_host.h"
#include "../prim/barrier.cuh"
#include "../symm/driver_api.h"

namespace cb {

struct GroupedParams {
  CUtensorMap tm_a;   // [max_rows, K]
  CUtensorMap tm_b;   // [E_local * N, K]   (expert slabs stacked along rows)
  CUtensorMap tm_c;   // [max_rows, N]      (up projection only)
  GemmShape g;        // M = max_rows (upper bound), N, K
  const int* mblk_expert;  // [max_rows / 128]
  const int* n_mblocks;    // device word: row blocks in use
  // down projection: scatter to token owners
  const int2* recv_meta;               // [max_rows] {owner rank, pair index} or {-1,-1}
  uint8_t* combine_peer[CB_MAX_RANKS]; // owner's combine buffer [T*K, N] bf16
  uint32_t* done_peer[CB_MAX_RANKS];   // owner's done words [W]
  uint32_t* done_ctas;                 // local scratch counter
  int rank, world;
  int early;
  uint32_t* status;
};

// kGatedUp (up projection only): the weight slab of every expert is stored with its rows
// interleaved - 128 gate rows, then the 128 up rows of the same outputs, and so on - and
// the epilogue writes silu(gate) * up, [rows, N/2], so H1 never exists in memory.  A 256-wide tile
// is such a block; a 128-wide one takes the same half of its gate and of its up rows, in two boxes.
template <class Cfg, bool kDown, bool kGatedUp = false>
struct GroupedPolicy {
  using P = GroupedParams;
  static constexpr bool kGated = kGatedUp;
  static constexpr int kBHalfStep = kGatedUp && Cfg::BN == 128 ? 128 : 0;
  static_assert(!kGatedUp || Cfg::BN == 128 || Cfg::BN == 256, "half a block of gate and up rows, or a whole one");
  static_assert(!(kDown && kGatedUp), "the gated epilogue belongs to the up projection");
  // The kernel before is the receive kernel, the other product or the SwiGLU kernel of the unfused form: each
  // releases its dependents after its own wait or only by its end, so the plan has been complete since then,
  // and none of them writes weights (prim/pdl.cuh).
  __device__ static bool early_b(const P& p) { return p.early != 0; }
  __device__ static int num_tiles(const P& p) {
    int mb = *reinterpret_cast<const volatile int*>(p.n_mblocks);
    if (mb > p.g.num_m_blocks) mb = p.g.num_m_blocks;
    return mb * p.g.num_n_blocks;
  }
  // Column blocks of one row block run together: the A row block is read once
  // from HBM and the expert's weight slab stays in L2 across the expert's row blocks.
  __device__ static void tile_coord(const P& p, int tile, int* m, int* n) {
    *m = tile / p.g.num_n_blocks;
    *n = tile - *m * p.g.num_n_blocks;
  }
  __device__ static const CUtensorMap* map_a(const P& p, int) { return &p.tm_a; }
  __device__ static const CUtensorMap* map_b(const P& p) { return &p.tm_b; }
  __device__ static int a_row(const P&, int m_blk) { return m_blk * Cfg::BM; }
  __device__ static int b_row(const P& p, int m_blk, int n_blk) {
    const int first = p.mblk_expert[m_blk] * p.g.N;
    if constexpr (kBHalfStep != 0) return first + (n_blk >> 1) * 256 + (n_blk & 1) * 64;
    return first + n_blk * Cfg::BN;
  }
  __device__ static bool wait_a_ready(const P&, int, volatile int*) { return true; }
  static constexpr bool kDirect = kDown;
  static constexpr bool kSignalPerTile = false;  // one completion flag per kernel instead
  static constexpr bool kScatterRows = kDown;
  __device__ static void store_box(const P& p, int m_blk, int n_blk, int row, int col,
                                   const void* smem_box) {
    tma_store_2d(&p.tm_c, smem_box, n_blk * (kGatedUp ? Cfg::BN / 2 : Cfg::BN) + col,
                 m_blk * Cfg::BM + row);
  }
  __device__ static void direct_targets(const P&, int, int, DirectTargets* t) {
    t->n = 0;
    t->ld_bytes = 0;
    t->rows = Cfg::BM;
    t->cols = Cfg::BN;
  }
  // Destination of output row `row` of row block m_blk: the owner's combine slot, or null
  // for padding rows.
  __device__ static uint8_t* row_base(const P& p, int m_blk, int row) {
    const int2 m = p.recv_meta[static_cast<long long>(m_blk) * Cfg::BM + row];
    if (m.x < 0) return nullptr;
    return p.combine_peer[m.x] + static_cast<long long>(m.y) * p.g.N * 2;
  }
  __device__ static void tile_done(const P&, int, int, int) {}
};

template <class Cfg, bool kDown, bool kGatedUp>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
    grouped_gemm_kernel(const __grid_constant__ GroupedParams p) {
  extern __shared__ uint8_t smem_raw[];
  gemm_cta_main<Cfg, GroupedPolicy<Cfg, kDown, kGatedUp>>(p, p.g, p.status, blockIdx.x, gridDim.x,
                                                          smem_raw);
  if constexpr (kDown) {
    // Every CTA releases its rows; the last one tells every owner that this expert rank
    // is done (the owners' combine reduction waits for W such words).
    __syncthreads();
    if (threadIdx.x == 0) {
      fence_acq_rel_sys();
      if (atomicAdd(p.done_ctas, 1u) == gridDim.x - 1) {
        *p.done_ctas = 0u;
        fence_acq_rel_sys();
        for (int d = 0; d < p.world; ++d) {
          const int dest = (p.rank + d) % p.world;
          red_relaxed_sys_add(p.done_peer[dest] + p.rank, 1u);
        }
      }
    }
  }
}

template <class Cfg, bool kDown, bool kGatedUp = false>
static int launch_grouped(const GroupedParams& p, int ctas, bool early, cudaStream_t st) {
  static std::atomic<uint64_t> smem_done{0};
  cudaError_t e = allow_smem(
      reinterpret_cast<const void*>(grouped_gemm_kernel<Cfg, kDown, kGatedUp>), Cfg::SMEM_BYTES,
      smem_done);
  if (e != cudaSuccess) {
    set_last_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    return -1;
  }
  e = launch_gemm_kernel_pdl(grouped_gemm_kernel<Cfg, kDown, kGatedUp>, ctas, Cfg::THREADS,
                             Cfg::SMEM_BYTES, st, 1, false, early, p);
  if (e != cudaSuccess) {
    set_last_error(std::string("grouped gemm launch: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // namespace cb

using namespace cb;

extern "C" {

struct CbGroupedDesc {
  int max_rows, N, K, n_local_experts;
  int down;          // 0: up projection (C local), 1: down projection with combine scatter
  int rank, world;
  int ctas;
  int gated;         // up only: b is gate/up interleaved per 256 rows, c = silu(gate) * up
  int narrow;        // 0: tiles of a row block x 256 columns; 1: of 128 columns
  int early;         // 1: starts while the kernel before ends and fetches weights first
  const void* a;     // [max_rows, K] bf16
  const void* b;     // [n_local_experts * N, K] bf16
  void* c;           // up only: [max_rows, N] bf16, or [max_rows, N / 2] when gated
  const void* mblk_expert;
  const void* n_mblocks;
  const void* recv_meta;
  void* combine_peer[CB_MAX_RANKS];
  void* done_peer[CB_MAX_RANKS];
  void* done_ctas;
  void* status;
};

}  // extern "C"

namespace cb {
template <class Cfg>
static int run_grouped(const CbGroupedDesc* d, int ctas, cudaStream_t st) {
  const int n_multiple = d->gated ? 256 : Cfg::BN;
  if (d->max_rows % 128 != 0 || d->K % 8 != 0 || d->N % n_multiple != 0) {
    set_last_error("grouped gemm: max_rows % 128 == 0, K % 8 == 0, N % " + std::to_string(n_multiple) +
                   " == 0 required");
    return -1;
  }
  GroupedParams p;
  if (make_tmap_2d(&p.tm_a, d->a, TMAP_BF16, d->K, d->max_rows, (unsigned long long)d->K * 2,
                   Cfg::BK, Cfg::BM, true))
    return -1;
  if (make_tmap_2d(&p.tm_b, d->b, TMAP_BF16, d->K, (unsigned long long)d->n_local_experts * d->N,
                   (unsigned long long)d->K * 2, Cfg::BK,
                   d->gated && Cfg::BN == 128 ? Cfg::BN / 2 : Cfg::BN, true))
    return -1;
  if (d->gated && d->down) {
    set_last_error("grouped gemm: the gated epilogue belongs to the up projection");
    return -1;
  }
  if (!d->down) {
    const unsigned long long c_cols = d->gated ? d->N / 2 : d->N;
    if (make_tmap_2d(&p.tm_c, d->c, TMAP_BF16, c_cols, d->max_rows, c_cols * 2, Cfg::EPI_COLS, 32,
                     true))
      return -1;
  } else {
    p.tm_c = p.tm_a;
  }
  p.g.M = d->max_rows;
  p.g.N = d->N;
  p.g.K = d->K;
  p.g.num_m_blocks = d->max_rows / 128;
  p.g.num_n_blocks = d->N / Cfg::BN;
  p.g.num_k_blocks = (d->K + Cfg::BK - 1) / Cfg::BK;
  p.g.alpha = 1.0f;
  p.mblk_expert = static_cast<const int*>(d->mblk_expert);
  p.n_mblocks = static_cast<const int*>(d->n_mblocks);
  p.recv_meta = static_cast<const int2*>(d->recv_meta);
  for (int r = 0; r < CB_MAX_RANKS; ++r) {
    p.combine_peer[r] = static_cast<uint8_t*>(d->combine_peer[r]);
    p.done_peer[r] = static_cast<uint32_t*>(d->done_peer[r]);
  }
  p.done_ctas = static_cast<uint32_t*>(d->done_ctas);
  p.rank = d->rank;
  p.world = d->world;
  p.status = static_cast<uint32_t*>(d->status);
  const bool early = d->early != 0;
  p.early = d->early;
  if (d->down) return launch_grouped<Cfg, true>(p, ctas, early, st);
  return d->gated ? launch_grouped<Cfg, false, true>(p, ctas, early, st)
                  : launch_grouped<Cfg, false, false>(p, ctas, early, st);
}
}  // namespace cb

extern "C" {

int cb_moe_grouped_gemm(const CbGroupedDesc* d, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int ctas = d->ctas > 0 ? d->ctas : 148;
  return d->narrow ? run_grouped<GemmCfg<128, 6, false>>(d, ctas, st)
                   : run_grouped<GemmCfg<256, 4, false>>(d, ctas, st);
}

}  // extern "C"
