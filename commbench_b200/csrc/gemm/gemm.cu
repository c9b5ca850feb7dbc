// Plain (single-GPU) tcgen05 GEMM entry points and the tensor-map helper.
// C[M,N] = alpha * A[M,K] * B[N,K]^T, bf16 or fp8-e4m3 inputs, bf16 output.
//
// This is the local GEMM every fused path is built from, and the kernel that
// runs when the world size is 1.  The reference has the equivalent as
// `matmul::kernel` (datasets/example053_thunderkitten_gemm_ar_easy/nv/
// empty_thunderkitten_gemm_ar.cu:84-191).
#include "gemm_sm100.cuh"
#include "gemm_small.cuh"

#include <math.h>

#include <string>

#include "../symm/driver_api.h"
#include "launch.h"
#include "tmap_host.h"

namespace cb {

int make_tmap_2d(CUtensorMap* out, const void* base, TmapDtype dt, unsigned long long inner,
                 unsigned long long outer, unsigned long long row_stride_bytes,
                 unsigned box_inner, unsigned box_outer, bool swizzle128) {
  const DriverApi& d = driver_api();
  if (!d.ok) {
    set_last_error("tensor map: " + d.why);
    return -1;
  }
  const unsigned esz = dt == TMAP_BF16 ? 2 : (dt == TMAP_U8 ? 1 : 4);
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) {
    set_last_error("tensor map: base address is not 16-byte aligned");
    return -1;
  }
  if (row_stride_bytes % 16ull != 0) {
    set_last_error("tensor map: row stride is not a multiple of 16 bytes");
    return -1;
  }
  if ((box_inner * esz) % 16u != 0 || box_inner > 256u || box_outer > 256u) {
    set_last_error("tensor map: bad box");
    return -1;
  }
  if (swizzle128 && box_inner * esz != 128u) {
    set_last_error("tensor map: 128-byte swizzle needs a 128-byte inner box");
    return -1;
  }
  const CUtensorMapDataType cdt = dt == TMAP_BF16  ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                  : dt == TMAP_U8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                                  : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {row_stride_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = d.cuTensorMapEncodeTiled(
      out, cdt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error(cu_err("cuTensorMapEncodeTiled", r));
    return -1;
  }
  return 0;
}

struct PlainParams {
  CUtensorMap tm_a, tm_b, tm_c;
  CUtensorMap tm_c_half;   // 32-column boxes, for tile widths that are no multiple of 64
  GemmShape g;
  uint32_t* status;
  int raster_group;
};

template <class Cfg>
struct PlainPolicy {
  using P = PlainParams;
  static constexpr bool kPdl = true;
  static constexpr bool kDirect = false;
  static constexpr bool kSignalPerTile = false;
  static constexpr bool kScatterRows = false;
  __device__ static int b_row(const P&, int, int n_blk) { return n_blk * Cfg::BN; }
  __device__ static int num_tiles(const P& p) { return p.g.num_m_blocks * p.g.num_n_blocks; }
  __device__ static void tile_coord(const P& p, int tile, int* m, int* n) {
    raster_tile(tile, p.g.num_m_blocks, p.g.num_n_blocks, p.raster_group, m, n);
  }
  __device__ static const CUtensorMap* map_a(const P& p, int) { return &p.tm_a; }
  __device__ static const CUtensorMap* map_b(const P& p) { return &p.tm_b; }
  __device__ static int a_row(const P&, int m_blk) { return m_blk * Cfg::BM; }
  __device__ static bool wait_a_ready(const P&, int, volatile int*) { return true; }
  __device__ static void store_box(const P& p, int m_blk, int n_blk, int row, int col,
                                   const void* smem_box) {
    tma_store_2d(&p.tm_c, smem_box, n_blk * Cfg::BN + col, m_blk * Cfg::BM + row);
  }
  __device__ static void store_half_box(const P& p, int m_blk, int n_blk, int row, int col,
                                        const void* smem_box) {
    tma_store_2d(&p.tm_c_half, smem_box, n_blk * Cfg::BN + col, m_blk * Cfg::BM + row);
  }
  __device__ static void tile_done(const P&, int, int, int) {}
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
    gemm_plain_kernel(const __grid_constant__ PlainParams p) {
  extern __shared__ uint8_t smem_raw[];
  gemm_cta_main<Cfg, PlainPolicy<Cfg>>(p, p.g, p.status, blockIdx.x, gridDim.x, smem_raw);
}

static int g_sm_count = 0;
static int sm_count() {
  if (g_sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm_count <= 0) g_sm_count = 148;
  }
  return g_sm_count;
}

template <class Cfg>
static int launch_plain(const void* a, const void* b, void* c, int M, int N, int K, float alpha,
                        uint32_t* status, int max_ctas, cudaStream_t st,
                        unsigned long long* trace = nullptr, const float* a_scale = nullptr,
                        const float* b_scale = nullptr, const uint32_t* sfa = nullptr,
                        const uint32_t* sfb = nullptr) {
  PlainParams p;
  const TmapDtype dt = Cfg::FP8 ? TMAP_U8 : TMAP_BF16;
  const unsigned esz = Cfg::FP8 ? 1 : 2;
  if (make_tmap_2d(&p.tm_a, a, dt, K, M, (unsigned long long)K * esz, Cfg::BK, Cfg::CTA_M, true))
    return -1;
  if (make_tmap_2d(&p.tm_b, b, dt, K, N, (unsigned long long)K * esz, Cfg::BK, Cfg::B_ROWS, true))
    return -1;
  if (make_tmap_2d(&p.tm_c, c, TMAP_BF16, N, M, (unsigned long long)N * 2, Cfg::EPI_COLS, 32,
                   true))
    return -1;
  if constexpr (Cfg::BN % Cfg::EPI_COLS != 0) {
    if (make_tmap_2d(&p.tm_c_half, c, TMAP_BF16, N, M, (unsigned long long)N * 2, 32, 32, false))
      return -1;
  }
  p.g.M = M;
  p.g.N = N;
  p.g.K = K;
  p.g.num_m_blocks = (M + Cfg::BM - 1) / Cfg::BM;
  p.g.num_n_blocks = (N + Cfg::BN - 1) / Cfg::BN;
  p.g.num_k_blocks = (K + Cfg::BK - 1) / Cfg::BK;
  p.g.alpha = alpha;
  p.g.trace = trace;
  p.g.a_scale = a_scale;
  p.g.b_scale = b_scale;
  p.g.sfa = sfa;
  p.g.sfb = sfb;
  p.g.sfa_rows = M;
  p.g.sfb_rows = N;
  p.status = status;
  // Row blocks per raster panel: the panel's A rows (panel x K) stay in L2 while the B tiles stream past
  // them, so the panel is kept near 32 MB - but no lower than 2048 rows.  With a longer K the tiles that run
  // together share what they read at the same K instead, and that is least when they cover a square (2048 rows
  // x about as many columns): 8192 x 8192 x 28672 bf16 took 3430 us with two row blocks of 256 to a panel,
  // 3345 with four, 3100 with six, 3010 to 3030 with eight, 3040 with sixteen.
  {
    const long long panel_rows = (32ll << 20) / (static_cast<long long>(K) * esz);
    int grp = static_cast<int>(panel_rows / Cfg::BM);
    if (grp < 2048 / Cfg::BM) grp = 2048 / Cfg::BM;
    if (grp > 16) grp = 16;
    p.raster_group = grp;
  }
  {
    static std::atomic<uint64_t> smem_done{0};
    cudaError_t e = allow_smem(reinterpret_cast<const void*>(gemm_plain_kernel<Cfg>),
                               Cfg::SMEM_BYTES, smem_done);
    if (e != cudaSuccess) {
      set_last_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
      return -1;
    }
  }
  int tiles = p.g.num_m_blocks * p.g.num_n_blocks;
  int ctas = sm_count();
  if (max_ctas > 0 && max_ctas < ctas) ctas = max_ctas;
  if (tiles * Cfg::PAIR < ctas) ctas = tiles * Cfg::PAIR;
  ctas -= ctas % Cfg::PAIR;
  if (ctas < Cfg::PAIR) {
    set_last_error("gemm: a tile of a CTA pair needs a limit of at least two CTAs");
    return -1;
  }
  cudaError_t e = launch_gemm_kernel_pdl(gemm_plain_kernel<Cfg>, ctas, Cfg::THREADS, Cfg::SMEM_BYTES,
                                         st, Cfg::PAIR, false, true, p);
  if (e != cudaSuccess) {
    set_last_error(std::string("gemm launch: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

// A narrower tile of a CTA pair is worth it where it fills the last wave: 8192 x 3584 x 8192 is 448 tiles of
// 256 x 256 on 74 pairs, 7 waves for 6.05, and 512 of 256 x 224, 6.92.  All pairs together are bound by what
// they draw out of L2, so a tile's time falls by less than its width; the cost below puts the line between 256
// and 224 (192 and 224 with hardware block scales) where it was measured, 256 / 224 wide in us: the shape
// above bf16 339 / 328, fp8 169 / 164 (192 / 224 with block scales: 185 / 173); 3000 x 8192 x 3584 124 / 119,
// 67 / 65; 4096 x 7168 x 2048 with block scales 57 / 53; the other way 8192 x 8192 x 4096 353 / 361, 185 / 190,
// 2048 x 4096 x 4096 with block scales 36 / 40.
// Calls in a row, under the power cap: the shape above fp8 199.6 -> 191.5 us, with block scales 213.8 -> 202.
static float pair_tile_cost(int bn) { return static_cast<float>(bn + 512); }
static long long pair_waves(long long m256, int N, int bn, int sms) {
  return (m256 * ((N + bn - 1) / bn) + sms / 2 - 1) / (sms / 2);
}
// Tile width with hardware block scales.  Below eight K blocks a tile takes as long as its store boxes of 64
// columns, and the half box counts as one: 4347 x 8104 x 768, 10 / 9 waves, 192 / 224 wide 35.2 / 41.6 us, 6993 x
// 7504 x 768 (16 / 13) 50.6 / 54.5, 1718 x 4296 x 768 (3 / 2) 13.1 / 12.4.  Over 60 shapes of 1 to 6 K blocks whose
// cost above is lower with 224, taking that cost for all K is 3.5 % off the better width, this rule 0.2 %.
static int mx_pair_tile(int M, int N, int K, int sms) {
  const long long m256 = (M + 255) / 256;
  const float w224 = static_cast<float>(pair_waves(m256, N, 224, sms));
  const float w192 = static_cast<float>(pair_waves(m256, N, 192, sms));
  const bool wide = w224 * pair_tile_cost(224) < w192 * pair_tile_cost(192) && (K >= 1024 || w224 * 4.f < w192 * 3.f);
  return wide ? 224 : 192;
}

// Which kernel and tile a GEMM runs on, by a model of its time in microseconds.  kbytes: bytes of one
// K row (K x element size).  Per-128-byte-K-block times of a CTA that nothing else holds up, measured on
// one m-block: persistent pairs on 256 x 256 tiles 0.315, single CTAs 0.33, the small kernel's 64 / 128 /
// 256-wide tiles 0.16 / 0.21 / 0.34 (0.19 / 0.30 / 0.485 where rows do not start on 128-byte lines, since
// every box row then touches two); all CTAs together draw at most 17 TB/s out of L2 (12.5), weights
// arrive at 6 TB/s from memory, and a persistent tile takes 2.5 us however short its K loop
// (its epilogue).  Over 150 random shapes (M 1-8192, N 512-16384, K 512-8192, bf16 and fp8), called in
// a row with three sets of operands in turn, the choice takes 1.0 % more than the best of all variants on
// (geometric) average and over 5 % more for 9 of them (1.8 % and 18 with the constants of before: pairs 0.30,
// single CTAs 0.36, 11 TB/s); the worst is 6 x 1792 x 5456, 8.0 us in four parts and 6.1 in eight.
struct GemmChoice {
  int bn;      // persistent: 64 ... 512 as in cb_gemm_bf16; small kernel: its tile width
  int split;   // 0: persistent kernel; else the small kernel's K splits
};
// Two limits that a loop meets together: a little above the larger one.
static float both_us(float a, float b) {
  const float a3 = a * a * a, b3 = b * b * b;
  return cbrtf(sqrtf(a3 * a3 + b3 * b3));
}
static GemmChoice choose_gemm(int M, int N, long long kbytes, int sms) {
  const float nkb = static_cast<float>((kbytes + 127) / 128);
  const float l2_rate = kbytes % 128 == 0 ? 17e6f : 12.5e6f;   // bytes per us
  const float hbm_us = static_cast<float>(N) * static_cast<float>(kbytes) / 6e6f;
  const long long m128 = (M + 127) / 128, m256 = (M + 255) / 256;
  GemmChoice best = {512, 0};
  float best_us = 1e30f;
  const auto offer = [&](int bn, int split, float us) {
    if (us < best_us) {
      best_us = us;
      best = {bn, split};
    }
  };
  {  // persistent kernels: pairs on 256 x 256 and 256 x 224, single CTAs on 128 x 256
    // (224 from 18 K blocks on: in shorter loops the epilogue counts, which gains nothing)
    for (int bn = 256; bn >= (nkb >= 18.f ? 224 : 256); bn -= 32) {
      const long long pairs = m256 * ((N + bn - 1) / bn);
      const float pair_ctas = 2.f * static_cast<float>(pairs < sms / 2 ? pairs : sms / 2);
      const float cta_bytes = static_cast<float>(128 + bn / 2) * 128.f;   // per CTA and K block
      const float pair_kb =
          fmaxf(0.315f * pair_tile_cost(bn) / pair_tile_cost(256), pair_ctas * cta_bytes / l2_rate);
      const float waves = static_cast<float>(pair_waves(m256, N, bn, sms));
      offer(2 * bn, 0, 7.7f + fmaxf(waves * fmaxf(nkb * pair_kb, 2.5f), hbm_us));
    }
    const long long singles = m128 * ((N + 255) / 256), sw = (singles + sms - 1) / sms;
    const float single_ctas = static_cast<float>(singles < sms ? singles : sms);
    const float single_kb = fmaxf(0.33f, single_ctas * 49152.f / l2_rate);
    offer(256, 0, 6.5f + fmaxf(static_cast<float>(sw) * fmaxf(nkb * single_kb, 2.5f), hbm_us));
  }
  const int a_rows = M < 128 ? (M + 7) / 8 * 8 : 128;
  const int widths[3] = {64, 128, 256};
  const bool lines = kbytes % 128 == 0;
  const float kb_us[3] = {lines ? 0.16f : 0.19f, lines ? 0.21f : 0.30f, lines ? 0.34f : 0.485f};
  for (int i = 0; i < 3; ++i)
    for (int split = 1; split <= 8; split *= 2) {
      if (static_cast<float>(split) > nkb) break;
      const long long ctas = m128 * ((N + widths[i] - 1) / widths[i]) * split;
      // one wave only; clusters do not pack a GPC's SMs completely
      if (ctas > (split <= 2 ? sms : split == 4 ? sms * 9 / 10 : sms * 4 / 5)) break;
      const float per_kb = fmaxf(kb_us[i], static_cast<float>(ctas) *
                                               static_cast<float>(a_rows + widths[i]) * 128.f / l2_rate);
      const float tile_kb = static_cast<float>(a_rows * widths[i]) * 4.f / 1024.f;
      const float reduce = split == 1 ? 0.5f + tile_kb * 0.025f
                                      : (split == 8 ? 3.7f : 1.7f) + tile_kb * 0.05f *
                                            static_cast<float>(split - 1) / static_cast<float>(split);
      const float steps = static_cast<float>((static_cast<int>(nkb) + split - 1) / split);
      offer(widths[i], split, 2.7f + both_us(steps * per_kb, hbm_us) + reduce);
    }
  return best;
}

// Tile of the persistent kernels for a caller that limits the CTAs to `max_ctas`: pairs on 256 x 256
// tiles when there are plenty of them (and the limit admits a pair), narrower tiles for skinny
// problems.
static int persistent_tile(int M, int N, int max_ctas) {
  const long long m_blocks = (M + 127) / 128;
  if (max_ctas >= 2 && static_cast<long long>((M + 255) / 256) * ((N + 255) / 256) * 2 >= sm_count()) return 512;
  if (m_blocks * ((N + 255) / 256) >= sm_count()) return 256;
  if (m_blocks * ((N + 127) / 128) >= sm_count()) return 128;
  return 64;
}

template <int BN, bool FP8, int SPLIT>
static int launch_small(const SmallParams& p, int tiles, cudaStream_t st) {
  using Cfg = SmallCfg<BN, FP8>;
  static std::atomic<uint64_t> smem_done{0};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(gemm_small_kernel<Cfg, SPLIT>),
                             Cfg::SMEM_BYTES, smem_done);
  if (e == cudaSuccess)
    e = launch_gemm_kernel_pdl(gemm_small_kernel<Cfg, SPLIT>, tiles * SPLIT, Cfg::THREADS,
                               Cfg::SMEM_BYTES, st, SPLIT, false, true, p);
  if (e != cudaSuccess) {
    set_last_error(std::string("gemm launch: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

template <int BN, bool FP8>
static int run_small(const void* a, const void* b, void* c, int M, int N, int K, float alpha,
                     int split, uint32_t* status, cudaStream_t st) {
  using Cfg = SmallCfg<BN, FP8>;
  SmallParams p;
  const TmapDtype dt = FP8 ? TMAP_U8 : TMAP_BF16;
  const unsigned long long pitch = static_cast<unsigned long long>(K) * (FP8 ? 1 : 2);
  p.a_rows = M < Cfg::BM ? (M + 7) / 8 * 8 : Cfg::BM;
  p.stages = Cfg::stages(p.a_rows);
  if (make_tmap_2d(&p.tm_a, a, dt, K, M, pitch, Cfg::BK, static_cast<unsigned>(p.a_rows), true))
    return -1;
  if (make_tmap_2d(&p.tm_b, b, dt, K, N, pitch, Cfg::BK, Cfg::BN, true)) return -1;
  if ((reinterpret_cast<uintptr_t>(c) & 15u) != 0) {
    set_last_error("gemm: C is not 16-byte aligned");
    return -1;
  }
  p.c = static_cast<__nv_bfloat16*>(c);
  p.M = M;
  p.N = N;
  p.num_m = (M + Cfg::BM - 1) / Cfg::BM;
  p.num_kb = (K + Cfg::BK - 1) / Cfg::BK;
  p.alpha = alpha;
  p.status = status;
  const int tiles = p.num_m * ((N + BN - 1) / BN);
  if (split > p.num_kb) {
    set_last_error("gemm: more K splits than K blocks");
    return -1;
  }
  switch (split) {
    case 1: return launch_small<BN, FP8, 1>(p, tiles, st);
    case 2: return launch_small<BN, FP8, 2>(p, tiles, st);
    case 4: return launch_small<BN, FP8, 4>(p, tiles, st);
    case 8: return launch_small<BN, FP8, 8>(p, tiles, st);
    default: set_last_error("gemm: K split must be 1, 2, 4 or 8"); return -1;
  }
}

template <bool FP8>
static int run_small_bn(const void* a, const void* b, void* c, int M, int N, int K, float alpha,
                        int bn, int split, uint32_t* status, cudaStream_t st) {
  switch (bn) {
    case 64: return run_small<64, FP8>(a, b, c, M, N, K, alpha, split, status, st);
    case 128: return run_small<128, FP8>(a, b, c, M, N, K, alpha, split, status, st);
    case 256: return run_small<256, FP8>(a, b, c, M, N, K, alpha, split, status, st);
    default: set_last_error("gemm: small tiles are 64, 128 or 256 wide"); return -1;
  }
}

}  // namespace cb

using namespace cb;

extern "C" {

// bf16: A [M,K], B [N,K], C [M,N], all row-major and 16-byte aligned; K % 8 == 0, N % 8 == 0.
// `bn` picks the tile: 256, 128 or 64 = one CTA per 128 x bn tile; 512 = a CTA pair per
// 256 x 256 tile, 448 = a pair per 256 x 224 tile, 384 = a pair per 256 x 128 tile; 0 = choose
// from the shape.
// `status` may be null.  Returns 0 or -1 (cb_last_error()).
int cb_gemm_bf16(const void* a, const void* b, void* c, int M, int N, int K, float alpha, int bn,
                 int max_ctas, void* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 8) != 0 || (N % 8) != 0) {
    set_last_error("cb_gemm_bf16: need M,N,K > 0, K % 8 == 0, N % 8 == 0");
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* s = static_cast<uint32_t*>(status);
  if (bn == 0) {
    const GemmChoice g = choose_gemm(M, N, 2ll * K, sm_count());
    if (g.split > 0 && max_ctas <= 0)
      return run_small_bn<false>(a, b, c, M, N, K, alpha, g.bn, g.split, s, st);
    bn = g.split > 0 || max_ctas == 1 ? persistent_tile(M, N, max_ctas) : g.bn;
  }
  switch (bn) {
    case 512:
      return launch_plain<GemmCfg<256, 6, false, 2>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 448:
      return launch_plain<GemmCfg<224, 6, false, 2>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 384:
      return launch_plain<GemmCfg<128, 8, false, 2>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 256:
      return launch_plain<GemmCfg<256, 4, false>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 128:
      return launch_plain<GemmCfg<128, 6, false>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 64:
      return launch_plain<GemmCfg<64, 8, false>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    default:
      set_last_error("cb_gemm_bf16: bn must be 0, 64, 128, 256, 384, 448 or 512");
      return -1;
  }
}

// What bn = 0 picks: tile width + 1000 x K splits (0 splits: a persistent kernel).
int cb_gemm_choice(int M, int N, int K, int fp8) {
  const GemmChoice g = choose_gemm(M, N, static_cast<long long>(K) * (fp8 ? 1 : 2), sm_count());
  return g.bn + 1000 * g.split;
}

// Tile width of a CTA pair that cb_gemm_fp8_mx picks (no limit on the CTAs).
int cb_gemm_mx_choice(int M, int N, int K) { return mx_pair_tile(M, N, K, sm_count()); }

// The split-K kernel with a given tile width (64, 128, 256) and number of K splits (1, 2, 4, 8).
int cb_gemm_small(const void* a, const void* b, void* c, int M, int N, int K, float alpha, int fp8,
                  int bn, int split, void* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % (fp8 ? 16 : 8)) != 0 || (N % 8) != 0) {
    set_last_error("cb_gemm_small: need M,N,K > 0, K % 8 == 0 (fp8: 16), N % 8 == 0");
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* s = static_cast<uint32_t*>(status);
  return fp8 ? run_small_bn<true>(a, b, c, M, N, K, alpha, bn, split, s, st)
             : run_small_bn<false>(a, b, c, M, N, K, alpha, bn, split, s, st);
}

// cb_gemm_bf16 with the role trace switched on: `trace` = 8 x (number of SMs) 64-bit words
// of device memory (see GemmShape::trace for what each CTA writes).  bn: 512 or 256.
int cb_gemm_bf16_traced(const void* a, const void* b, void* c, int M, int N, int K, float alpha,
                        int bn, void* trace, void* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 8) != 0 || (N % 8) != 0 || trace == nullptr) {
    set_last_error("cb_gemm_bf16_traced: need M,N,K > 0, K % 8 == 0, N % 8 == 0, a trace buffer");
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* s = static_cast<uint32_t*>(status);
  unsigned long long* t = static_cast<unsigned long long*>(trace);
  if (bn == 512)
    return launch_plain<GemmCfg<256, 6, false, 2>>(a, b, c, M, N, K, alpha, s, 0, st, t);
  if (bn == 256) return launch_plain<GemmCfg<256, 4, false>>(a, b, c, M, N, K, alpha, s, 0, st, t);
  set_last_error("cb_gemm_bf16_traced: bn must be 256 or 512");
  return -1;
}

// fp8 e4m3 inputs with ONE scale per tensor folded into alpha; K % 16 == 0.
int cb_gemm_fp8(const void* a, const void* b, void* c, int M, int N, int K, float alpha, int bn,
                int max_ctas, void* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 16) != 0 || (N % 8) != 0) {
    set_last_error("cb_gemm_fp8: need M,N,K > 0, K % 16 == 0, N % 8 == 0");
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* s = static_cast<uint32_t*>(status);
  if (bn == 0) {
    const GemmChoice g = choose_gemm(M, N, K, sm_count());
    if (g.split > 0 && max_ctas <= 0)
      return run_small_bn<true>(a, b, c, M, N, K, alpha, g.bn, g.split, s, st);
    bn = g.split > 0 || max_ctas == 1 ? persistent_tile(M, N, max_ctas) : g.bn;
  }
  switch (bn) {
    case 512:
      return launch_plain<GemmCfg<256, 6, true, 2>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 448:
      return launch_plain<GemmCfg<224, 6, true, 2>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 256:
      return launch_plain<GemmCfg<256, 4, true>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 128:
      return launch_plain<GemmCfg<128, 6, true>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    case 64:
      return launch_plain<GemmCfg<64, 8, true>>(a, b, c, M, N, K, alpha, s, max_ctas, st);
    default:
      set_last_error("cb_gemm_fp8: bn must be 0, 64, 128, 256, 448 or 512");
      return -1;
  }
}

// Block-scaled fp8: a [M,K] e4m3 with a_scale [M, K/128] fp32 (one scale per row and 128
// columns), b [N,K] e4m3 with b_scale [ceil(N/128), K/128] (one per 128 x 128 block); K % 128 == 0.
// C = alpha * (a * a_scale) (b * b_scale)^T in bf16.  The quantised operands feed the tensor
// cores directly; every 128-wide K block's partial sum is scaled and accumulated in fp32
// registers.  One CTA per 128 x 256 tile; `pair` is accepted and makes no difference (a pair per
// 256 x 256 tile was slower at every size, see gemm_sm100.cuh).
int cb_gemm_fp8_blockscaled(const void* a, const void* a_scale, const void* b, const void* b_scale,
                            void* c, int M, int N, int K, float alpha, int pair, int max_ctas,
                            void* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K % 128) != 0 || (N % 8) != 0 || a_scale == nullptr ||
      b_scale == nullptr) {
    set_last_error("cb_gemm_fp8_blockscaled: need M,N,K > 0, K % 128 == 0, N % 8 == 0, scales");
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t* s = static_cast<uint32_t*>(status);
  const float* as = static_cast<const float*>(a_scale);
  const float* bs = static_cast<const float*>(b_scale);
  (void)pair;
  return launch_plain<GemmCfg<256, 3, true, 1, true>>(a, b, c, M, N, K, alpha, s, max_ctas, st,
                                                      nullptr, as, bs);
}

// Block-scaled fp8 with POWER-OF-TWO scales applied by the tensor core: a [M,K], b [N,K] e4m3;
// sfa [ceil(K/512), M] and sfb [ceil(K/512), N] 32-bit words, each packing the exponent bytes
// (value 2^(byte - 127)) of four consecutive 128-wide K blocks of one operand row, lowest byte
// first (cb_quant_blockscaled_pow2 writes them; for a 128 x 128-block weight every row of a
// block carries the block's byte).  K % 128 == 0.
int cb_gemm_fp8_mx_traced(const void* a, const void* sfa, const void* b, const void* sfb, void* c,
                          int M, int N, int K, float alpha, int max_ctas, void* trace,
                          void* status, void* stream);

int cb_gemm_fp8_mx(const void* a, const void* sfa, const void* b, const void* sfb, void* c, int M,
                   int N, int K, float alpha, int max_ctas, void* status, void* stream) {
  return cb_gemm_fp8_mx_traced(a, sfa, b, sfb, c, M, N, K, alpha, max_ctas, nullptr, status,
                               stream);
}

// The same with the MMA role's trace on (`trace`: 8 x number-of-SMs 64-bit words, may be null).
int cb_gemm_fp8_mx_traced(const void* a, const void* sfa, const void* b, const void* sfb, void* c,
                          int M, int N, int K, float alpha, int max_ctas, void* trace,
                          void* status, void* stream) {
  // max_ctas < 0 selects the one-CTA-per-tile form (128 x 192 tiles) instead of CTA pairs.
  const bool single = max_ctas < 0;
  if (single) max_ctas = 0;
  if (M <= 0 || N <= 0 || K <= 0 || (K % 128) != 0 || (N % 8) != 0 || sfa == nullptr ||
      sfb == nullptr) {
    set_last_error("cb_gemm_fp8_mx: need K % 128 == 0, N % 8 == 0 and both scale arrays");
    return -1;
  }
  if (single)
    return launch_plain<GemmCfg<192, 4, true, 1, false, true>>(
        a, b, c, M, N, K, alpha, static_cast<uint32_t*>(status), max_ctas,
        static_cast<cudaStream_t>(stream), static_cast<unsigned long long*>(trace), nullptr,
        nullptr, static_cast<const uint32_t*>(sfa), static_cast<const uint32_t*>(sfb));
  const int sms = max_ctas > 1 && max_ctas < sm_count() ? max_ctas : sm_count();
  if (mx_pair_tile(M, N, K, sms) == 224)
    return launch_plain<GemmCfg<224, 6, true, 2, false, true>>(
        a, b, c, M, N, K, alpha, static_cast<uint32_t*>(status), max_ctas,
        static_cast<cudaStream_t>(stream), static_cast<unsigned long long*>(trace), nullptr, nullptr,
        static_cast<const uint32_t*>(sfa), static_cast<const uint32_t*>(sfb));
  return launch_plain<GemmCfg<192, 6, true, 2, false, true>>(
      a, b, c, M, N, K, alpha, static_cast<uint32_t*>(status), max_ctas,
      static_cast<cudaStream_t>(stream), static_cast<unsigned long long*>(trace), nullptr, nullptr,
      static_cast<const uint32_t*>(sfa), static_cast<const uint32_t*>(sfb));
}

}  // extern "C"
