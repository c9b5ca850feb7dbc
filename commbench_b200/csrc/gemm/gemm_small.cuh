// GEMM for problems whose tiles are too few to fill the chip: decode batches, narrow layers.
//   C[M,N] = alpha * A[M,K] * B[N,K]^T, bf16 or fp8 e4m3 in, fp32 accumulation, bf16 out
//
// The persistent core (gemm_sm100.cuh) walks K serially in one CTA per tile; with fewer tiles than
// SMs a call lasts as long as its K loop, and that loop cannot run faster than its two issuing
// warps: waits, election, four MMAs and a commit are about 500 cycles per 128-byte K block whatever
// the tile's width.  This kernel therefore
//   * splits K over the CTAs of a cluster (1, 2, 4 or 8): every CTA leaves its fp32 partial tile in its
//     own shared memory and, after a cluster barrier, adds up and stores its share of the tile, reading
//     the partners' parts through distributed shared memory in rank order - no workspace, no
//     atomics, the same bits every time;
//   * hands operands over KPS K blocks at a time: one wait, one election, one commit for 4 x KPS MMAs;
//   * loads only the rows of A that exist (a box of M rounded up to 8), since the rows beyond are never
//     stored, into ring slots of that height: with 48 rows 6 instead of 4 slots of two 64-wide K blocks, so that
//     more weights are on their way (bound by them: 48 x 3584 x 8192 in 64-wide tiles 16.6 -> 15.9 us, 128-wide
//     15.5 -> 14.8, 48 x 8192 x 3584 14.3 -> 13.8, all with weights out of memory);
//   * is chained with programmatic dependent launch, so that its set-up overlaps the tail of the
//     kernel before.
// One tile per cluster.  Every mbarrier wait is bounded; an abort leaves through the cluster barriers.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "../prim/cluster.cuh"
#include "../prim/pdl.cuh"
#include "../prim/tcgen05.cuh"
#include "../prim/tma.cuh"
#include "gemm_sm100.cuh"

namespace cb {

template <int BN_, bool FP8_>
struct SmallCfg {
  static constexpr int BN = BN_;
  static constexpr bool FP8 = FP8_;
  static constexpr int BM = 128;
  static constexpr int BK = FP8_ ? 128 : 64;               // elements per 128-byte row
  static constexpr int KPS = BN_ <= 128 ? 2 : 1;           // K blocks per ring stage
  static constexpr int STAGES = BN_ == 128 ? 3 : 4;
  static constexpr int A_BYTES = BM * 128;
  static constexpr int B_BYTES = BN_ * 128;
  static constexpr int KB_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGE_BYTES = KPS * KB_BYTES;
  static constexpr int PITCH = BN_ + 4;                    // floats per staged row: no bank conflicts
  static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
  static constexpr int MAX_STAGES = 12;   // barriers of a ring: 10 slots with 8 rows of A in 64-wide tiles, 5 in others
  static constexpr int SMEM_BYTES = RING_BYTES + 1024;
  // Ring slots for A boxes of a_rows rows.  The MMA reads 128 rows from an A slot's start: what follows the
  // rows that were loaded is other operands, whose products are never stored, but it has to lie in the ring.
  static constexpr int stages(int a_rows) {
    const int kb = a_rows * 128 + B_BYTES;
    const int beyond = A_BYTES > kb ? A_BYTES - kb : 0;
    const int n = (RING_BYTES - beyond) / (KPS * kb);
    return n < MAX_STAGES ? n : MAX_STAGES;
  }
  static constexpr int THREADS = 192;                      // producer, MMA, 4 epilogue warps
  static_assert(BM * PITCH * 4 <= RING_BYTES, "the staged tile reuses the operand ring");
  static_assert(SMEM_BYTES <= 232448 - 256, "over the 227 KB shared-memory limit");
};

struct SmallParams {
  CUtensorMap tm_a, tm_b;   // boxes: 128 bytes x a_rows, 128 bytes x BN
  __nv_bfloat16* c;
  int M, N, num_m, num_kb;  // K blocks of the whole product
  int a_rows;               // rows of the A box
  int stages;               // ring slots: Cfg::stages(a_rows)
  float alpha;
  uint32_t* status;
};

template <class Cfg>
struct SmallCtl {
  uint64_t full[Cfg::MAX_STAGES], empty[Cfg::MAX_STAGES], done;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

template <class Cfg, int SPLIT>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
    gemm_small_kernel(const __grid_constant__ SmallParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
  __shared__ SmallCtl<Cfg> ctl;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const int rank = SPLIT > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / SPLIT;
  // row blocks of a column block run side by side: they share the B tile through L2
  const int n_blk = tile / p.num_m, m_blk = tile - n_blk * p.num_m;
  const int kb0 = p.num_kb * rank / SPLIT, nkb = p.num_kb * (rank + 1) / SPLIT - kb0;

  if (threadIdx.x == 0) {
    tmap_prefetch(&p.tm_a);
    tmap_prefetch(&p.tm_b);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 1);
    }
    mbar_init(&ctl.done, 1);
    ctl.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_base, Cfg::BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctl.tmem_base);
  const uint32_t a_bytes = static_cast<uint32_t>(p.a_rows) * 128u;
  const uint32_t kb_step = a_bytes + Cfg::B_BYTES, stage_step = Cfg::KPS * kb_step;
  const uint32_t stages = static_cast<uint32_t>(p.stages);
  pdl_launch_dependents();
  pdl_wait();   // operands, and readers of C, of the kernels before

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    const uint32_t ring_addr = smem_u32(ring), full0 = smem_u32(&ctl.full[0]);
    uint32_t stage = 0, phase = 0, slot = ring_addr;
    for (int kb = 0; kb < nkb; kb += Cfg::KPS) {
      if (!mbar_wait_traced(&ctl.empty[stage], phase ^ 1u, &ctl.abort_flag, p.status, 0x100 + stage,
                            false, nullptr))
        break;
      if (elect_one()) {
        const int sub = nkb - kb < Cfg::KPS ? nkb - kb : Cfg::KPS;
        const uint32_t bar = full0 + stage * 8u;
        mbar_arrive_expect_tx_addr(bar, kb_step * sub);
#pragma unroll
        for (int i = 0; i < Cfg::KPS; ++i) {
          if (i >= sub) break;
          const uint32_t sa = slot + i * kb_step;
          const int x = (kb0 + kb + i) * Cfg::BK;
          tma_load_2d_addr(sa + a_bytes, &p.tm_b, x, n_blk * Cfg::BN, bar);
          tma_load_2d_addr(sa, &p.tm_a, x, m_blk * Cfg::BM, bar);
        }
      }
      __syncwarp();
      slot += stage_step;
      if (++stage == stages) {
        stage = 0;
        slot = ring_addr;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------- MMA
    constexpr uint32_t idesc = make_idesc(Cfg::BM, Cfg::BN, Cfg::FP8 ? 0u : 1u);
    const uint64_t a_desc0 = make_sw128_kmajor_desc(smem_u32(ring));
    uint32_t stage = 0, phase = 0;
    const uint64_t kb_desc = kb_step >> 4, b_desc = a_bytes >> 4, stage_desc = stage_step >> 4;
    uint64_t a_desc = a_desc0;
    bool ok = true;
    for (int kb = 0; kb < nkb; kb += Cfg::KPS) {
      if (!mbar_wait_traced(&ctl.full[stage], phase, &ctl.abort_flag, p.status, 0x300 + stage, false,
                            nullptr)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const int sub = nkb - kb < Cfg::KPS ? nkb - kb : Cfg::KPS;
      if (elect_one()) {
#pragma unroll
        for (int i = 0; i < Cfg::KPS; ++i) {
          if (i >= sub) break;
          const uint64_t ad = a_desc + i * kb_desc;
          const uint64_t bd = ad + b_desc;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t accum = (kb > 0 || i > 0 || k > 0) ? 1u : 0u;
            if constexpr (Cfg::FP8)
              mma_fp8_ss(tmem, ad + 2u * k, bd + 2u * k, idesc, accum);
            else
              mma_bf16_ss(tmem, ad + 2u * k, bd + 2u * k, idesc, accum);
          }
        }
        mma_commit(&ctl.empty[stage]);
      }
      __syncwarp();
      a_desc += stage_desc;
      if (++stage == stages) {
        stage = 0;
        a_desc = a_desc0;
        phase ^= 1u;
      }
    }
    if (ok && elect_one()) mma_commit(&ctl.done);
    __syncwarp();
  }

  // ------------------------------------------------------------------ epilogue
  const int rows = p.M - m_blk * Cfg::BM < Cfg::BM ? p.M - m_blk * Cfg::BM : Cfg::BM;
  float* stagef = reinterpret_cast<float*>(ring);
  if (warp >= 2) {
    const uint32_t q = warp & 3u;
    const int r = static_cast<int>(q * 32u + lane);
    // `done` also says that no load and no MMA uses the ring any more.
    if (mbar_wait_traced(&ctl.done, 0, &ctl.abort_flag, p.status, 0x400, false, nullptr)) {
      tc_fence_after_sync();
      if (static_cast<int>(q) * 32 < rows) {
#pragma unroll 1
        for (int c = 0; c < Cfg::BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(tmem + ((q * 32u) << 16) + c * 32u, v);
          tmem_wait_ld();
          if (r < rows) {
            float4* dst = reinterpret_cast<float4*>(stagef + r * Cfg::PITCH + c * 32);
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              dst[i / 4] = make_float4(__uint_as_float(v[i]), __uint_as_float(v[i + 1]),
                                       __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
          }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  if constexpr (SPLIT > 1) cluster_sync_all();
  else __syncthreads();

  // Units of 8 columns, this CTA's share of the tile; parts are added in rank order.
  {
    constexpr int kUnits = Cfg::BN / 8;
    const int units = rows * kUnits;
    const int u1 = units * (rank + 1) / SPLIT;
    uint32_t base[SPLIT];
#pragma unroll
    for (int s = 0; s < SPLIT; ++s)
      base[s] = SPLIT > 1 ? map_to_cta(smem_u32(stagef), static_cast<uint32_t>(s)) : smem_u32(stagef);
    for (int u = units * rank / SPLIT + static_cast<int>(threadIdx.x); u < u1; u += Cfg::THREADS) {
      const int r = u / kUnits, cu = u - r * kUnits;
      const int col = n_blk * Cfg::BN + cu * 8;
      if (col >= p.N) continue;
      const uint32_t off = static_cast<uint32_t>(r * Cfg::PITCH + cu * 8) * 4u;
      float4 x[SPLIT], y[SPLIT];
#pragma unroll
      for (int s = 0; s < SPLIT; ++s) {
        x[s] = ld_cluster_v4(base[s] + off);
        y[s] = ld_cluster_v4(base[s] + off + 16u);
      }
#pragma unroll
      for (int s = 1; s < SPLIT; ++s) {
        x[0] = make_float4(x[0].x + x[s].x, x[0].y + x[s].y, x[0].z + x[s].z, x[0].w + x[s].w);
        y[0] = make_float4(y[0].x + y[s].x, y[0].y + y[s].y, y[0].z + y[s].z, y[0].w + y[s].w);
      }
      uint4 o;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
      h[0] = __floats2bfloat162_rn(x[0].x * p.alpha, x[0].y * p.alpha);
      h[1] = __floats2bfloat162_rn(x[0].z * p.alpha, x[0].w * p.alpha);
      h[2] = __floats2bfloat162_rn(y[0].x * p.alpha, y[0].y * p.alpha);
      h[3] = __floats2bfloat162_rn(y[0].z * p.alpha, y[0].w * p.alpha);
      *reinterpret_cast<uint4*>(p.c + static_cast<size_t>(m_blk * Cfg::BM + r) * p.N + col) = o;
    }
  }
  // Partners may still be reading this CTA's part.
  if constexpr (SPLIT > 1) cluster_sync_all();
  else __syncthreads();
  if (*reinterpret_cast<volatile int*>(&ctl.abort_flag) != 0) {
    // A wait gave up: loads may still be landing here.  Bounded grace period.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem, Cfg::BN);
  }
}

}  // namespace cb
