// Split-key attention forward for calls whose query tiles are too few to fill the chip: decode (a
// few query rows per sequence over a long cache) and short prefill chunks.
//
// What bounds a decode call is reading the cache once: B x Skv x Hkv x 512 bytes.  The tile-pair
// kernel (fa_cp.cuh) gives every query HEAD of a batch its own CTA, so the heads of a group read
// the same keys again, 255 of its 256 query rows are padding, and a batch x head count that is
// small or no multiple of the SM count leaves SMs idle.  Here:
//   * the rows of a 128-row tile are (query row, head of the group) couples of ONE key/value head,
//     loaded as a {64, group, rows} TMA box, so that keys are read once per group;
//   * the work is the flat list of (query tile, batch, key/value head, key block) in that order,
//     cut into equal contiguous ranges, one per CTA, whatever the shapes: a range may start and end
//     inside an item, and a CTA walks its range as a few SEGMENTS of one item each.  Under a causal
//     mask early tiles have few blocks, and an item costs as much as SP_ITEM_COST blocks beside its
//     own (5.5 us for an item of one block, 1.4 us for a block of a long one), so there every item
//     counts that many blocks more in the cut;
//   * inside a CTA two softmax streams take alternate key blocks of the segment, each with its own
//     S / P / O in tensor memory, so that the chain QK -> softmax -> PV of one block overlaps that of
//     the next and the loads (three K and two V tiles in flight, the next segment's Q) never wait
//     for it.  At the end of a segment each stream merges half of the columns of both - a
//     tensor-memory lane is readable from both warp-groups, only (max, sum) goes through shared memory;
//   * a segment that is a whole item writes its output rows; one that is cut leaves its unnormalised
//     fp32 O and (max, sum), which a second kernel, launched as a programmatic dependent, merges
//     per row in the order of the keys.  At most two segments of a CTA are cut - the one it takes over
//     from the CTA before and the one it hands on - so the workspace is two tiles per CTA, 20 MB
//     at most, whatever the batch.
// Measured, tile-pair kernel -> this, kernels alone: 16 sequences x 1 query over 6001 keys, 32 / 8 heads:
// 398 -> 69 us (5.7 TB/s of 6.6; calls in a row 76 to 78); 32 x 16384 keys, 64 / 8 heads: 3783 -> 325 us
// (6.6 TB/s); 1 x 16384 keys, 8 / 8 heads: 259 -> 20 us.
//
// Every mbarrier wait is bounded (see mbarrier.cuh).
#include <math.h>

#include <string>

#include "../gemm/launch.h"
#include "../prim/pdl.cuh"
#include "../symm/driver_api.h"
#include "cp_launch.h"
#include "fa_cp.cuh"

namespace cb {

static constexpr int SP_MAX_QT = 64;                                 // query tiles per batch and head
static constexpr int SP_ITEM_COST = 3;
static constexpr int SP_MERGE_THREADS = 128;
// Microseconds of a unit, of a unit where a batch and head has one query tile (an item of 6 blocks with few rows
// took 10.7 in all), of the merge and of a launch's start and end on the device.
static constexpr float SP_BLOCK_US = 1.35f, SP_ONE_TILE_US = 0.85f, SP_MERGE_US = 6.5f, SP_START_US = 5.7f;

// What a call takes when calls follow each other: on the device, but no less than on the host, where a
// cut costs a workspace and a second launch (measured through flash_attention, 7.1 and 11 us; with 7.5 a call
// that is not cut and takes no longer on the device counts as bound by the host).  Calls that are both bound by
// the host are told apart by the device.
struct CallTime {
  float device;
  bool merge;
  bool better_than(const CallTime& o) const {
    const float a = fmaxf(device, merge ? 11.f : 7.5f), b = fmaxf(o.device, o.merge ? 11.f : 7.5f);
    return a < b || (a == b && device < o.device);
  }
};

struct SplitPlan {
  int B, Sq, Skv, Hq, Hkv, group;
  int qrows;                 // query rows per tile (times group = rows of the tile)
  int nqt;                   // query tiles
  int item_cost;             // units an item counts beside its key blocks
  int per;                   // units per CTA
  int ctas;
  int max_parts;             // CTAs that an item's blocks may be spread over, at most
  int merge;                 // some row is not finished by the first kernel
  int q_offset, kv_offset, causal;
  int nblk[SP_MAX_QT];       // visible key blocks of a tile
  int first[SP_MAX_QT + 1];  // units of the tiles before, for one (batch, head)
};

struct FaSplitParams {
  CUtensorMap tm_q, tm_k, tm_v;   // {128, heads, rows, batch}
  SplitPlan pl;
  float scale_log2;
  float* part_o;                  // [CTA][taken over / handed on][tile row][128] unnormalised
  float2* part_ml;                // [CTA][taken over / handed on][tile row] {max (log2 units), sum}
  __nv_bfloat16* o;               // [B, Sq, Hq, 128]
  float* lse;                     // [B, Hq, Sq] or null
  uint32_t* status;
};

struct SplitCtl {
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[CP_KST], k_empty[CP_KST];
  uint64_t v_full[CP_VST], v_empty[CP_VST];
  uint64_t s_full[2], p_first[2], p_rest[2], pv_done[2];   // per stream; P in halves of 64 keys
  uint64_t seg_full, seg_done;   // both streams' O and (max, sum) of a segment: complete, read
  float2 ml[2][CP_BM];           // (max, sum) of the segment per stream and row
  uint32_t tmem_base;
  int abort_flag;
};

static constexpr int SP_TILES = (2 + CP_KST + CP_VST) * CP_TILE;   // Q x2 | K ring | V ring
static constexpr int SP_SMEM = SP_TILES + static_cast<int>(sizeof(SplitCtl));
static_assert(SP_SMEM <= 232448, "over the 227 KB shared-memory limit");

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, int x, int y,
                                            int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}

// 32 bytes, a whole sector, in one store: rows are 512 bytes apart, and half-sector stores of a
// strided row cost the memory system twice.
__device__ __forceinline__ void st_global_v8(float* dst, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// The segments of one CTA's range of the flat list; every role walks its own copy.  Units are
// 32-bit: the plan keeps their total below 2^30.
struct SplitWalk {
  int pos, end;   // flat units: this segment's first, the range's end
  int qt, bh;     // current item: query tile, batch * Hkv + key/value head
  int k0, n;      // its blocks k0 .. k0 + n - 1 belong to this segment

  __device__ __forceinline__ bool start(const SplitPlan& pl, int cta) {
    const int total = pl.first[pl.nqt] * pl.B * pl.Hkv;
    pos = cta * pl.per;
    end = pos + pl.per < total ? pos + pl.per : total;
    qt = 0;
    return locate(pl);
  }
  __device__ __forceinline__ bool next(const SplitPlan& pl) {
    pos += n;
    return locate(pl);
  }
  // Moves `pos` to the next key block of the range.
  __device__ __forceinline__ bool locate(const SplitPlan& pl) {
    const int items = pl.B * pl.Hkv;
    while (pos < end) {
      while (pos >= pl.first[qt + 1] * items) ++qt;
      const int len = pl.nblk[qt] + pl.item_cost;
      const int in_tile = pos - pl.first[qt] * items;
      bh = in_tile / len;
      const int skip = pl.item_cost - (in_tile - bh * len);   // units before the item's blocks
      if (skip > 0) pos += skip;
      k0 = skip > 0 ? 0 : -skip;
      n = pl.nblk[qt] - k0;
      if (n > end - pos) n = end - pos;
      if (n > 0) return true;
    }
    return false;
  }
};

// Slot of a cut segment of a CTA: the one that begins with its item's first block is handed on, the other
// was taken over.
__device__ __forceinline__ uint32_t split_slot(uint32_t cta, bool begins_item) {
  return 2u * cta + (begins_item ? 1u : 0u);
}

__global__ void __launch_bounds__(CP_THREADS, 1)
    fa_split_kernel(const __grid_constant__ FaSplitParams p) {
  // Seven tiles and the control block leave less than the 1 KB that aligning by hand may take, so the
  // array itself carries the alignment of the swizzled tiles.
  extern __shared__ __align__(1024) uint8_t split_smem[];
  uint8_t* sQ = split_smem;
  if ((smem_u32(sQ) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_status(p.status, CB_BAD_ARGUMENT, 0, 0xF3F);
    return;
  }
  uint8_t* sK = sQ + 2 * CP_TILE;
  uint8_t* sV = sK + CP_KST * CP_TILE;
  SplitCtl& ctl = *reinterpret_cast<SplitCtl*>(split_smem + SP_TILES);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const SplitPlan& pl = p.pl;
  const int tile_rows = pl.qrows * pl.group;
  const uint32_t active = static_cast<uint32_t>(tile_rows + 31) / 32;   // softmax warps per stream

  if (threadIdx.x == 0) {
    for (int i = 0; i < CP_KST; ++i) {
      mbar_init(&ctl.k_full[i], 1);
      mbar_init(&ctl.k_empty[i], 1);
    }
    for (int i = 0; i < CP_VST; ++i) {
      mbar_init(&ctl.v_full[i], 1);
      mbar_init(&ctl.v_empty[i], 1);
    }
    mbar_init(&ctl.seg_full, 2 * active);
    mbar_init(&ctl.seg_done, 2 * active);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl.q_full[i], 1);
      mbar_init(&ctl.q_empty[i], 1);
      mbar_init(&ctl.s_full[i], 1);
      mbar_init(&ctl.p_first[i], active);
      mbar_init(&ctl.p_rest[i], active);
      mbar_init(&ctl.pv_done[i], 1);
    }
    ctl.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();   // the merge kernel waits for this grid's completion itself
  pdl_wait();                // operands, and readers of results and workspace, of the kernels before
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctl.tmem_base);
  // stream t: S (fp32, 128 columns; the first 64 hold P as bf16 pairs after the softmax) at column
  // 256 t, O at column 256 t + 128.

  // 128 x 72 + 256 x 216 registers = 64,512, what 384 threads x 168 were launched with.
  if (warp < 4) {
    cp_reg_dec<72>();
    if (warp == 0) {
      if (lane == 0) {
        // -------------------------------------------------------------- producer
        SplitWalk w;
        bool ok = true;
        int seg = 0, g = 0;
        for (bool more = w.start(pl, blockIdx.x); ok && more; more = w.next(pl), ++seg) {
          const int b = w.bh / pl.Hkv, kvh = w.bh - b * pl.Hkv, qs = seg & 1;
          if (seg > 1)
            ok = mbar_wait(&ctl.q_empty[qs], ((seg >> 1) - 1) & 1, &ctl.abort_flag, p.status, 0xF00);
          if (!ok) break;
          mbar_arrive_expect_tx(&ctl.q_full[qs], static_cast<uint32_t>(tile_rows) * 256u);
          for (int h = 0; h < 2; ++h)
            tma_load_4d(sQ + qs * CP_TILE + h * CP_SUB, &p.tm_q, 64 * h, kvh * pl.group,
                        w.qt * pl.qrows, b, &ctl.q_full[qs]);
          for (int j = 0; ok && j < w.n; ++j, ++g) {
            const int ks = g % CP_KST, kuse = g / CP_KST, vs = g % CP_VST, vuse = g / CP_VST;
            const int row = (w.k0 + j) * CP_BN;
            if (kuse > 0)
              ok = mbar_wait(&ctl.k_empty[ks], (kuse - 1) & 1, &ctl.abort_flag, p.status, 0xF01);
            if (!ok) break;
            mbar_arrive_expect_tx(&ctl.k_full[ks], CP_TILE);
            for (int h = 0; h < 2; ++h)
              tma_load_4d(sK + ks * CP_TILE + h * CP_SUB, &p.tm_k, 64 * h, kvh, row, b,
                          &ctl.k_full[ks]);
            if (vuse > 0)
              ok = mbar_wait(&ctl.v_empty[vs], (vuse - 1) & 1, &ctl.abort_flag, p.status, 0xF02);
            if (!ok) break;
            mbar_arrive_expect_tx(&ctl.v_full[vs], CP_TILE);
            for (int h = 0; h < 2; ++h)
              tma_load_4d(sV + vs * CP_TILE + h * CP_SUB, &p.tm_v, 64 * h, kvh, row, b,
                          &ctl.v_full[vs]);
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------- MMA
      // The whole warp walks the schedule and waits; one elected lane issues.
      constexpr uint32_t idesc_s = make_idesc(128, 128, 1u);
      constexpr uint32_t idesc_pv = make_idesc(128, 128, 1u) | (1u << 16);  // V is MN-major
      const uint64_t q_desc0 = make_sw128_kmajor_desc(smem_u32(sQ));
      const uint64_t k_desc0 = make_sw128_kmajor_desc(smem_u32(sK));
      const uint64_t v_desc0 = cp_mnmajor_desc(smem_u32(sV));
      constexpr uint64_t kTileStep = static_cast<uint64_t>(CP_TILE >> 4);
      constexpr uint64_t kSubStep = static_cast<uint64_t>(CP_SUB >> 4);
      auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t detail) -> bool {
        return mbar_wait_warp(bar, parity, &ctl.abort_flag, p.status, detail);
      };
      int g0 = 0;                 // blocks before this segment
      uint32_t pv_count[2] = {0u, 0u};
      uint64_t q_desc = q_desc0;
      auto issue_qk = [&](int j) -> bool {
        const int g = g0 + j, s = g % CP_KST, t = j & 1;
        if (!wait_all(&ctl.k_full[s], (g / CP_KST) & 1, 0xF11)) return false;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t ka = k_desc0 + s * kTileStep;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint64_t off = (kk >> 2) * kSubStep + 2u * (kk & 3);
            mma_bf16_ss(tmem + 256u * t, q_desc + off, ka + off, idesc_s, kk > 0 ? 1u : 0u);
          }
          mma_commit(&ctl.s_full[t]);
          mma_commit(&ctl.k_empty[s]);
        }
        __syncwarp();
        return true;
      };
      auto issue_pv = [&](int j) -> bool {
        const int g = g0 + j, s = g % CP_VST, t = j & 1;
        const uint32_t par = pv_count[t] & 1u;
        if (!wait_all(&ctl.p_first[t], par, 0xF20 + t)) return false;
        if (!wait_all(&ctl.v_full[s], (g / CP_VST) & 1, 0xF22)) return false;
        ++pv_count[t];
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t va = v_desc0 + s * kTileStep;
          const uint32_t d = tmem + 256u * t + 128u;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_bf16_ts(d, tmem + 256u * t + 8u * kk, va + kk * (2048u >> 4), idesc_pv,
                        (j > 1 || kk > 0) ? 1u : 0u);
        }
        __syncwarp();
        if (!wait_all(&ctl.p_rest[t], par, 0xF24 + t)) return false;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t va = v_desc0 + s * kTileStep;
          const uint32_t d = tmem + 256u * t + 128u;
#pragma unroll
          for (int kk = 4; kk < 8; ++kk)
            mma_bf16_ts(d, tmem + 256u * t + 8u * kk, va + kk * (2048u >> 4), idesc_pv, 1u);
          mma_commit(&ctl.pv_done[t]);
          mma_commit(&ctl.v_empty[s]);
        }
        __syncwarp();
        return true;
      };
      SplitWalk w;
      bool ok = true;
      int seg = 0;
      for (bool more = w.start(pl, blockIdx.x); ok && more; more = w.next(pl), ++seg) {
        ok = wait_all(&ctl.q_full[seg & 1], (seg >> 1) & 1, 0xF10);
        q_desc = q_desc0 + (seg & 1) * kTileStep;
        for (int j = 0; ok && j < 2 && j < w.n; ++j) ok = issue_qk(j);
        for (int j = 0; ok && j < w.n; ++j) {
          // A stream's first product of a segment overwrites the O of its last one: that was read
          // before its softmax warps hand over (p_first) the first block of this segment.
          ok = issue_pv(j);
          if (ok && j + 2 < w.n) ok = issue_qk(j + 2);
        }
        if (ok && elect_one()) mma_commit(&ctl.q_empty[seg & 1]);
        __syncwarp();
        g0 += w.n;
      }
    }
  } else {
    cp_reg_inc<216>();
    // ----------------------------------------------------------------- softmax
    const int t = warp >= 8 ? 1 : 0;
    const uint32_t q = warp & 3u;
    const int r = static_cast<int>(q * 32u + lane);        // tile row of this thread
    const uint32_t lane_addr = (q * 32u) << 16;
    const uint32_t tS = tmem + 256u * t + lane_addr;
    const uint32_t tO = tS + 128u;
    const int q_in_tile = r / pl.group;
    SplitWalk w;
    bool ok = q < active;
    uint32_t count = 0;                                    // blocks this stream has seen
    int seg = 0;
    for (bool more = w.start(pl, blockIdx.x); ok && more; more = w.next(pl), ++seg) {
      const int tile_first = pl.q_offset + w.qt * pl.qrows;   // position of the tile's first query
      const int q_pos = tile_first + q_in_tile;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = t; ok && j < w.n; j += 2) {
        if (!mbar_wait(&ctl.s_full[t], count & 1u, &ctl.abort_flag, p.status, 0xF30 + t)) {
          ok = false;
          break;
        }
        ++count;
        tc_fence_after_sync();
        uint32_t s[128];
        tmem_ld_32x32_at(tS, &s[0]);
        tmem_ld_32x32_at(tS + 32u, &s[32]);
        tmem_ld_32x32_at(tS + 64u, &s[64]);
        tmem_ld_32x32_at(tS + 96u, &s[96]);
        tmem_wait_ld();
        const int kb = (w.k0 + j) * CP_BN;
        const int key0 = pl.kv_offset + kb;
        const int kv_left = pl.Skv - kb;
        const bool need_mask = kv_left < CP_BN || (pl.causal && key0 + CP_BN - 1 > tile_first);
        if (need_mask) cp_mask_tail(s, pl.causal ? min(kv_left, q_pos - key0 + 1) : kv_left);
        float mx8[8];
        cp_row_max(s, mx8);
        cp_update_max(mx8, tO, p.scale_log2, j > 1, r < tile_rows, m_ref, l);
        uint64_t sum4[4] = {0ull, 0ull, 0ull, 0ull};
        cp_probabilities<0, 0, 64>(s, p.scale_log2, m_ref, need_mask, sum4);
        tmem_st_32x32_at(tS, &s[0]);
        tmem_wait_st();
        // Both streams' O of the segment before must have been read before this hand-over.
        if (j < 2 && seg > 0 &&
            !mbar_wait(&ctl.seg_done, (seg - 1) & 1, &ctl.abort_flag, p.status, 0xF32)) {
          ok = false;
          break;
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.p_first[t]);
        cp_probabilities<0, 64, 128>(s, p.scale_log2, m_ref, need_mask, sum4);
        tmem_st_32x32_at(tS + 32u, &s[32]);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.p_rest[t]);
        cp_add_sums(sum4, l);
      }
      if (!ok) break;
      // -------------------------------------------- end of the segment: merge the streams
      if (t < w.n) {
        ok = mbar_wait(&ctl.pv_done[t], (count - 1u) & 1u, &ctl.abort_flag, p.status, 0xF34 + t);
      } else if (seg > 0) {   // no block, so no wait for the last segment's readers yet
        ok = mbar_wait(&ctl.seg_done, (seg - 1) & 1, &ctl.abort_flag, p.status, 0xF33);
      }
      if (!ok) break;
      ctl.ml[t][r] = make_float2(m_ref, l);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.seg_full);
      if (!mbar_wait(&ctl.seg_full, seg & 1, &ctl.abort_flag, p.status, 0xF36)) break;
      tc_fence_after_sync();
      const float2 ml0 = ctl.ml[0][r], ml1 = ctl.ml[1][r];
      const float m = fmaxf(ml0.x, ml1.x);
      // A stream without a visible key has no O: its columns may hold anything.
      const bool use0 = ml0.y != 0.f, use1 = ml1.y != 0.f;
      const float a0 = use0 ? exp2f(ml0.x - m) : 0.f, a1 = use1 ? exp2f(ml1.x - m) : 0.f;
      const float lsum = (use0 ? a0 * ml0.y : 0.f) + (use1 ? a1 * ml1.y : 0.f);
      const int b = w.bh / pl.Hkv, kvh = w.bh - b * pl.Hkv;
      const int srow = w.qt * pl.qrows + q_in_tile, h = kvh * pl.group + (r - q_in_tile * pl.group);
      const bool row_ok = r < tile_rows && srow < pl.Sq;
      const bool whole = w.n == pl.nblk[w.qt];
      const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
      const size_t part = static_cast<size_t>(split_slot(blockIdx.x, w.k0 == 0)) * tile_rows + r;
#pragma unroll 1
      for (int c = 2 * t; c < 2 * t + 2; ++c) {
        uint32_t o0[32], o1[32];
        tmem_ld_32x32(tmem + lane_addr + 128u + c * 32u, o0);
        tmem_ld_32x32(tmem + lane_addr + 384u + c * 32u, o1);
        tmem_wait_ld();
        float o[32];
#pragma unroll
        for (int i = 0; i < 32; ++i)
          o[i] = (use0 ? a0 * __uint_as_float(o0[i]) : 0.f) + (use1 ? a1 * __uint_as_float(o1[i]) : 0.f);
        if (!row_ok) continue;
        if (whole) {
          __nv_bfloat16* dst =
              p.o + ((static_cast<size_t>(b) * pl.Sq + srow) * pl.Hq + h) * CP_D + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              hh[k] = __floats2bfloat162_rn(o[i + 2 * k] * inv, o[i + 2 * k + 1] * inv);
            *reinterpret_cast<uint4*>(dst + i) = v;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 8) st_global_v8(p.part_o + part * CP_D + c * 32 + i, o + i);
        }
      }
      if (t == 0 && row_ok) {
        if (!whole)
          p.part_ml[part] = make_float2(m, lsum);
        else if (p.lse != nullptr)
          p.lse[(static_cast<size_t>(b) * pl.Hq + h) * pl.Sq + srow] =
              lsum > 0.f ? m * 0.6931471805599453f + logf(lsum) : -INFINITY;
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.seg_done);
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*reinterpret_cast<volatile int*>(&ctl.abort_flag) != 0) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

// Merges the partial results of a row: out = sum_i 2^(m_i - M) O_i / sum_i 2^(m_i - M) l_i, in the
// order of the key blocks, with the maximum kept running.  A lane holds four of the 128 columns.
// kWide: the CTA's four warps take a quarter of a row's parts each (decode: few rows, many parts);
// else a warp takes a row.  Bound by latency, so a step loads (max, sum) and O of eight parts
// together and indices are 32-bit.
template <bool kWide>
__global__ void __launch_bounds__(SP_MERGE_THREADS, 6)
    fa_split_merge_kernel(const __grid_constant__ FaSplitParams p) {
  pdl_wait();
  const SplitPlan& pl = p.pl;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  constexpr uint32_t kWarps = SP_MERGE_THREADS / 32;
  const uint32_t row = kWide ? blockIdx.x : blockIdx.x * kWarps + warp;
  const uint32_t Hq = pl.Hq, Sq = pl.Sq, group = pl.group, per = pl.per;
  if (row >= pl.B * Sq * Hq) return;
  const uint32_t bs = row / Hq, h = row - bs * Hq;
  const uint32_t b = bs / Sq, s = bs - b * Sq;
  const uint32_t kvh = h / group, qt = s / pl.qrows;
  const uint32_t r = (s - qt * pl.qrows) * group + (h - kvh * group);
  const uint32_t tile_rows = pl.qrows * group;
  const uint32_t items = pl.B * pl.Hkv, item = b * pl.Hkv + kvh;
  const uint32_t n = pl.nblk[qt];
  const uint32_t start = pl.first[qt] * items + item * (n + pl.item_cost) + pl.item_cost;
  const uint32_t cta0 = start / per;   // its part i is CTA cta0 + i's
  const int parts = n == 0 ? 0 : static_cast<int>((start + n - 1) / per - cta0 + 1);
  if (parts == 1) return;           // the row is final
  const float2* ml = p.part_ml + r;
  const float4* po = reinterpret_cast<const float4*>(p.part_o + static_cast<size_t>(r) * CP_D) + lane;

  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float m = -INFINITY, l = 0.f;
  const int chunk = kWide ? (parts + static_cast<int>(kWarps) - 1) / static_cast<int>(kWarps) : parts;
  const int i0 = kWide ? static_cast<int>(warp) * chunk : 0;
  const int i1 = i0 + chunk < parts ? i0 + chunk : parts;
#pragma unroll 1
  for (int base = i0; base < i1; base += 8) {
    float4 v[8];
    float2 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x[u] = make_float2(-INFINITY, 0.f);
      if (base + u < i1) {
        const uint32_t row = split_slot(cta0 + base + u, base + u == 0) * tile_rows;
        x[u] = ml[row];
        v[u] = po[row * (CP_D / 4)];
      }
    }
    float m_new = m;
#pragma unroll
    for (int u = 0; u < 8; ++u) m_new = fmaxf(m_new, x[u].x);
    const float keep = m == -INFINITY ? 0.f : exp2f(m - m_new);
    m = m_new;
    l *= keep;
    acc = make_float4(acc.x * keep, acc.y * keep, acc.z * keep, acc.w * keep);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (x[u].y != 0.f) {          // a part without a visible key adds nothing
        const float w = exp2f(x[u].x - m);
        l += w * x[u].y;
        acc.x += w * v[u].x;
        acc.y += w * v[u].y;
        acc.z += w * v[u].z;
        acc.w += w * v[u].w;
      }
    }
  }
  if constexpr (kWide) {
    __shared__ float4 sh_o[kWarps][32];
    __shared__ float2 sh_ml[kWarps];
    sh_o[warp][lane] = acc;
    if (lane == 0) sh_ml[warp] = make_float2(m, l);
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (uint32_t i = 1; i < kWarps; ++i) m = fmaxf(m, sh_ml[i].x);
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    l = 0.f;
#pragma unroll
    for (uint32_t i = 0; i < kWarps; ++i) {
      if (sh_ml[i].y == 0.f) continue;
      const float4 v = sh_o[i][lane];
      const float w = exp2f(sh_ml[i].x - m);
      l += w * sh_ml[i].y;
      acc.x += w * v.x;
      acc.y += w * v.y;
      acc.z += w * v.z;
      acc.w += w * v.w;
    }
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  __nv_bfloat162 o2[2] = {__floats2bfloat162_rn(acc.x * inv, acc.y * inv),
                          __floats2bfloat162_rn(acc.z * inv, acc.w * inv)};
  *reinterpret_cast<uint2*>(p.o + static_cast<size_t>(row) * CP_D + lane * 4) =
      *reinterpret_cast<uint2*>(o2);
  if (lane == 0 && p.lse != nullptr)
    p.lse[(static_cast<size_t>(b) * Hq + h) * Sq + s] =
        l > 0.f ? m * 0.6931471805599453f + logf(l) : -INFINITY;
}

// A call is cut, and given to this kernel, at one and the same price of a unit.
static float unit_us(const SplitPlan& pl) { return pl.nqt == 1 ? SP_ONE_TILE_US : SP_BLOCK_US; }

// Fills the plan; false when the call does not fit this kernel (or has no key block at all).
static bool split_plan(SplitPlan& pl, int B, int Sq, int Skv, int Hq, int Hkv, int q_offset,
                       int kv_offset, int causal, int sms) {
  pl.B = B;
  pl.Sq = Sq;
  pl.Skv = Skv;
  pl.Hq = Hq;
  pl.Hkv = Hkv;
  pl.group = Hq / Hkv;
  pl.q_offset = q_offset;
  pl.kv_offset = kv_offset;
  pl.causal = causal;
  if (pl.group > CP_BM) return false;
  pl.qrows = CP_BM / pl.group;
  if (pl.qrows > Sq) pl.qrows = Sq;
  pl.nqt = (Sq + pl.qrows - 1) / pl.qrows;
  if (pl.nqt > SP_MAX_QT) return false;
  const int all = (Skv + CP_BN - 1) / CP_BN;
  pl.item_cost = causal && pl.nqt > 1 ? SP_ITEM_COST : 0;
  pl.first[0] = 0;
  int blocks = 0;
  for (int i = 0; i < pl.nqt; ++i) {
    int n = all;
    if (causal) {
      const int rows = i + 1 < pl.nqt ? (i + 1) * pl.qrows : Sq;
      const long long lim = static_cast<long long>(q_offset) + rows - 1 - kv_offset;
      const long long c = lim < 0 ? 0 : lim / CP_BN + 1;
      if (c < n) n = static_cast<int>(c);
    }
    pl.nblk[i] = n;
    blocks += n;
    pl.first[i + 1] = pl.first[i] + n + pl.item_cost;
  }
  const long long items = static_cast<long long>(B) * Hkv;
  const long long total = static_cast<long long>(pl.first[pl.nqt]) * items;
  if (blocks < 1 || total > 0x3fffffffll) return false;
  if (static_cast<long long>(B) * Sq * Hq > 0x3fffffffll) return false;   // 32-bit rows in the merge
  pl.per = static_cast<int>((total + sms - 1) / sms);
  if (pl.nqt == 1) {
    // Whole items per CTA when that costs less than the merge.
    const long long whole = (items + sms - 1) / sms * pl.nblk[0];
    const CallTime uncut = {SP_START_US + unit_us(pl) * static_cast<float>(whole), false};
    if (uncut.better_than({SP_START_US + unit_us(pl) * static_cast<float>(pl.per) + SP_MERGE_US, true}))
      pl.per = static_cast<int>(whole);
  }
  pl.ctas = static_cast<int>((total + pl.per - 1) / pl.per);
  pl.max_parts = (all + pl.per - 2) / pl.per + 1;
  pl.merge = 0;
  for (int i = 0; i < pl.nqt; ++i)
    if (pl.nblk[i] == 0) pl.merge = 1;      // rows that see no key get their zeros there
  for (int c = 1, qt = 0; c < pl.ctas && pl.merge == 0; ++c) {
    const long long pos = static_cast<long long>(c) * pl.per;
    while (pos >= pl.first[qt + 1] * items) ++qt;
    const long long in_item = (pos - pl.first[qt] * items) % (pl.nblk[qt] + pl.item_cost);
    if (in_item > pl.item_cost) pl.merge = 1;   // cut inside an item
  }
  return true;
}

static int split_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
    return 148;
  return n;
}

// Which kernel takes a call, from a model of both in microseconds.  The tile-pair kernel takes
// kPairBlock for a key block of its 256 rows and is as long as its longest item or its share of all
// of them; the split kernel takes unit_us for a unit of its 128 rows, plus the merge.
// Measured, calls in a row, split / pair (B, Sq, Skv, Hq, Hkv): (1, 537, 537, 8, 2) 12.2 / 15.4 us,
// (1, 8192, 8192, 4, 4) 93 / 128; near the line (1, 64, 64, 4, 4) 7.7 / 7.3, (1, 300, 300, 4, 1) 12.2 / 11.9,
// (1, 896, 896, 16, 4) 20.3 / 19.4, (1, 1280, 1280, 16, 8) 27.7 / 26.3, (1, 2000, 2777, 16, 4) 52 / 47,
// (1, 1000, 7000, 32, 8) 111 / 116; beyond it, every key visible, (2, 218, 995, 32, 8) 26.8 / 21.8; one query
// tile, more items than SMs: (20, 1, 1275, 8, 8) 29 / 42, (24, 4, 1403, 8, 8) 36 / 47, (25, 128, 1275, 8, 8)
// 37 / 47.  Over 68
// shapes of that range the choice takes 1.1 % more than the better kernel on average (2.1 % with the constants
// of before the two kernels and their call path became faster).
static bool split_wins(const SplitPlan& pl, int sms) {
  constexpr float kPairBlock = 1.8f, kPairStart = 7.f;
  const float pair_tiles = static_cast<float>((pl.Sq + 2 * CP_BM - 1) / (2 * CP_BM));
  float blocks = 0.f;
  for (int i = 0; i < pl.nqt; ++i) blocks += static_cast<float>(pl.nblk[i]);
  const float avg = blocks / static_cast<float>(pl.nqt);
  const float share = avg * pair_tiles * static_cast<float>(pl.Hq) * static_cast<float>(pl.B) /
                      static_cast<float>(sms);
  const float longest = static_cast<float>(pl.nblk[pl.nqt - 1]);
  const CallTime pair = {kPairStart + kPairBlock * (share > longest ? share : longest), false};
  const CallTime split = {SP_START_US + (pl.merge ? SP_MERGE_US : 0.f) +
                              unit_us(pl) * static_cast<float>(pl.per),
                          pl.merge != 0};
  return split.better_than(pair);
}

// Rows of partial results, and the bytes they take (none when no item is cut).
static size_t split_rows(const SplitPlan& pl) {
  return 2ull * pl.ctas * pl.qrows * pl.group;
}
static long long split_bytes(const SplitPlan& pl) {
  return pl.merge ? static_cast<long long>(split_rows(pl) * (CP_D * sizeof(float) + sizeof(float2)))
                  : 0;
}

static int split_tmap(CUtensorMap* out, const void* base, int heads, int rows, int batch,
                      int box_heads, int box_rows) {
  const DriverApi& d = driver_api();
  if (!d.ok) {
    set_last_error("tensor map: " + d.why);
    return -1;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) {
    set_last_error("attention: tensors must be 16-byte aligned");
    return -1;
  }
  const cuuint64_t row_bytes = static_cast<cuuint64_t>(heads) * CP_D * 2ull;
  cuuint64_t dims[4] = {CP_D, static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(rows),
                        static_cast<cuuint64_t>(batch)};
  cuuint64_t strides[3] = {CP_D * 2ull, row_bytes, row_bytes * static_cast<cuuint64_t>(rows)};
  cuuint32_t box[4] = {64, static_cast<cuuint32_t>(box_heads), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = d.cuTensorMapEncodeTiled(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                                        const_cast<void*>(base), dims, strides, box, estr,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error(cu_err("cuTensorMapEncodeTiled(split attention)", r));
    return -1;
  }
  return 0;
}

}  // namespace cb

using namespace cb;

extern "C" {

// Bytes of workspace with which cb_attn_split runs this call (0: none, no item is cut), or -1: the
// call belongs to the tile-pair kernel (cb_attn_fwd4).
long long cb_attn_split_bytes(int B, int Sq, int Skv, int Hq, int Hkv, int q_offset, int kv_offset,
                              int causal) {
  if (B < 1 || Sq < 1 || Skv < 1 || Hq < 1 || Hkv < 1 || Hq % Hkv != 0) return -1;
  SplitPlan pl;
  const int sms = split_sms();
  if (!split_plan(pl, B, Sq, Skv, Hq, Hkv, q_offset, kv_offset, causal, sms)) return -1;
  if (!split_wins(pl, sms)) return -1;
  return split_bytes(pl);
}

// Arguments as cb_attn_fwd4 (lse may be null); `workspace`: at least cb_attn_split_bytes() bytes,
// 32-byte aligned, used until the launches on `stream` have completed.
int cb_attn_split(const void* q, const void* k, const void* v, void* o, void* lse, int B, int Sq,
                  int Skv, int Hq, int Hkv, int q_offset, int kv_offset, int causal, float scale,
                  void* workspace, long long workspace_bytes, void* status, void* stream) {
  if (B < 1 || Sq < 1 || Skv < 1 || Hq < 1 || Hkv < 1 || Hq % Hkv != 0) {
    set_last_error("attention: bad shape (Hq must be a multiple of Hkv)");
    return -1;
  }
  FaSplitParams p;
  if (!split_plan(p.pl, B, Sq, Skv, Hq, Hkv, q_offset, kv_offset, causal, split_sms())) {
    set_last_error("split attention: more query tiles or heads per group than this kernel takes, "
                   "or no visible key");
    return -1;
  }
  const long long need = split_bytes(p.pl);
  if (need > 0 && (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 31u) != 0 ||
                   workspace_bytes < need)) {
    set_last_error("split attention: workspace missing, misaligned or too small");
    return -1;
  }
  if (split_tmap(&p.tm_q, q, Hq, Sq, B, p.pl.group, p.pl.qrows)) return -1;
  if (split_tmap(&p.tm_k, k, Hkv, Skv, B, 1, CP_BN)) return -1;
  if (split_tmap(&p.tm_v, v, Hkv, Skv, B, 1, CP_BN)) return -1;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.part_o = static_cast<float*>(workspace);
  p.part_ml = reinterpret_cast<float2*>(p.part_o + split_rows(p.pl) * CP_D);
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = static_cast<float*>(lse);
  p.status = static_cast<uint32_t*>(status);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  static std::atomic<uint64_t> smem_done{0};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(fa_split_kernel), SP_SMEM, smem_done);
  if (e == cudaSuccess) {
    e = launch_pdl(fa_split_kernel, dim3(static_cast<unsigned>(p.pl.ctas)), dim3(CP_THREADS), SP_SMEM, st, p);
  }
  if (e == cudaSuccess && p.pl.merge) {
    const long long rows = static_cast<long long>(B) * Sq * Hq;
    if (p.pl.max_parts > 8)
      e = launch_pdl(fa_split_merge_kernel<true>, dim3(static_cast<unsigned>(rows)),
                     dim3(SP_MERGE_THREADS), 0, st, p);
    else
      e = launch_pdl(fa_split_merge_kernel<false>,
                     dim3(static_cast<unsigned>((rows + 3) / 4)), dim3(SP_MERGE_THREADS), 0, st, p);
  }
  if (e != cudaSuccess) {
    set_last_error(std::string("split attention launch: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // extern "C"
