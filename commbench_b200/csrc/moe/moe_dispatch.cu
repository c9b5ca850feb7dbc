// Dispatch push (fp8 quantisation fused into the send), dequantising receive,
// SwiGLU and the weighted combine reduction.  See moe_kernels.cu for the overall
// design and the reference counterparts.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../prim/barrier.cuh"
#include "../prim/pdl.cuh"

namespace cb {
void set_last_error(const std::string& s);

enum : uint32_t { PH_MOE_ARRIVE2 = 48, PH_MOE_COMBINE2 = 49 };

// Eight e4m3 values times their block's scale, as bf16.
__device__ __forceinline__ uint4 expand_fp8x8(uint2 raw, float s) {
  const __nv_fp8x2_storage_t* p8 = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
  uint4 o;
  __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p8[i], __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
    ob[i] = __floats2bfloat162_rn(f.x * s, f.y * s);
  }
  return o;
}

struct MoeSendArgs {
  const __nv_bfloat16* x;     // [T, H] this rank's tokens
  const int* topk_idx;        // [T*K]
  const int* slot;            // [T*K] position of a selection among this rank's of the same expert
  const int* send_row_base;   // [E] first destination row
  __nv_bfloat16* a_out;       // bf16 [max_rows, H] grouped-GEMM input of THIS rank
  uint8_t* recv_x[CB_MAX_RANKS];      // fp8 [max_rows, H] on each rank
  float* recv_scale[CB_MAX_RANKS];    // [max_rows, H/128]
  int2* recv_meta[CB_MAX_RANKS];      // [max_rows] {source rank, source pair index}
  uint32_t* arrived[CB_MAX_RANKS];    // [E/W] rows arrived per local expert
  int rank, world, T, K, H, E, max_rows;
  uint32_t* status;
  int per_token;              // 1: one copy of a token per destination RANK (see the kernel)
};

// Token-major dispatch: a warp loads up to 1024 columns of a token ONCE, quantises them ONCE
// (per-128-channel absmax -> scale -> e4m3) and writes them to every row that the token's K
// selections have; all slices of a token belong to one CTA, which at its end bumps the arrival counter
// of every expert it wrote rows for.
//
// Rows for another rank go there as fp8 plus scales.  Rows for an expert of THIS rank never take
// the fp8 detour through memory: the quantised values, expanded to bf16 exactly as the receive
// kernel would, are written straight into the grouped GEMM's input.
//
// per_token = 0 (expanded layout): every (token, expert) selection carries its own copy of the
// token, written at its final row of the destination's per-expert receive buffer.
// per_token = 1: a token crosses NVLink once per destination RANK, however many of that rank's
// experts it selected (the non-expanded mode of the reference's dispatch,
// datasets/example081_deepep_jit_dispatch_copy_epilogue/nv/
// empty_deepep_jit_dispatch_copy_epilogue.cu:11,49-58: `kDoExpand`).  The copy goes to row
// rank * T + token of the destination's buffer - a position both sides can compute, so no
// second count exchange is needed - sent by the first of the token's selections that lives on
// that rank; every selection still writes its {source rank, pair} word at its final row, and the
// receive kernel expands from there.
//
// Bound by the bytes written.  At 4096 tokens, top-8 of 32 local experts, H = 7168 an expert-major
// grid (every selection loads and quantises its token again, 128 CTAs) took 417 us and the receive
// kernel's expansion 253 us; this kernel takes 115 us (528 MB, 4.6 TB/s) and the receive kernel only
// marks padding.
static constexpr int kSendCols = 1024;   // columns per warp and step: 4 x 16 bytes per lane
__global__ void __launch_bounds__(256)
    moe_dispatch_send_kernel(const __grid_constant__ MoeSendArgs a) {
  pdl_wait();                // chained with programmatic dependent launch: see prim/pdl.cuh
  pdl_launch_dependents();
  extern __shared__ int sent[];    // [E] rows this CTA has written per expert
  const int El = a.E / a.world;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = a.H / 128;
  const int slices = (a.H + kSendCols - 1) / kSendCols;
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) sent[e] = 0;
  __syncthreads();
  // Tokens of a CTA: so many at a time that their slices fill the 8 warps.
  const int batch = slices < 8 ? 8 / slices : 1;
  for (int t0 = blockIdx.x * batch; t0 < a.T; t0 += gridDim.x * batch) {
    const int n = min(batch, a.T - t0) * slices;
    for (int unit = warp; unit < n; unit += 8) {
      const int token = t0 + unit / slices, slice = unit % slices;
      // H is a multiple of 256: a 256-column group is whole or absent for all lanes.
      const uint4* __restrict__ src =
          reinterpret_cast<const uint4*>(a.x + static_cast<size_t>(token) * a.H + slice * kSendCols);
      const int ng = min(kSendCols, a.H - slice * kSendCols) / 256;
      uint4 raw[4];
#pragma unroll
      for (int g = 0; g < 4; ++g)
        raw[g] = g < ng ? __ldg(src + g * 32 + lane) : make_uint4(0, 0, 0, 0);
      uint2 q[4];
      float sc[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[g]);
        __nv_bfloat162 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])),
                                   __hmax2(__habs2(h[2]), __habs2(h[3])));
        // 16 lanes share one 128-channel group
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) m = __hmax2(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float2 mf = __bfloat1622float2(m);
        const float amax = fmaxf(fmaxf(0.f, mf.x), mf.y);
        sc[g] = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
        const float inv = 1.0f / sc[g];
        uint32_t w[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 v0 = __bfloat1622float2(h[2 * i]), v1 = __bfloat1622float2(h[2 * i + 1]);
          const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(
              make_float2(v0.x * inv, v0.y * inv), __NV_SATFINITE, __NV_E4M3);
          const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(
              make_float2(v1.x * inv, v1.y * inv), __NV_SATFINITE, __NV_E4M3);
          w[i] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
        }
        q[g] = make_uint2(w[0], w[1]);
        raw[g] = expand_fp8x8(q[g], sc[g]);   // what a row of this rank gets
      }
      unsigned ranks_sent = 0u;   // per_token: other ranks that have the token already
      for (int k0 = 0; k0 < a.K; k0 += 32) {
        // lane l holds selection k0 + l: expert, destination row, whether the payload goes there
        int e = -1, row = 0;
        if (k0 + lane < a.K) {
          const int pair = token * a.K + k0 + lane;
          e = a.topk_idx[pair];
          if (e >= a.E) e = -1;
          if (e >= 0) {
            row = a.send_row_base[e] + a.slot[pair];
            if (row >= a.max_rows) e = -1;   // the plan kernel already reported the overflow
          }
        }
        const int dst = e >= 0 ? e / El : -1;
        bool payload = e >= 0;
        if (a.per_token) {                   // an earlier selection on that rank sends the token
          const unsigned same = __match_any_sync(0xffffffffu, dst);
          if (dst >= 0 && dst != a.rank)
            payload = (same & ((1u << lane) - 1u)) == 0u && ((ranks_sent >> dst) & 1u) == 0u;
          ranks_sent |= __reduce_or_sync(0xffffffffu, dst >= 0 ? 1u << dst : 0u);
        }
        if (slice == 0 && e >= 0) {
          a.recv_meta[dst][row] = make_int2(a.rank, token * a.K + k0 + lane);
          atomicAdd(&sent[e], 1);
        }
        for (unsigned left = __ballot_sync(0xffffffffu, payload); left != 0u; left &= left - 1u) {
          const int l = __ffs(left) - 1;
          const int d = __shfl_sync(0xffffffffu, dst, l);
          const long long r = __shfl_sync(0xffffffffu, row, l);
          if (d == a.rank) {
            uint4* out = reinterpret_cast<uint4*>(a.a_out + r * a.H + slice * kSendCols);
#pragma unroll
            for (int g = 0; g < 4; ++g)
              if (g < ng) out[g * 32 + lane] = raw[g];
          } else {
            const long long dr = a.per_token ? static_cast<long long>(a.rank) * a.T + token : r;
            uint2* dq = reinterpret_cast<uint2*>(a.recv_x[d] + dr * a.H + slice * kSendCols);
            float* ds = a.recv_scale[d] + dr * groups + slice * (kSendCols / 128) + (lane >> 4);
#pragma unroll
            for (int g = 0; g < 4; ++g)
              if (g < ng) {
                dq[g * 32 + lane] = q[g];
                if ((lane & 15) == 0) ds[2 * g] = sc[g];
              }
          }
        }
      }
    }
  }
  // Every counter update is a release of its own: it covers what the whole CTA wrote before the
  // barrier, but only for the thread that makes it - a fence of another thread would not.
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x)
    if (sent[e] > 0)
      red_release_sys_add(a.arrived[e / El] + e % El, static_cast<uint32_t>(sent[e]));
}

struct MoeRecvArgs {
  const uint8_t* recv_x;      // fp8 [max_rows, H]
  const float* recv_scale;    // [max_rows, H/128]
  int2* recv_meta;            // [max_rows]
  __nv_bfloat16* a_out;       // bf16 [max_rows, H]  (grouped-GEMM input)
  uint32_t* arrived;          // [El]
  const int* recv_expected;   // [El]
  const int* recv_base;       // [El+1]
  int H, max_rows;
  unsigned long long timeout_ns;
  uint32_t* status;
  uint32_t* ctas_done;        // [El] zero-initialised words of this rank, or null (see the kernel)
  int per_token;              // 1: rows were sent once per token and rank; expand them here
  int T, K;                   // tokens per rank and selections per token (per_token only)
  int stage_rows;             // rows of recv_x / recv_scale (per_token only: world * T)
  int rank;                   // rows of this source rank are in a_out already (dispatch kernel)
};

// grid (El, slices).  Waits until the expert's rows are all in, then expands the rows that came
// from other ranks to bf16; this rank's own rows were written by its dispatch kernel.  Padding
// rows (up to the next multiple of 128) are marked with source rank -1 so later stages skip them;
// what they hold does not matter, since no row of a product depends on another row of A.
// With `ctas_done` set, the last CTA of an expert to finish clears that expert's arrival
// counter, so no separate fill launch is needed between two calls.  This is early enough: a peer
// cannot send rows of its NEXT call before it has this rank's combine rows of the current one,
// and those leave after this kernel in stream order.
__global__ void __launch_bounds__(256)
    moe_recv_dequant_kernel(const __grid_constant__ MoeRecvArgs a) {
  pdl_wait();                // chained with programmatic dependent launch: see prim/pdl.cuh
  const int j = blockIdx.x;
  const int expect = a.recv_expected[j];
  const int base = a.recv_base[j];
  const int padded = a.recv_base[j + 1] - base;
  bool ok = true;
  if (a.per_token) {
    // A row of this expert may have been sent on behalf of another expert of this rank (the
    // token's first selection here), so every counter of the rank has to be complete.  One
    // thread polls them one after the other (starting at its own): all must be complete
    // anyway, and few pollers leave the memory system to the rows still arriving.
    if (threadIdx.x == 0) {
      const int n = static_cast<int>(gridDim.x);
      for (int t = 0; t < n && ok; ++t) {
        const int i = (j + t) % n;
        const int ex = a.recv_expected[i];
        if (ex > 0)
          ok = wait_flag_ge_sys(a.arrived + i, static_cast<uint32_t>(ex), a.timeout_ns, a.status,
                                PH_MOE_ARRIVE2, i);
      }
    }
  } else if (threadIdx.x == 0 && expect > 0) {
    ok = wait_flag_ge_sys(a.arrived + j, static_cast<uint32_t>(expect), a.timeout_ns, a.status,
                          PH_MOE_ARRIVE2, j);
  }
  const bool all_ok = __syncthreads_and(ok ? 1 : 0) != 0;
  pdl_launch_dependents();   // not before: the product behind this kernel takes every SM's shared memory
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const int nvec = a.H / 8;
  const int groups = a.H / 128;
  // A warp's rows are `stride` apart; its lanes look at 32 of them at a time and the warp then
  // expands those that need it.
  const int stride = gridDim.y * warps;
  for (int r0 = blockIdx.y * warps + warp; all_ok && r0 < padded; r0 += 32 * stride) {
    const long long my = r0 + static_cast<long long>(lane) * stride;
    int2 m = make_int2(-1, -1);
    bool work = false;
    if (my < padded && base + my < a.max_rows) {
      if (my >= expect) {
        a.recv_meta[base + my] = m;
      } else {
        m = __ldcg(a.recv_meta + base + my);             // {source rank, source pair}
        work = m.x != a.rank;
      }
    }
    for (unsigned left = __ballot_sync(0xffffffffu, work); left != 0u; left &= left - 1u) {
      const int l = __ffs(left) - 1;
      const long long row = base + r0 + static_cast<long long>(l) * stride;
      uint4* __restrict__ out = reinterpret_cast<uint4*>(a.a_out + row * a.H);
      long long srow = row;
      if (a.per_token) {
        const int src = __shfl_sync(0xffffffffu, m.x, l), pair = __shfl_sync(0xffffffffu, m.y, l);
        srow = static_cast<long long>(src) * a.T + pair / a.K;
        if (src < 0 || pair < 0 || srow >= a.stage_rows) {   // never written: leave a zero row
          for (int v = lane; v < nvec; v += 32) out[v] = make_uint4(0, 0, 0, 0);
          continue;
        }
      }
      const uint2* __restrict__ q = reinterpret_cast<const uint2*>(a.recv_x + srow * a.H);
      const float* __restrict__ sc = a.recv_scale + srow * groups;
#pragma unroll 4
      for (int v = lane; v < nvec; v += 32) out[v] = expand_fp8x8(__ldcg(q + v), __ldcg(sc + v / 16));
    }
  }
  if (a.ctas_done != nullptr) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (a.per_token) {       // every CTA polls every counter: only the last CTA of the grid may clear
        if (atomicAdd(a.ctas_done, 1u) == gridDim.x * gridDim.y - 1) {
          for (unsigned i = 0; i < gridDim.x; ++i) a.arrived[i] = 0u;
          a.ctas_done[0] = 0u;
        }
      } else if (atomicAdd(a.ctas_done + j, 1u) == gridDim.y - 1) {
        a.arrived[j] = 0u;
        a.ctas_done[j] = 0u;
      }
    }
  }
}

// out[r, i] = silu(in[r, i]) * in[r, I + i]; rows taken from n_rows_dev (device word).
__global__ void swiglu_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                              const int* n_rows_dev, int I) {
  const long long rows = *n_rows_dev;
  const long long vec_per_row = I / 8;
  const long long total = rows * vec_per_row;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = idx / vec_per_row, c = idx % vec_per_row;
    const uint4 g = *reinterpret_cast<const uint4*>(in + r * 2 * I + c * 8);
    const uint4 u = *reinterpret_cast<const uint4*>(in + r * 2 * I + I + c * 8);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
    const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&u);
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = __bfloat1622float2(gh[i]);
      const float2 b = __bfloat1622float2(uh[i]);
      oh[i] = __floats2bfloat162_rn(a.x / (1.f + __expf(-a.x)) * b.x,
                                    a.y / (1.f + __expf(-a.y)) * b.y);
    }
    *reinterpret_cast<uint4*>(out + r * I + c * 8) = o;
  }
}

// y[t, :] = sum_k w[t,k] * buf[t, k, :] (+ bias0[t, :] + bias1[t, :])   after every expert rank
// has reported in.  The two optional bias inputs [T, H] bf16 are those of the reference's
// reduction epilogue (datasets/example083_deepep_jit_combine_reduce_epilogue/nv/
// empty_deepep_jit_combine_reduce_epilogue.cu:28): a shared-expert output or a residual can be
// added here instead of in another pass over y.
// `done` = W words on this rank (one per expert rank); cleared by the last CTA.
__global__ void __launch_bounds__(256)
    moe_combine_reduce_kernel(const __nv_bfloat16* __restrict__ buf, const float* __restrict__ w,
                              const int* __restrict__ topk_idx, __nv_bfloat16* __restrict__ y,
                              int T, int K, int H, uint32_t* done, int world,
                              unsigned long long timeout_ns, uint32_t* status,
                              uint32_t* done_ctas, const __nv_bfloat16* __restrict__ bias0,
                              const __nv_bfloat16* __restrict__ bias1) {
  pdl_wait();                // chained with programmatic dependent launch: see prim/pdl.cuh
  bool ok = true;
  if (threadIdx.x < static_cast<unsigned>(world))
    ok = wait_flag_ge_sys(done + threadIdx.x, 1u, timeout_ns, status, PH_MOE_COMBINE2,
                          threadIdx.x);
  const bool all_ok = __syncthreads_and(ok ? 1 : 0) != 0;
  pdl_launch_dependents();   // not before: what follows may take every SM's shared memory
  if (all_ok) {
    // A warp takes 32 vectors of one token; eight of the token's K rows are loaded before the
    // first is added (a masked selection's row is loaded too and left out of the sum), so the
    // kernel is bound by bandwidth instead of by K dependent loads.  Measured at 4096 tokens, K = 8,
    // H = 7168 (529 MB): 142 us, now 107 us (4.9 TB/s).
    const int nvec = H / 8;
    const unsigned per_token = (nvec + 31) / 32;
    const unsigned units = static_cast<unsigned>(T) * per_token;
    const unsigned lane = threadIdx.x & 31u;
    for (unsigned unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < units;
         unit += gridDim.x * blockDim.x >> 5) {
      const long long t = unit / per_token;
      const int v = static_cast<int>((unit % per_token) * 32 + lane);
      if (v >= nvec) continue;
      float acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.f;
      for (int b = 0; b < 2; ++b) {
        const __nv_bfloat16* bias = b == 0 ? bias0 : bias1;
        if (bias == nullptr) continue;
        const uint4 raw = *(reinterpret_cast<const uint4*>(bias + t * H) + v);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(h[i]);
          acc[2 * i] += f.x;
          acc[2 * i + 1] += f.y;
        }
      }
      for (int k0 = 0; k0 < K; k0 += 8) {
        uint4 raw[8];
        float wk[8];
        bool use[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          use[k] = k0 + k < K;
          if (use[k]) {
            const long long pair = t * K + k0 + k;
            raw[k] = __ldcg(reinterpret_cast<const uint4*>(buf + pair * H) + v);
            wk[k] = w[pair];
            use[k] = topk_idx[pair] >= 0;
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (!use[k]) continue;
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[k]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            acc[2 * i] += wk[k] * f.x;
            acc[2 * i + 1] += wk[k] * f.y;
          }
        }
      }
      uint4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      reinterpret_cast<uint4*>(y + t * H)[v] = o;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(done_ctas, 1u) == gridDim.x - 1) {
      for (int r = 0; r < world; ++r) done[r] = 0u;
      *done_ctas = 0u;
    }
  }
}

}  // namespace cb

using namespace cb;

extern "C" {

int cb_sizeof_moe_send_args() { return static_cast<int>(sizeof(MoeSendArgs)); }
int cb_sizeof_moe_recv_args() { return static_cast<int>(sizeof(MoeRecvArgs)); }

int cb_moe_dispatch_send(const MoeSendArgs* a, int max_ctas, void* stream) {
  if (a->H % 256 != 0 || a->E % a->world != 0 || a->E > 1024 || a->T < 1 || a->K < 1) {
    set_last_error("dispatch: hidden must be a multiple of 256, experts (at most 1024) divisible "
                   "by ranks, at least one token and selection");
    return -1;
  }
  const int slices = (a->H + kSendCols - 1) / kSendCols;
  const int batch = slices < 8 ? 8 / slices : 1;
  int ctas = (a->T + batch - 1) / batch;
  if (max_ctas > 0 && ctas > max_ctas) ctas = max_ctas;
  if (ctas < 1) ctas = 1;
  return launch_pdl(moe_dispatch_send_kernel, dim3(ctas), dim3(256), a->E * sizeof(int),
                    static_cast<cudaStream_t>(stream), *a) == cudaSuccess
             ? 0
             : -1;
}

int cb_moe_recv_dequant(const MoeRecvArgs* a, int n_local_experts, int slices, void* stream) {
  if (a->per_token && (a->T < 1 || a->K < 1 || a->stage_rows < 1)) {
    set_last_error("receive: the per-token form needs T, K and stage_rows");
    return -1;
  }
  dim3 grid(n_local_experts, slices < 1 ? 1 : slices);
  return launch_pdl(moe_recv_dequant_kernel, grid, dim3(256), 0,
                    static_cast<cudaStream_t>(stream), *a) == cudaSuccess
             ? 0
             : -1;
}

int cb_moe_swiglu(const void* in, void* out, const void* n_rows_dev, int I, void* stream) {
  if (I % 8 != 0) return -1;
  swiglu_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out),
      static_cast<const int*>(n_rows_dev), I);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// bias0 / bias1: optional [T, H] bf16 tensors added to the weighted sum (may be null).
int cb_moe_combine_reduce_bias(const void* buf, const void* w, const void* topk_idx, void* y,
                               int T, int K, int H, void* done, int world,
                               unsigned long long timeout_ns, void* status, void* done_ctas,
                               const void* bias0, const void* bias1, void* stream) {
  if (H % 8 != 0) return -1;
  return launch_pdl(moe_combine_reduce_kernel, dim3(592), dim3(256), 0,
                    static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(buf),
                    static_cast<const float*>(w), static_cast<const int*>(topk_idx),
                    static_cast<__nv_bfloat16*>(y), T, K, H, static_cast<uint32_t*>(done), world,
                    timeout_ns, static_cast<uint32_t*>(status), static_cast<uint32_t*>(done_ctas),
                    static_cast<const __nv_bfloat16*>(bias0),
                    static_cast<const __nv_bfloat16*>(bias1)) == cudaSuccess
             ? 0
             : -1;
}

int cb_moe_combine_reduce(const void* buf, const void* w, const void* topk_idx, void* y, int T,
                          int K, int H, void* done, int world, unsigned long long timeout_ns,
                          void* status, void* done_ctas, void* stream) {
  return cb_moe_combine_reduce_bias(buf, w, topk_idx, y, T, K, H, done, world, timeout_ns, status,
                                    done_ctas, nullptr, nullptr, stream);
}

}  // extern "C"
