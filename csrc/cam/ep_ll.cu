// Low-latency (decode) expert-parallel dispatch: per-expert counts are all-gathered through peer memory, then every
// (token, k) is quantised to fp8 e4m3 (fp32 scale per 1x128 block) and stored straight into its final row of the
// destination rank's expert-major slab, which the grouped GEMM reads with TMA without any repacking.
//
// The reference's decode path pushes int8 tokens into fixed [srcRank][localExpert] window slots and compacts them
// on the receiver before the GEMM (src/cam/comm_operator/ascend_kernels/fused_deep_moe/op_kernel/fused_deep_moe/
// raw_distributed/cam_moe_distribute_dispatch.h:433-488 SendToMoeExpert, :781-861 LocalWindowCopy). Here the counts
// travel first (one small NVLink round), so senders know the exact destination rows and the compaction pass
// disappears; rows of one expert are ordered by source rank, then by (token, k) - the same order as the reference's
// compacted expandX (status index = localExpert * R + srcRank, :625-633).
#include "ep_ll_dispatch.cuh"
#include "ep_params.h"

namespace umdk {
namespace {

constexpr int kLLThreads = 512;
constexpr int kLLWarps = kLLThreads / 32;

struct LLDispatchArgs {
  EpLLGeom g;
  EpLLOffsets off;
  PeerTable peers;
  LLDispatchIO io;
};

__global__ void __launch_bounds__(kLLThreads, 1) ep_ll_dispatch_kernel(const LLDispatchArgs a) {
  extern __shared__ __align__(16) uint8_t ll_scratch[];
  ll_dispatch_body<kLLThreads, 32>(a.g, a.off, a.peers, a.io, ll_scratch, nullptr);
}

// Low-latency combine as an operator of its own (the counterpart of the fused kernel's tail for callers that ran
// their own expert computation between low_latency_dispatch and low_latency_combine): every bf16 row of the slab goes
// back to its token's owner over NVLink into the owner's combine buffer (the slot comes from the row metadata the
// dispatch left beside the slab), completion flags go to every peer, and after all peers' flags have arrived the owner
// sums its rows with the routing weights. No host synchronisation: the row count is read from group_off on the
// device. Reference: cam_moe_distribute_combine.h:238-320 (status set / wait), :627-717 (weighted sum).
struct LLCombineArgs {
  EpLLGeom g;
  EpLLOffsets off;
  PeerTable peers;
  const __nv_bfloat16* y;     // [>= n, H] expert outputs in slab row order
  const int* group_off;       // [E_local + 1]; n = group_off[E_local]
  const int64_t* topk_idx;    // [T, K]
  const float* topk_w;        // [T, K]
  __nv_bfloat16* out;         // [T, H]
  int T;
  uint32_t* ctrl;             // [0] epoch (advanced here), [1] send-done, [2] reduce-done
  int* status;
  int phase_mask;             // bit0: send rows + flags; bit1: wait flags + weighted sum + epoch advance
};

__global__ void __launch_bounds__(kLLThreads, 1) ep_ll_combine_kernel(const LLCombineArgs a) {
  const EpLLGeom& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ uint32_t s_epoch;
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    s_epoch = a.ctrl[0];
    s_ok = 1;
  }
  __syncthreads();
  const uint32_t epoch = s_epoch;
  const uint64_t tag = (uint64_t)epoch + 1;
  uint8_t* self = a.peers.base[g.rank];
  if (a.phase_mask & 1) {
    const int n = min(a.group_off[g.E_local], g.n_cap);
    const int* meta = reinterpret_cast<const int*>(self + a.off.slab_meta[0]);
    // one work item = 4 KiB of one row (32 lanes x 8 x 16 bytes): all loads of an item are in flight together
    const int nvec = g.H / 8;
    const int nparts = (nvec + 255) / 256;
    for (int item = blockIdx.x * kLLWarps + warp; item < n * nparts; item += gridDim.x * kLLWarps) {
      const int row = item / nparts, part = item - row * nparts;
      const int owner = meta[2 * row], slot = meta[2 * row + 1];
      if (owner < 0 || owner >= g.R || slot < 0 || slot >= g.T_cap * g.K) {
        if (lane == 0) umdk_set_status(a.status, UMDK_ERR_OVERFLOW, UMDK_PH_COMBINE_DATA, owner, slot);
        continue;
      }
      const int4* src = reinterpret_cast<const int4*>(a.y + (size_t)row * g.H);
      uint8_t* dst = a.peers.base[owner] + a.off.comb_buf[0] + (size_t)slot * g.H * 2;
      int4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = part * 256 + u * 32 + lane;
        v[u] = i < nvec ? __ldg(src + i) : make_int4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = part * 256 + u * 32 + lane;
        if (i < nvec) st_na_v4(dst + (size_t)i * 16, v[u]);
      }
    }
    if (cta_done_is_last(&a.ctrl[1], gridDim.x)) {
      // the call ends here for this rank's slab: its arrival words go back to zero before the flags that let the
      // peers start their next dispatch
      uint32_t* exp_cnt = reinterpret_cast<uint32_t*>(self + a.off.exp_cnt[0]);
      for (int i = threadIdx.x; i < g.E_local; i += blockDim.x) exp_cnt[i] = 0;
      __threadfence_system();
      __syncthreads();
      if (threadIdx.x < g.R) {
        st_release_sys(reinterpret_cast<uint64_t*>(a.peers.base[threadIdx.x] + a.off.comb_flag[0]) + g.rank, tag);
      }
    }
  }
  if (!(a.phase_mask & 2)) return;
  if (threadIdx.x < g.R) {
    const uint64_t* f = reinterpret_cast<const uint64_t*>(self + a.off.comb_flag[0]) + threadIdx.x;
    if (!wait_flag_ge_sys(f, tag)) {
      umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_COMBINE_DATA, threadIdx.x, (int)epoch);
      s_ok = 0;
    }
  }
  __syncthreads();
  if (s_ok) {
    ll_weighted_reduce<kLLThreads>(self + a.off.comb_buf[0], a.topk_idx, a.topk_w, a.out, nullptr, a.T, g.K, g.H);
  }
  if (cta_done_is_last(&a.ctrl[2], gridDim.x)) {
    if (threadIdx.x == 0) a.ctrl[0] = epoch + 1;
  }
}

// The same for a group of ONE rank: every row already lies in this GPU's memory, so the weighted sum reads it where it is.
// Each CTA inverts the row metadata (row -> slot) into a slot -> row table in shared memory (a few KB), which replaces
// the pass through the combine buffer, the completion flags and the grid-wide wait on them. Bound by latency: one table,
// one round of row loads. Measured: 1024 rows of 7168 to 128 tokens 34.8 -> 12.9 us; with the metadata fetched beside the row
// count and the call ended by the first CTA instead of the last 9.5 -> 7.7 (calls back to back in a graph), 1 token 5.8 -> 4.4.
// With the next item's rows, weights and indices fetched while one is summed, and no row waiting for its index (inputs in turn, the
// kernel alone) 13.5 -> 9.9, 2048 rows to 256 tokens 23.1 -> 16.7. kSlots: rows of a pass; with eight for every top-k the instructions for
// rows that are not there cost more than the rest (142 tokens, top-1, 5.0; 6.6 with eight, 4.1 with two).
constexpr int kLLLocalSlots = 11264;   // [T * K] ints in 44 KB of shared memory
template <int kSlots>
__global__ void __launch_bounds__(kLLThreads, 1) ep_ll_combine_local_kernel(const LLCombineArgs a) {
  extern __shared__ int s_rowof[];
  const EpLLGeom& g = a.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* self = a.peers.base[g.rank];
  // the metadata of rows that may not be there are read too (they are memory of the heap): one round trip with the row count
  const int2* meta = reinterpret_cast<const int2*>(self + a.off.slab_meta[0]);
  const int first = threadIdx.x < g.n_cap ? threadIdx.x : 0;
  const int second = threadIdx.x + kLLThreads < g.n_cap ? threadIdx.x + kLLThreads : 0;
  const int2 m0 = __ldg(meta + first), m1 = __ldg(meta + second);
  const int n = min(a.group_off[g.E_local], g.n_cap);
  const int slots = a.T * g.K;
  for (int i = threadIdx.x; i < slots; i += kLLThreads) s_rowof[i] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kLLThreads) {
    const int2 m = i < kLLThreads ? m0 : i < 2 * kLLThreads ? m1 : __ldg(meta + i);
    if (m.x != g.rank || m.y < 0 || m.y >= g.T_cap * g.K) {
      umdk_set_status(a.status, UMDK_ERR_OVERFLOW, UMDK_PH_COMBINE_DATA, m.x, m.y);
    } else if (m.y < slots) {
      s_rowof[m.y] = i;
    }
  }
  __syncthreads();
  const int nvec = g.H / 8;
  const int nchunk = (nvec + 31) / 32;
  // Rows, weights and indices of the next item are on their way while this one is summed: rounds of items overlap.
  struct Rows {
    int4 vals[kSlots];
    float wk[kSlots];
  };
  auto fetch = [&](int item, int k0, Rows* r) {
    const int t = item / nchunk, v = (item - t * nchunk) * 32 + lane;
    long long idx[kSlots];
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      const int k = k0 + u;
      const int row = k < g.K && v < nvec ? s_rowof[t * g.K + k] : -1;
      idx[u] = row >= 0 ? a.topk_idx[(size_t)t * g.K + k] : -1;
      r->wk[u] = row >= 0 ? a.topk_w[(size_t)t * g.K + k] : 0.f;
      r->vals[u] = row >= 0 ? ld_nc_v4(reinterpret_cast<const int4*>(a.y + (size_t)row * g.H) + v) : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      if (idx[u] < 0) {
        r->wk[u] = 0.f;
        r->vals[u] = make_int4(0, 0, 0, 0);
      }
    }
  };
  auto add = [&](const Rows& r, float* acc) {
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      float f[8];
      bf16x8_to_float(r.vals[u], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(r.wk[u], f[i], acc[i]);
    }
  };
  Rows cur, next;
  const int stride = gridDim.x * kLLWarps;
  int item = blockIdx.x * kLLWarps + warp;
  if (item < a.T * nchunk) fetch(item, 0, &cur);
  for (; item < a.T * nchunk; item += stride) {
    const int t = item / nchunk, v = (item - t * nchunk) * 32 + lane;
    if (item + stride < a.T * nchunk) fetch(item + stride, 0, &next);
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    add(cur, acc);
    for (int k0 = kSlots; k0 < g.K; k0 += kSlots) {
      fetch(item, k0, &cur);
      add(cur, acc);
    }
    if (v < nvec) {
      int4 o;
      __nv_bfloat162* po = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) po[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      reinterpret_cast<int4*>(a.out + (size_t)t * g.H)[v] = o;
    }
    cur = next;
  }
  if (blockIdx.x == 0) {   // the call ends: arrival words back to zero, next epoch (nobody else reads either during this kernel)
    uint32_t* exp_cnt = reinterpret_cast<uint32_t*>(self + a.off.exp_cnt[0]);
    for (int i = threadIdx.x; i < g.E_local; i += blockDim.x) exp_cnt[i] = 0;
    if (threadIdx.x == 0) a.ctrl[0] += 1;
  }
}

// Stand-alone fp8 e4m3 1x128 quantisation of local rows (shared expert input, tests).
__global__ void __launch_bounds__(256) quant_fp8_kernel(const __nv_bfloat16* __restrict__ x, int T, int H,
                                                        uint8_t* __restrict__ q, float* __restrict__ s) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = H / 128;
  for (int t = blockIdx.x * 8 + warp; t < T; t += gridDim.x * 8) {
    const int4* xrow = reinterpret_cast<const int4*>(x + (size_t)t * H);
    for (int b0 = 0; b0 < nblk; b0 += 4) {
      const int blk = b0 + (lane >> 3);
      const bool active = blk < nblk;
      float f[16];
      if (active) {
        bf16x8_to_float(__ldg(xrow + blk * 16 + (lane & 7) * 2), f);
        bf16x8_to_float(__ldg(xrow + blk * 16 + (lane & 7) * 2 + 1), f + 8);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = 0.f;
      }
      float scale;
      const int4 v = quant16(f, &scale);
      if (active) {
        *reinterpret_cast<int4*>(q + (size_t)t * H + blk * 128 + (lane & 7) * 16) = v;
        if ((lane & 7) == 0) s[(size_t)t * nblk + blk] = scale;
      }
    }
  }
}

}  // namespace
}  // namespace umdk

using namespace umdk;


struct UmdkEpLLLayout {
  uint64_t cnt, cnt_flag, data_flag, comb_flag, slab_x, slab_s, slab_meta, comb_buf, total;
  int n_cap;
  uint64_t exp_cnt;   // arrival words per local expert
};

// Offsets of the low-latency regions inside each rank's symmetric heap, and the heap size needed.
UMDK_API int umdk_ep_ll_layout(int R, int E, int K, int H, int T_cap, UmdkEpLLLayout* out) {
  EpLLGeom g;
  if (int rc = fill_ll_geom(&g, R, 0, E, K, H, T_cap)) return rc;
  const EpLLOffsets o = ep_ll_offsets(g);
  out->cnt = o.cnt[0];
  out->cnt_flag = o.cnt_flag[0];
  out->data_flag = o.data_flag[0];
  out->comb_flag = o.comb_flag[0];
  out->slab_x = o.slab_x[0];
  out->slab_s = o.slab_s[0];
  out->slab_meta = o.slab_meta[0];
  out->comb_buf = o.comb_buf[0];
  out->exp_cnt = o.exp_cnt[0];
  out->total = o.total;
  out->n_cap = g.n_cap;
  return 0;
}

// CTAs of a dispatch on a GPU with `sms` SMs. num_ctas 0, one rank: an item (2 KiB of a token) for every warp, 32 CTAs at least.
// 32 / as many as that, us, with the combine: 142 tokens of 6656, top-1 of 160 16.3 / 13.0, 256 of 7168, top-8 of 256
// 40.4 / 34.5; no difference where 32 hold all items. With more ranks always 32: every CTA waits for the peers' counts, and
// while they are late the other SMs belong to whatever runs beside it (a GEMM, another micro-batch's dispatch, for which a
// peer may be waiting).
UMDK_API int umdk_ep_ll_dispatch_grid(int R, int T, int H, int num_ctas, int sms) {
  const int items = T * ((H / 128 + 15) / 16);
  int grid = 32;
  if (num_ctas > 0) grid = num_ctas;
  else if (R == 1 && items > 32 * kLLWarps) grid = (items + kLLWarps - 1) / kLLWarps;
  return grid < sms ? grid : sms;
}

static_assert(kUmdkMaxRanks == kMaxRanks, "parameter blocks");

UMDK_API int umdk_ep_ll_dispatch(const UmdkEpLLDispatchParams* p, void* stream) {
  LLDispatchArgs a;
  if (int rc = fill_ll_geom(&a.g, p->R, p->rank, p->E, p->K, p->H, p->T_cap)) return rc;
  if (p->T > p->T_cap) return -UMDK_ERR_BAD_ARG;
  a.off = ep_ll_offsets(a.g);
  for (int i = 0; i < kMaxRanks; ++i) a.peers.base[i] = i < p->R ? static_cast<uint8_t*>(p->peers[i]) : nullptr;
  a.io.x = static_cast<const __nv_bfloat16*>(p->x);
  a.io.topk_idx = p->topk_idx;
  a.io.send_idx = p->send_idx;
  a.io.num_per_expert = p->num_per_expert;
  a.io.T = p->T;
  a.io.group_off = p->group_off;
  a.io.recv_per_expert = p->recv_per_expert;
  a.io.ctrl = p->ctrl;
  a.io.status = p->status;
  a.io.meet_cycles = umdk_rendezvous_cycles();
  a.io.phase_mask = p->phase_mask ? p->phase_mask : 3;
  const int grid = umdk_ep_ll_dispatch_grid(p->R, p->T, p->H, p->num_ctas, sm_count());
  if (!p->send_idx) {
    // layout inside the kernel: 16-bit counters and positions, so at most 65535 entries per expert and a table that
    // fits in shared memory
    if (p->num_per_expert || p->T > 2048 || p->E > 1024) return -UMDK_ERR_BAD_ARG;
  } else if (!p->num_per_expert) {
    return -UMDK_ERR_BAD_ARG;
  }
  const size_t dyn = ll_dispatch_smem_bytes(p->T, p->E, p->K, kLLWarps, p->send_idx == nullptr);
  if (dyn > 200 * 1024) return -UMDK_ERR_BAD_ARG;
  if (dyn > 40 * 1024) {
    UMDK_CUDA_CHECK(cudaFuncSetAttribute(ep_ll_dispatch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  }
  ep_ll_dispatch_kernel<<<grid, kLLThreads, dyn, static_cast<cudaStream_t>(stream)>>>(a);
  UMDK_CUDA_CHECK(cudaGetLastError());
  return 0;
}

UMDK_API int umdk_ep_ll_combine(const UmdkEpLLCombineParams* p, void* stream) {
  LLCombineArgs a;
  if (int rc = fill_ll_geom(&a.g, p->R, p->rank, p->E, p->K, p->H, p->T_cap)) return rc;
  if (p->T > p->T_cap || p->T < 0) return -UMDK_ERR_BAD_ARG;
  a.off = ep_ll_offsets(a.g);
  for (int i = 0; i < kMaxRanks; ++i) a.peers.base[i] = i < p->R ? static_cast<uint8_t*>(p->peers[i]) : nullptr;
  a.y = static_cast<const __nv_bfloat16*>(p->y);
  a.group_off = p->group_off;
  a.topk_idx = p->topk_idx;
  a.topk_w = p->topk_w;
  a.out = static_cast<__nv_bfloat16*>(p->out);
  a.T = p->T;
  a.ctrl = p->ctrl;
  a.status = p->status;
  a.phase_mask = p->phase_mask ? p->phase_mask : 3;
  if (p->R == 1 && a.phase_mask == 3 && p->T * p->K <= kLLLocalSlots) {
    const int items = p->T * ((p->H / 8 + 31) / 32);   // one warp each
    int grid = p->num_ctas > 0 ? p->num_ctas : (items + kLLWarps - 1) / kLLWarps;
    if (grid > sm_count()) grid = sm_count();
    if (grid < 1) grid = 1;
    const auto combine = p->K <= 2   ? ep_ll_combine_local_kernel<2>
                         : p->K <= 4 ? ep_ll_combine_local_kernel<4>
                                     : ep_ll_combine_local_kernel<8>;
    combine<<<grid, kLLThreads, sizeof(int) * p->T * p->K, static_cast<cudaStream_t>(stream)>>>(a);
    UMDK_CUDA_CHECK(cudaGetLastError());
    return 0;
  }
  int grid = p->num_ctas > 0 ? p->num_ctas : 64;
  if (grid > sm_count()) grid = sm_count();
  ep_ll_combine_kernel<<<grid, kLLThreads, 0, static_cast<cudaStream_t>(stream)>>>(a);
  UMDK_CUDA_CHECK(cudaGetLastError());
  return 0;
}

UMDK_API int umdk_quant_fp8_1x128(const void* x, int T, int H, void* q, float* s, void* stream) {
  if (T < 0 || H < 128 || (H % 128)) return -UMDK_ERR_BAD_ARG;
  if (T == 0) return 0;
  int grid = (T + 7) / 8;
  if (grid > 4 * sm_count()) grid = 4 * sm_count();
  quant_fp8_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(x), T, H,
                                                                      static_cast<uint8_t*>(q), s);
  UMDK_CUDA_CHECK(cudaGetLastError());
  return 0;
}
