// Tensor-parallel fused GEMM + collective kernels with CTA pairs (one `tcgen05.mma.cta_group::2` per 256 x 256 output
// tile; 128 or 64 columns where that ends sooner, see tile_columns). Same protocol, heap layout and arguments as tp_gemm.cu
// - copy CTAs that gather peer shards for MODE 0, push epilogue + owner reduce for MODE 1 - with the main loop of
// gemm_bf16_2sm.cu: each CTA of a pair stages 128 rows of A and half the rows of B per k-block and keeps its half of the
// accumulator in its own TMEM.
//
// The own shard never passes through the heap on its way to the tensor cores: MODE 0 reads it from the caller's tensor at once
// (the copy CTAs still publish it to the peers), and a group of one rank gives all 74 pairs to the GEMM. MODE 1 with one
// rank stores the product where it belongs instead of pushing it into the receive buffer and summing one addend. Bound by
// the tensor cores from there on. Measured with one rank, 8192 x 8192 times 7168 and 8192 x 3584 times 8192: 1510 -> 974 us
// of kernel time for the two (1.48 PFLOP/s in a burst), 1627 -> 1145 us back to back under the power limit.
// An odd number of 128-row blocks leaves the last tile's second CTA without rows (it repeats the leader's and stores nothing):
// 8064 x 6656 times 4096 and 8064 x 1536 times 6656 took 1720 us on single CTAs through the heap and take 438 here (8 passes behind a
// pause; 400 back to back 1685 and 460).
#include "tp_common.cuh"

#include <cuda_runtime.h>

namespace umdk {
namespace {

constexpr int BMH = 128;
constexpr int BK = 64;
constexpr int kThreads = kTpThreads;
constexpr int kABytes = BMH * BK * 2;
constexpr int kEpiBufBytes = 32 * 64 * 2;
constexpr int kEpiBytes = 4 * 2 * kEpiBufBytes;

template <int BN>   // columns of a pair's tile: 64, 128 or 256
struct Cfg {
  static constexpr int kBNH = BN / 2;
  static constexpr int kBBytes = kBNH * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BN == 256 ? 6 : 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + 256 + 1024;
  static constexpr int kTmemCols = 2 * BN;
};

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
tp_gemm_2sm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmOwn,
                   const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC, const TpArgs a) {
  using C = Cfg<BN>;
  constexpr int kStages = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + kStages * C::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + kEpiBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kStages;
  uint64_t* tfull = bars + 2 * kStages;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  __shared__ uint32_t s_epoch;
  __shared__ int s_ok;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_epoch = a.ctrl[0];
    s_ok = 1;
  }
  __syncthreads();
  const uint32_t epoch = s_epoch;
  const int slot = epoch & 1;
  const uint64_t tag = (uint64_t)epoch + 1;
  // the last row block of a shard has rows for the leader only where Ts is an odd multiple of 128
  const int mb_per_chunk = (a.Ts + 2 * BMH - 1) / (2 * BMH);
  const int nb = a.N / BN;
  const int kb_total = a.K / BK;
  const int num_tiles = a.R * mb_per_chunk * nb;
  // even: whole pairs take the copy role. A group of one rank has nothing to copy, every pair computes.
  const int n_copy = a.mode == 0 && a.R > 1 ? a.n_copy : 0;
  // MODE 1 with one rank: the product is the result, so it is stored as such (no receive buffer, no second pass over it)
  const bool local_rs = a.mode == 1 && a.R == 1 && (a.phase_mask & 3) == 3;
  // arrivals per call and source: row blocks of 128 x tiles of 256 columns (the launcher takes no others where ranks exchange)
  // x 4 epilogue warps
  const uint32_t per_src = (uint32_t)(a.Ts / BMH) * (uint32_t)(a.N / 256) * 4u;
  const bool is_copy_cta = (int)blockIdx.x < n_copy;

  if (a.mode == 0 && is_copy_cta) {
    // dedicated copy CTAs (whole pairs): the GEMM ring and barrier area serve as the bulk-copy ring
    tp_copy_role_bulk(a, n_copy, slot, tag, epoch, &s_ok, smem, bars);
  } else {
    const uint32_t cta = cluster_ctarank();
    const int pair = ((int)blockIdx.x - n_copy) >> 1;
    const int num_pairs = ((int)gridDim.x - n_copy) >> 1;
    if (threadIdx.x == 0) {
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tfull[i], 1);
        mbar_init(&tempty[i], 8);   // leader's copy: four epilogue warps of each CTA
      }
      mbar_fence_init();
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      tma_prefetch_desc(&tmC);
    }
    if (warp == 2) {
      tmem_alloc_pair(tmem_slot, C::kTmemCols);
      tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int my_tiles_end = (a.mode == 1 && !(a.phase_mask & 1)) ? 0 : num_tiles;
    // tile t -> chunk i = t / tiles_per_chunk (source / owner rank (rank + shift + i) % R; MODE 0 starts with the own
    // shard, MODE 1 ends with the own rows), 256-row block and 256-column block inside the chunk
    const int tiles_per_chunk = mb_per_chunk * nb;
    // inside a chunk, groups of kGroupM row blocks are swept column by column: the ~74 tiles in flight then share
    // 8 A panels and ~9 B panels, which stay in L2
    constexpr int kGroupM = 8;
    auto tile_coords = [&](int t, int* m0, int* n0, int* peer, bool* rows) {
      const int i = t / tiles_per_chunk, r = t - i * tiles_per_chunk;
      const int p = (a.rank + (a.mode == 0 ? 0 : 1) + i) % a.R;
      const int per_group = kGroupM * nb;
      const int g = r / per_group, rg = r - g * per_group;
      const int gm = min(kGroupM, mb_per_chunk - g * kGroupM);
      const int mblk = g * kGroupM + rg % gm, nblk = rg / gm;
      *peer = p;
      *rows = mblk * 2 * BMH + (int)cta * BMH < a.Ts;   // whether this CTA has rows in this tile
      *m0 = p * a.Ts + mblk * 2 * BMH + (*rows ? (int)cta * BMH : 0);   // its 128 rows (else the leader's, to have some)
      *n0 = nblk * BN;
    };

    if (warp == 0) {
      if (elect_one()) {
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        int have_chunk = -1;
        const uint32_t full0 = map_to_cta(&full[0], 0);
        for (int t = pair; t < my_tiles_end && ok; t += num_pairs) {
          int m0, n0, peer;
          bool rows;
          tile_coords(t, &m0, &n0, &peer, &rows);
          // MODE 0: the own shard is read from the caller's tensor, at once and without passing through the heap
          const bool own = a.mode == 0 && peer == a.rank;
          if (a.mode == 0 && !own && peer != have_chunk) {
            if (!wait_flag_ge_gpu(&a.chunk_done[peer], (uint32_t)tag * (uint32_t)n_copy)) {
              umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_AG_CHUNK, peer, t);
              break;
            }
            have_chunk = peer;
            fence_proxy_async_all();
          }
          for (int kb = 0; kb < kb_total; ++kb) {
            if (!mbar_wait(&empty[s], ph ^ 1)) {
              umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_TMA_EMPTY, t, kb);
              ok = false;
              break;
            }
            if (cta == 0) mbar_expect_tx(&full[s], 2 * C::kStageBytes);
            const uint32_t leader_full = full0 + s * 8;
            uint8_t* sa = smem + s * C::kStageBytes;
            tma_load_2d_pair(sa, own ? &tmOwn : &tmA, leader_full, kb * BK, own ? m0 - peer * a.Ts : m0);
            tma_load_2d_pair(sa + kABytes, &tmB, leader_full, kb * BK, n0 + (int)cta * C::kBNH);
            if (++s == kStages) {
              s = 0;
              ph ^= 1;
            }
          }
        }
      }
    } else if (warp == 1 && cta == 0) {
      if (elect_one()) {
        constexpr uint32_t idesc = umma_idesc(kFmtBF16, kFmtBF16, 2 * BMH, BN);
        const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem));
        int s = 0;
        uint32_t ph = 0;
        int it = 0;
        bool ok = true;
        for (int t = pair; t < my_tiles_end && ok; t += num_pairs, ++it) {
          const int ab = it & 1;
          const uint32_t aph = (it >> 1) & 1;
          if (!mbar_wait(&tempty[ab], aph ^ 1)) {
            umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_TMEM_EMPTY, t, 0);
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + ab * BN;
          for (int kb = 0; kb < kb_total; ++kb) {
            if (!mbar_wait(&full[s], ph)) {
              umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_TMA_FULL, t, kb);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t adesc = desc0 + s * (C::kStageBytes >> 4);
            const uint64_t bdesc = adesc + (kABytes >> 4);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_f16_pair(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) ? 1u : 0u);
            umma_commit_both(smem_u32(&empty[s]));
            if (++s == kStages) {
              s = 0;
              ph ^= 1;
            }
          }
          if (ok) umma_commit_both(smem_u32(&tfull[ab]));
        }
      }
    } else if (warp >= 4) {
      const int ew = warp - 4;
      uint8_t* my_epi = epi + ew * 2 * kEpiBufBytes;
      int it = 0, buf = 0;
      for (int t = pair; t < my_tiles_end; t += num_pairs, ++it) {
        int m0, n0, peer;
        bool rows;
        tile_coords(t, &m0, &n0, &peer, &rows);
        const int ab = it & 1;
        const uint32_t aph = (it >> 1) & 1;
        if (!mbar_wait_warp(&tfull[ab], aph)) {
          umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_TMEM_FULL, t, 0);
          break;
        }
        tc_fence_after();
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + ab * BN;
        if (!rows) {
          // the product of the leader's rows once more: nobody wants it
        } else if (a.mode == 0 || local_rs) {
#pragma unroll 1
          for (int c = 0; c < BN / 64; ++c) {
            uint32_t r[64];
            tmem_ld_x32(t_addr + c * 64, r);
            tmem_ld_x32(t_addr + c * 64 + 32, r + 32);
            if (lane == 0) tma_store_wait_read<1>();
            __syncwarp();
            tmem_ld_wait();
            uint8_t* dst = my_epi + buf * kEpiBufBytes + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t p[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[j * 8 + 2 * q]),
                                                         __uint_as_float(r[j * 8 + 2 * q + 1]));
                p[q] = *reinterpret_cast<uint32_t*>(&h);
              }
              *reinterpret_cast<uint4*>(dst + ((j ^ (lane & 7)) << 4)) = make_uint4(p[0], p[1], p[2], p[3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmC, my_epi + buf * kEpiBufBytes, n0 + c * 64, m0 + ew * 32);
              tma_store_commit();
            }
            buf ^= 1;
          }
        } else {
          // rows m0 + ew*32 .. +31 of the full result belong to rank `peer`. Each 32 x 64 chunk goes through the
          // warp's swizzled staging buffer so that the stores to the owner are whole 128-byte lines (4 rows per
          // instruction) instead of 32 scattered 16-byte pieces.
          const int lrow0 = m0 - peer * a.Ts + ew * 32;
          uint8_t* tile_base = a.peers.base[peer] + a.recv_off[slot] + (((size_t)a.rank * a.Ts + lrow0) * a.N + n0) * 2;
          uint8_t* stage = my_epi;
#pragma unroll 1
          for (int c = 0; c < BN / 64; ++c) {
            uint32_t r[64];
            tmem_ld_x32(t_addr + c * 64, r);
            tmem_ld_x32(t_addr + c * 64 + 32, r + 32);
            tmem_ld_wait();
            uint8_t* dst = stage + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t p[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[j * 8 + 2 * q]),
                                                         __uint_as_float(r[j * 8 + 2 * q + 1]));
                p[q] = *reinterpret_cast<uint32_t*>(&h);
              }
              *reinterpret_cast<uint4*>(dst + ((j ^ (lane & 7)) << 4)) = make_uint4(p[0], p[1], p[2], p[3]);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int row = i * 4 + (lane >> 3), seg = lane & 7;
              const int4 v = *reinterpret_cast<const int4*>(stage + row * 128 + ((seg ^ (row & 7)) << 4));
              st_na_v4(tile_base + (size_t)row * a.N * 2 + c * 128 + seg * 16, v);
            }
            __syncwarp();
          }
          __threadfence_system();
          __syncwarp();
          if (lane == 0) {
            red_add_release_sys(reinterpret_cast<uint32_t*>(a.peers.base[peer] + a.arrive_off) + a.rank, 1u);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(&tempty[ab], 0));
      }
      if ((a.mode == 0 || local_rs) && lane == 0) tma_store_wait<0>();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer may still signal this CTA's barriers or read its operands until here
    if (warp == 2) {
      tc_fence_after();
      tmem_dealloc_pair(tmem_base, C::kTmemCols);
    }

    if (a.mode == 1 && (a.phase_mask & 2) && !local_rs) {
      tp_owner_reduce(a, per_src, slot, tag, epoch, &s_ok);
    }
  }
  if (cta_done_is_last(&a.ctrl[1], gridDim.x)) {
    if (threadIdx.x == 0 && (a.phase_mask & 2)) a.ctrl[0] = epoch + 1;
    // the counters that a call takes part in keep step with the epoch on the short paths too
    if (threadIdx.x == 0 && a.mode == 0 && a.R == 1) a.chunk_done[0] = (uint32_t)tag * (uint32_t)a.n_copy;
    if (threadIdx.x == 0 && local_rs)
      *reinterpret_cast<uint32_t*>(a.peers.base[0] + a.arrive_off) = (uint32_t)tag * per_src;
  }
}

}  // namespace

template <int BN>
static int launch(const TpArgs& a, const CUtensorMap& tmA, const CUtensorMap& tmOwn, const void* w, const CUtensorMap& tmC, int grid,
                  cudaStream_t stream) {
  CUtensorMap tmB;
  if (make_tmap_2d(&tmB, TMAP_BF16, w, a.K, a.N, (uint64_t)a.K * 2, BK, Cfg<BN>::kBNH, TMAP_SW_128B)) return -UMDK_ERR_BAD_ARG;
  UMDK_CUDA_CHECK(cudaFuncSetAttribute(tp_gemm_2sm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::kSmemBytes));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg<BN>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  UMDK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, tp_gemm_2sm_kernel<BN>, tmA, tmOwn, tmB, tmC, a));
  return 0;
}

// Columns of a pair's tiles: the widest unless narrower ones end sooner. A pair's time is its number of tiles times what one
// takes: K / 64 steps of 520 / 310 / 215 cycles for 256 / 128 / 64 columns (265 for 128 on few pairs; the barriers of a step
// bound the 64), and 1000 / 300 / 200 for what the last epilogue adds. Measured with one rank in us, 256 / 128 / 64 columns:
// 256 x 8192 x 1024 (rows, K, columns) 47.1 / 28.4 / 25.2, 640 x 4096 x 2560 29.9 / 21.0 / 27.1, 1536 x 2048 x 4096
// 31.3 / 28.0 / 39.7, 1024 x 8192 x 4096 53.2 / 56.9 / 84.4, 8064 x 6656 x 4096 296 / 379 / 646.
// Where ranks exchange partial results tiles have 256 columns: the arrivals are counted in those.
static int tile_columns(int mode, int R, int Ts, int N, int K, int phase_mask, int pairs) {
  if (mode == 1 && !(R == 1 && (phase_mask & 3) == 3)) return 256;
  const long rows = (long)R * ((Ts + 255) / 256);
  const long step[3] = {520, 310, 215}, ends[3] = {1000, 300, 200};
  int best = 256;
  long least = 0;
  for (int i = 0; i < 3; ++i) {
    const int bn = 256 >> i;
    const long waves = (rows * (N / bn) + pairs - 1) / pairs, t = waves * (K / BK) * step[i] + ends[i];
    if (i == 0 || t + t / 20 < least) {   // 5 %: at equal times the wider tiles read less
      least = t;
      best = bn;
    }
  }
  return best;
}

// Launch of the CTA-pair kernel; called by umdk_tp_gemm. Returns 0 or a negative error.
int tp_gemm_2sm_launch(const TpArgs& a, const void* A, const void* w, void* out, int grid, cudaStream_t stream) {
  const int M = a.R * a.Ts;
  CUtensorMap tmA, tmOwn, tmC;
  if (make_tmap_2d(&tmOwn, TMAP_BF16, a.x_local, a.K, a.mode == 0 ? a.Ts : M, (uint64_t)a.K * 2, BK, BMH, TMAP_SW_128B))
    return -UMDK_ERR_BAD_ARG;
  if (make_tmap_2d(&tmA, TMAP_BF16, A, a.K, M, (uint64_t)a.K * 2, BK, BMH, TMAP_SW_128B)) return -UMDK_ERR_BAD_ARG;
  if (make_tmap_2d(&tmC, TMAP_BF16, out, a.N, a.mode == 0 ? M : a.Ts, (uint64_t)a.N * 2, 64, 32, TMAP_SW_128B))
    return -UMDK_ERR_BAD_ARG;
  const int pairs = (grid - (a.mode == 0 && a.R > 1 ? a.n_copy : 0)) / 2;
  switch (tile_columns(a.mode, a.R, a.Ts, a.N, a.K, a.phase_mask, pairs)) {
    case 64: return launch<64>(a, tmA, tmOwn, w, tmC, grid, stream);
    case 128: return launch<128>(a, tmA, tmOwn, w, tmC, grid, stream);
    default: return launch<256>(a, tmA, tmOwn, w, tmC, grid, stream);
  }
}

}  // namespace umdk

// Columns of the tiles that a launch on `pairs` CTA pairs takes (64, 128 or 256).
UMDK_API int umdk_tp_tile_columns(int mode, int R, int Ts, int N, int K, int phase_mask, int pairs) {
  if (mode < 0 || mode > 1 || R < 1 || Ts < 128 || N < 256 || K < 64 || pairs < 1) return -UMDK_ERR_BAD_ARG;
  return umdk::tile_columns(mode, R, Ts, N, K, phase_mask, pairs);
}
