// Sparse top-k MLA flash-attention decode over a paged KV cache, on tcgen05 tensor cores.
//
// Shapes (DeepSeek-V3 style multi-head latent attention with absorbed projections): per sequence one query token,
// 128 heads, each head a 576-vector (512 latent + 64 rope); every head attends to the SAME key rows, which are the
// 576-wide latent rows of the paged cache, and the value of a key is the first 512 entries of that row. Only the
// `topk` rows listed in `indices` take part (-1 or >= seq_len: masked).
//
// Mapping to the hardware: the 128 heads are exactly the M = 128 rows of one tcgen05 MMA, and one sequence (one
// split of its key list) is handled by a CLUSTER OF TWO CTAs that split the work by feature dimension:
//   CTA 0 owns latent dims [0, 256), CTA 1 owns latent dims [256, 512); the 64 rope dims are taken in turn, chunk by chunk.
// Per chunk of 48 selected keys each CTA
//   gathers only ITS dims of the 48 rows (640 or 512 bytes per row; no byte of the cache is read twice),
//   computes a PARTIAL S[128 x 48] = Q[:, own dims] * K[:, own dims]^T   (20 or 16 MMAs of K = 16),
//   sends the partial to its partner through distributed shared memory and adds the partner's partial,
//   runs the online softmax (one head per thread; both CTAs arrive at the same P),
//   and accumulates its own 256 output columns O[128 x 256] += P[128 x 48] * V[48 x own latent dims]  (3 MMAs),
//   reading V from the SAME gathered tile through an MN-major descriptor.
// Splitting by dimension halves the resident Q (80 KB instead of 144 KB), which makes room for a ring of key tiles, and
// halves the Q*K^T work of each SM. Q moves to TMEM before the first chunk and P never leaves it: both are A operands read
// out of TMEM, so that shared memory (128 bytes a clock) only feeds the key tiles to the MMAs; two of the five stages of the
// ring lie where Q was.
// TMEM columns: S 48, two P of 24, Q 160, O 256. Roles inside a CTA (20 warps):
//   warps 0-7  softmax in two sets of four, which take whole chunks in turn: tcgen05.ld of S, add the partner's partial,
//              maximum (passed on from set to set), exp2, P to TMEM, lazy rescale of O
//   warps 8-11 exchange: tcgen05.ld of the same S and asynchronous stores of it into the partner's shared memory,
//              so that the round trip between the two CTAs is off the softmax warps' critical path
//   warps 12, 13 MMA issuers (one elected thread each), of Q * K^T and of P * V: S(c + 2) is made while the softmax of c runs
//   warps 14-19 gather producers: TMA tile::gather4 copies (four selected rows x 128 bytes per instruction, written
//              in the 128-byte-swizzled layout the MMA descriptors expect), completion counted in bytes on the
//              stage's barrier. A warp issues its lanes' copies some 80 cycles apart and different warps side by side:
//              48-key tiles of 640-byte pieces from 128 CTAs take 96 us for 2048 keys out of one warp, 57 us out of two,
//              45 us out of four or more (3.7 TB/s of random 640-byte reads; 22 bytes per SM and clock when they hit
//              L2). Gathering with 16-byte cp.async reaches the same 15 - 19 bytes with 16 warps, plain loads half of it.
// What bounds it now: a stage of the ring is filled in 3100 cycles (1200 of issue, 1900 until the last row is there) and held for
// 6400 (Q * K^T 600, 1250 of it waiting for S's columns; partials on their way 1400; add and maximum 900, exp2 750, P to TMEM 950,
// P * V 600): five stages give one chunk per 1930 cycles. The st.async of the partials (24 KB a chunk, 24 bytes a clock) keep the
// shared-memory queue that every barrier and load of the softmax goes through busy half of the time. With one set of eight
// warps a chunk (24 keys a thread) the softmax chain itself was the limit, 2600 cycles. Batch 64, 2048 of 32768 keys: 70.9 / 62.5 us,
// 128 x 1024 79.9 / 69.8, 23 x 1000 in three splits 26.0 / 24.7 (the rope dims in CTA 0 alone: 62.6, 71.3, 24.9); splits of one or two
// chunks have nothing to overlap and pay for a thread's 48 keys: 61 x 70 11.1 / 11.4, 1 x 2048 15.2 / 15.5. In between (one set): Q
// as an A operand in shared memory kept one thread issuing MMAs for 2240 cycles a chunk; copies by cp.async or plain loads, partials
// by bulk copies out of a sending buffer (79.7 against 73.9 us), the merge launched while the splits run were no faster, nor (two
// sets) are rows fetched into L2 ahead of the gather (62.5 / 66.9).
// What a call costs around its chunks (us of a call in a CUDA graph, before / after): the first tiles are on their way as soon as
// their rows are known and while Q moves, the partner is only waited for where it is first written to; one warp sets the barriers up;
// the result leaves through shared memory in whole pieces of rows; the last meeting of the two CTAs is signed up for before the
// epilogue. 1 x 2048 keys in 22 splits 18.8 / 15.2, 23 x 1000 in 3 29.5 / 26.0, 61 x 70 13.0 / 11.1, 64 x 2048 71.9 / 70.9.
// The running maximum is only raised when it grows by more than 8 (in log2 units); P then stays below 2^8 and the
// accumulated O needs rescaling only a few times per row instead of in most chunks.
// Every wait is bounded; a CTA that gives up raises the abort flag of both CTAs so the partner leaves at once.
// There is no attention code in the reference project; the op is specified by the serving configuration only.
#include "common.h"
#include "mla_waits.h"
#include "ptx.cuh"

namespace umdk {
namespace {

constexpr int kHeads = 128;
constexpr int kDim = 576;
constexpr int kDimV = 512;
constexpr int kPage = 64;
constexpr int kChunk = 48;                       // keys per pipeline step
constexpr int kStages = 5;
constexpr int kFreeStages = 3;   // the others lie where Q is until it has moved to TMEM
constexpr int kMaxSlabs = 5;                     // 64-dim slabs per CTA: 4 latent (+ 1 rope in CTA 0)
constexpr int kQSlabBytes = kHeads * 128;        // 16 KB
constexpr int kKSlabBytes = kChunk * 128;        // 6 KB
constexpr int kQBytes = kMaxSlabs * kQSlabBytes; // 81920
constexpr int kStageBytes = kMaxSlabs * kKSlabBytes;  // 30720
constexpr int kXBytes = kChunk * kHeads * 4;     // 24 KB, [key / 4][head][4] fp32; two of them, for chunks in turn
constexpr int kMaxChunks = 43;                   // 2064 keys per split at most
constexpr int kMaxKeys = kMaxChunks * kChunk;
constexpr int kSets = 2;            // softmax warp sets: set s (warps 4s .. 4s + 3) takes chunks s, s + 2, ...
constexpr int kSoftWarps = 4 * kSets;
constexpr int kExchangeWarp = kSoftWarps;        // warps 8..11
constexpr int kMmaWarp = kExchangeWarp + 4;      // warp 12: Q * K^T
constexpr int kPvWarp = kMmaWarp + 1;            // warp 13: P * V
constexpr int kProducerWarp = kPvWarp + 1;       // warps 14..19
constexpr int kProducerWarps = 6;
constexpr int kThreads = 32 * (kProducerWarp + kProducerWarps);
constexpr int kRowsPerThread = (kMaxKeys + kThreads - 1) / kThreads;
constexpr int kTmemCols = 512;
constexpr int kColS = 0;                         // S: kChunk columns
constexpr int kColP = kChunk;                    // two P buffers of kChunk / 2 columns
constexpr int kColQ = 2 * kChunk;                // Q as bf16 pairs, 32 columns per 64-dim slab
constexpr int kColO = 256;
static_assert(kColQ + kMaxSlabs * 32 <= kColO, "TMEM budget");
constexpr int kOffK = 0;
constexpr int kOffQ = kFreeStages * kStageBytes;
constexpr int kOffX1 = kStages * kStageBytes;      // begins in Q's memory: the partner writes there once Q has left it
constexpr int kOffX0 = kOffX1 + kXBytes;
constexpr int kOffRows = kOffX0 + kXBytes;
constexpr int kMaskWords = ((kMaxKeys + 31) / 32 + 2) / 2 * 2;   // a bit per key, and the word that the last chunk's 64 bits end in
constexpr int kOffMask = kOffRows + kMaxKeys * 4;
constexpr int kOffMax = kOffMask + (kMaskWords * 4 + 63) / 64 * 64;   // [2][128] running maxima of the last two chunks
constexpr int kOffSum = kOffMax + 2 * kHeads * 4;   // [kSets][128] (sum, its maximum) of the sets
constexpr int kOffTail = kOffSum + kSets * kHeads * 8;
constexpr int kSmemBytes = 1024 + kOffTail + 512;
static_assert(kSmemBytes <= 232448, "shared memory budget");
static_assert(kStages * kStageBytes <= kOffQ + kQBytes && kOffQ + kQBytes <= kOffX0, "what lies in Q's memory waits for it");
// The epilogue's way out: 32 rows of 512 bytes per softmax warp, a pitch that keeps both directions free of bank conflicts.
constexpr int kOutPitch = 512 + 16, kOutPitch16 = 256 + 16;
static_assert(kSoftWarps * 32 * kOutPitch <= kOffX1, "the epilogue's rows end in front of the exchange buffers");
static_assert(kStageBytes % 1024 == 0 && kKSlabBytes % 1024 == 0, "swizzle atoms must stay 1024-byte aligned");

struct MlaArgs {
  const __nv_bfloat16* kv;   // [num_pages, 64, 576]
  const int* block_table;    // [B, max_pages]
  const int* indices;        // [B, topk]
  const int* seq_lens;       // [B] or null
  __nv_bfloat16* out;        // [B, 128, 512]
  float* lse;                // [B, 128]
  float* part_o;             // [B, splits, 128, 512] fp32 (splits > 1)
  float* part_lse;           // [B, splits, 128]
  int B, topk, max_pages, num_pages, num_splits;
  float scale_log2;
  int* status;
  // optional [16] cycle counters of the first CTA (diagnose mode). Softmax thread 0 (chunks 0, 2, ...): [0] wait S, [1] TMEM
  // load, [4] wait partner's partial, [5] add + max, wait for the other set's maximum, exp2, [6] wait for P's buffer (and for the
  // P*V before a rescale), [7] rescale + P store. Exchange thread 0: [2] wait partner-free, [3] remote stores. Q*K thread: [8]
  // wait tile, [9] wait until S has been read, [11] issue, [15] all of it once Q is in TMEM. P*V thread: [10] wait P, [12] issue
  // and wait for the product before. First producer warp: [13] wait free stage, [14] issue.
  long long* diag;
};

// Bounded waits that also leave when either CTA of the pair has raised the abort flag.
template <bool kCluster>
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (kCluster ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(smem_u32(bar), parity)) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (!(kCluster ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(smem_u32(bar), parity))) {
    if ((++spins & 31u) == 0) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kSpinLimitCycles) return false;
    }
  }
  return true;
}
// Asynchronous 16-byte store into the partner CTA's shared memory; the bytes are counted on the partner's mbarrier
// (complete_tx), so the sender needs no release fence that would wait for every store to be acknowledged.
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d,
                                            uint32_t cluster_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   cluster_addr),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"(cluster_bar)
               : "memory");
}
// Four rows of a 2-D tensor (row numbers r.x .. r.w, `col` = first element of the box in each row) into four
// consecutive 128-byte rows of shared memory; the tensor map has a box of {64 elements, 1 row} and the 128-byte swizzle.
__device__ __forceinline__ void tma_gather4(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int col, int4 r) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5, %6, %7}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(col), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; issued by ONE thread. A: lane = row, each 32-bit column two consecutive K elements.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
               "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
// 2^x with the special-function unit's native approximation (2 ulp; -inf gives 0): P is rounded to bf16 anyway.
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
sparse_mla_decode_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                         const MlaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_sm = smem + kOffQ;
  uint8_t* k_sm = smem + kOffK;
  int* rows_sm = reinterpret_cast<int*>(smem + kOffRows);
  uint32_t* mask_sm = reinterpret_cast<uint32_t*>(smem + kOffMask);
  float* max_sm = reinterpret_cast<float*>(smem + kOffMax);
  float2* sum_sm = reinterpret_cast<float2*>(smem + kOffSum);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffTail);
  uint64_t* bar_q = bars;            // 1
  // Arrivals are one per WARP: the lanes order their own accesses before a __syncwarp() and lane 0 arrives, so a
  // barrier sees 4 arrivals per phase instead of 128 (128 arrivals on one barrier, remote ones above all, cost
  // more than the work they guard).
  uint64_t* bar_full = bars + 1;     // kStages, one arrival that expects the tile's bytes from the TMA gathers
  uint64_t* bar_empty = bar_full + kStages;    // kStages, one commit
  uint64_t* bar_step = bar_empty + kStages;    // kMlaBars: see mla_waits.h
  uint64_t* bar_xfull = bar_step + kMlaBars;   // 2, one local arrival that expects the 24 KB the partner's st.async stores deliver
  uint64_t* bar_xfree = bar_xfull + 2;   // 2, 4 arrivals from a set of the partner's softmax warps: its X may be overwritten
  uint64_t* bar_xq = bar_xfull + 4;      // 8 arrivals from the partner's softmax warps: Q has left the memory of its second X
  uint64_t* bar_qt = bar_xfull + 5;      // 8 softmax-warp arrivals: Q is in TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_xfull + 6);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int b = blockIdx.y;
  const int half = static_cast<int>(cluster_ctarank());   // == blockIdx.x & 1
  const int split = blockIdx.x >> 1;
  const int per_split = ((a.topk + a.num_splits - 1) / a.num_splits + kChunk - 1) / kChunk * kChunk;
  const int k_begin = split * per_split;
  const int k_end = min(a.topk, k_begin + per_split);
  const int num_chunks = (k_end - k_begin + kChunk - 1) / kChunk;   // at least one: splits without keys are not launched
  // 64-dim slabs of chunk c in this CTA: its 4 latent ones, and the rope one in turn with the partner
  auto slabs_of = [&](int c) { return (c & 1) == half ? 5 : 4; };
  const int seq_len = a.seq_lens ? a.seq_lens[b] : 0x7fffffff;

  if (warp == kThreads / 32 - 1) {
    auto init = [&](uint64_t* bar, int n, uint32_t count) {
      if (lane < n) mbar_init(bar + lane, count);
    };
    init(bar_q, 1, 1);
    init(bar_full, 2 * kStages, 1);   // and bar_empty
    if (lane < kMlaBars) mbar_init(&bar_step[lane], mla_arrivals(lane));
    init(bar_xfull, 2, 1);
    init(bar_xfree, 2, kSoftWarps / kSets);
    init(bar_xq, 2, kSoftWarps);   // and bar_qt
    mbar_fence_init();
    fence_proxy_async_smem();   // the barriers' initial state, before the copy engine counts on it
    __syncwarp();
    if (lane == 0) {
      *s_abort = 0;
      mbar_expect_tx(bar_q, kQBytes);   // Q is on its way while the rows are resolved
      for (int j = 0; j < kMaxSlabs; ++j) {
        const int dim0 = j < 4 ? half * 256 + j * 64 : 512;
        tma_load_2d(q_sm + j * kQSlabBytes, &tmQ, bar_q, dim0, b * kHeads);
      }
      tma_prefetch_desc(&tmKV);
    }
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  // Resolve every selected row of this split once: index -> page -> row number in the pool (-1 = masked). All indices of a
  // thread are loaded before the first page lookup, so that the split pays two round trips to memory and not two per step.
  {
    int idx[kRowsPerThread], page[kRowsPerThread];
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const int kpos = k_begin + tid + i * kThreads;
      idx[i] = kpos < k_end ? a.indices[(size_t)b * a.topk + kpos] : -1;
    }
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      if (idx[i] >= seq_len) idx[i] = -1;
      const int pg = idx[i] / kPage;
      page[i] = idx[i] >= 0 && pg < a.max_pages ? a.block_table[(size_t)b * a.max_pages + pg] : -1;
    }
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const int k = tid + i * kThreads;
      if (k - lane >= num_chunks * kChunk) break;   // whole warps
      int row = -1;
      if (idx[i] >= 0) {
        if (page[i] < 0 || page[i] >= a.num_pages) umdk_set_status(a.status, UMDK_ERR_OVERFLOW, UMDK_PH_NONE, b, idx[i]);
        else row = page[i] * kPage + (idx[i] % kPage);
      }
      if (k < num_chunks * kChunk) rows_sm[k] = row;
      const uint32_t takes_part = __ballot_sync(0xffffffffu, row >= 0);
      if (lane == 0) mask_sm[k >> 5] = takes_part;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();   // this CTA's barriers exist; a role waits for the partner's before it first signals across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t peer = static_cast<uint32_t>(half ^ 1);
  const uint32_t peer_abort = map_to_cta(const_cast<int*>(s_abort), peer);

  auto give_up = [&](int phase, int detail) {
    if (!*s_abort) umdk_set_status(a.status, UMDK_ERR_TIMEOUT, phase, b, detail);
    *s_abort = 1;
    st_cluster_u32(peer_abort, 1u);
  };

  // `group`: which of the warps that share 32 heads, for kMlaMax
  auto step_bar = [&](MlaStep step, int c, int group = 0) { return &bar_step[mla_wait(step, c).bar + group]; };
  auto step_over = [&](MlaStep step, int c, int group = 0) {
    return wait_bar<false>(step_bar(step, c, group), mla_wait(step, c).parity, s_abort);
  };
  auto x_buf = [&](int c) { return reinterpret_cast<float*>(smem + ((c & 1) ? kOffX1 : kOffX0)); };

  if (warp < kSoftWarps) {
    // ===================================== softmax ======================================================
    // Two sets of four warps (a thread per head and set) take whole chunks in turn, so that the waits and latencies of two chunks
    // overlap. What they share is the maximum that P and O are relative to: the set of chunk c needs the one of chunk c - 1 once
    // it has its own scores, and passes its own on before the exponentials.
    const int set = warp >> 2, group = warp & 3;
    const int head = group * 32 + lane;   // == TMEM lane
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(group * 32) << 16);
    if (group == 0 && lane == 0 && set < num_chunks) mbar_expect_tx(&bar_xfull[set], kXBytes);   // re-armed after every chunk
    const uint32_t peer_xfree = map_to_cta(&bar_xfree[set], peer);
    const uint32_t peer_xq = map_to_cta(bar_xq, peer);
    float m_own = -INFINITY, l_run = 0.f;   // l_run: this set's chunks, relative to m_own
    // Q moves from shared memory into TMEM once: as the A operand of every Q * K^T step it would otherwise be read out
    // of shared memory again for each chunk (80 KB for 48 keys, more than everything else together), and the shared
    // memory's 128 bytes a clock are what this kernel runs out of first.
    bool ok = __all_sync(0xffffffffu, wait_bar<false>(bar_q, 0, s_abort));
    const bool q_here = ok;
    for (int j = set; j < kMaxSlabs; j += kSets) {
      const uint8_t* qrow = q_sm + j * kQSlabBytes + head * 128;
      uint32_t w[32];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint4 v = *reinterpret_cast<const uint4*>(qrow + ((u ^ (head & 7)) << 4));
        w[4 * u] = v.x;
        w[4 * u + 1] = v.y;
        w[4 * u + 2] = v.z;
        w[4 * u + 3] = v.w;
      }
      tmem_st_x32(lane_addr + kColQ + j * 32, w);
    }
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_qt);
    cluster_wait();
    if (lane == 0) mbar_arrive_cluster_relaxed(peer_xq);
    if (!q_here) give_up(UMDK_PH_TMA_FULL, 0);
    const bool dg = a.diag != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0;
    int dt[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // 32 bits: registers are short
    int t_prev = clock();
    auto lap = [&](int i) {
      if (dg) {
        const int t = clock();
        dt[i] += t - t_prev;
        t_prev = t;
      }
    };
    // A wait that runs out ends the loop of its warp; the decision becomes common at the barrier of the epilogue.
    for (int c = set; c < num_chunks && ok; c += kSets) {
      ok = __all_sync(0xffffffffu, step_over(kMlaS, c));
      if (!ok) {
        give_up(UMDK_PH_TMEM_FULL, c);
        break;
      }
      lap(0);
      tc_fence_after();
      uint32_t sr[kChunk];
      tmem_ld_x16(lane_addr + kColS, sr);
      tmem_ld_x16(lane_addr + kColS + 16, sr + 16);
      tmem_ld_x16(lane_addr + kColS + 32, sr + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(step_bar(kMlaRead, c));
      lap(1);
      // the partner's partial comes in through the exchange warps of the other CTA
      ok = __all_sync(0xffffffffu, wait_bar<true>(&bar_xfull[c & 1], (c >> 1) & 1, s_abort));
      if (!ok) {
        give_up(UMDK_PH_GROUP_READY, 1000 + c);
        break;
      }
      lap(4);
      // S = own partial + partner's partial (raw dot products; the scale is folded into the exponent below)
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      const float4* xp = reinterpret_cast<const float4*>(x_buf(c)) + head;
#pragma unroll
      for (int j4 = 0; j4 < kChunk / 4; ++j4) {
        const float4 xv = xp[j4 * kHeads];
        sr[4 * j4] = __float_as_uint(__uint_as_float(sr[4 * j4]) + xv.x);
        sr[4 * j4 + 1] = __float_as_uint(__uint_as_float(sr[4 * j4 + 1]) + xv.y);
        sr[4 * j4 + 2] = __float_as_uint(__uint_as_float(sr[4 * j4 + 2]) + xv.z);
        sr[4 * j4 + 3] = __float_as_uint(__uint_as_float(sr[4 * j4 + 3]) + xv.w);
      }
      const int word = c + (c >> 1);   // bits 48 c ...
      const unsigned long long valid =
          (static_cast<unsigned long long>(mask_sm[word + 1]) << 32 | mask_sm[word]) >> ((c & 1) * 16) & ((1ull << kChunk) - 1ull);
      if (valid != (1ull << kChunk) - 1ull) {   // the same for every thread of the set
#pragma unroll
        for (int j = 0; j < kChunk; ++j)
          if (!((valid >> j) & 1ull)) sr[j] = __float_as_uint(-INFINITY);
      }
#pragma unroll
      for (int j = 0; j < kChunk; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(sr[j]));
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // every lane's loads of X have returned (mx depends on them); keep the arrival behind that dependence
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 0));
      // re-armed before the partner may send again (its permission needs this warp's arrival below)
      if (group == 0 && lane == 0 && c + kSets < num_chunks) mbar_expect_tx(&bar_xfull[c & 1], kXBytes);
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_relaxed(peer_xfree);
      mx *= a.scale_log2;   // scale_log2 > 0: the maximum of the scaled scores
      float m_run = -INFINITY;
      if (c >= 1) {
        ok = __all_sync(0xffffffffu, step_over(kMlaMax, c - 1, group));
        if (!ok) {
          give_up(UMDK_PH_GROUP_READY, 4000 + c);
          break;
        }
        m_run = max_sm[((c - 1) & 1) * kHeads + head];
      }
      // lazy maximum: raise it only when it grows by more than 8 (P stays below 2^8)
      const float m_new = mx > m_run + 8.f || m_run == -INFINITY ? fmaxf(m_run, mx) : m_run;
      max_sm[(c & 1) * kHeads + head] = m_new;
      __syncwarp();
      if (lane == 0) mbar_arrive(step_bar(kMlaMax, c, group));
      const float neg_m = m_new == -INFINITY ? 0.f : -m_new;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[kChunk / 2];
#pragma unroll
      for (int j = 0; j < kChunk / 2; ++j) {
        const float p0 = ex2_approx(fmaf(__uint_as_float(sr[2 * j]), a.scale_log2, neg_m));
        const float p1 = ex2_approx(fmaf(__uint_as_float(sr[2 * j + 1]), a.scale_log2, neg_m));
        sum4[j & 3] += p0 + p1;
        const __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
        pk[j] = *reinterpret_cast<const uint32_t*>(&hh);
      }
      // (a sum relative to -inf is 0)
      l_run = l_run * (m_own == m_new ? 1.f : ex2_approx(m_own - m_new)) + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      m_own = m_new;
      lap(5);
      // P(c) goes where P(c-2) was: its product is through
      if (c >= 2) {
        ok = __all_sync(0xffffffffu, step_over(kMlaFree, c - 2));
        if (!ok) {
          give_up(UMDK_PH_TMEM_EMPTY, 500 + c);
          break;
        }
      }
      // O (P(0) .. P(c-1), relative to m_run) is rescaled when P(c-1) * V has been added to it; without a rescale nothing here
      // waits for that product. Where nothing has been seen yet (m_run = -inf) O is zero.
      const float alpha = m_run == m_new || m_run == -INFINITY ? 1.f : ex2_approx(m_run - m_new);
      const bool scale_o = c >= 1 && __any_sync(0xffffffffu, alpha != 1.f);
      if (scale_o) {
        ok = __all_sync(0xffffffffu, step_over(kMlaO, c - 1));
        if (!ok) {
          give_up(UMDK_PH_TMEM_EMPTY, c);
          break;
        }
      }
      lap(6);
      tc_fence_after();
      if (scale_o) {
#pragma unroll 1
        for (int c0 = 0; c0 < 256; c0 += 32) {
          uint32_t o[32];
          tmem_ld_x32(lane_addr + kColO + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_x32(lane_addr + kColO + c0, o);
        }
        tmem_st_wait();
      }
      // P as the A operand of P * V, key pairs in 24 columns: through shared memory the store and its proxy fence alone took some
      // 800 cycles a chunk next to the MMAs' operand reads
      tmem_st_x16(lane_addr + kColP + (c & 1) * (kChunk / 2), pk);
      tmem_st_x8(lane_addr + kColP + (c & 1) * (kChunk / 2) + 16, pk + 16);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(step_bar(kMlaP, c));
      lap(7);
    }
    if (dg) {
      for (int i = 0; i < 8; ++i)
        if (i != 2 && i != 3) a.diag[i] = dt[i];
    }
    cluster_arrive();   // the last word to the partner has been said
    // ---- epilogue: this CTA's 256 output columns, half of them per set ----
    // (every decision below is the same for all eight warps: the TMEM loads are warp-collective)
    if (ok) {
      ok = __all_sync(0xffffffffu, step_over(kMlaEnd, 0));
      if (!ok) {   // the partner may have left
        if (!*s_abort) umdk_set_status(a.status, UMDK_ERR_TIMEOUT, UMDK_PH_TMEM_EMPTY, b, 2000);
        *s_abort = 1;
      }
    }
    // both sets' sums, relative to the last maximum
    sum_sm[set * kHeads + head] = make_float2(l_run, m_own);
    ok = bar_and<32 * kSoftWarps>(1, ok);
    const float2 other = sum_sm[(set ^ 1) * kHeads + head];
    const float m_run = fmaxf(m_own, other.y);
    l_run = l_run * (m_own == m_run ? 1.f : ex2_approx(m_own - m_run)) + other.x * (other.y == m_run ? 1.f : ex2_approx(other.y - m_run));
    tc_fence_after();
    if (ok) {
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const float lse2 = l_run > 0.f ? m_run + log2f(l_run) : -INFINITY;
      // A thread has a row of its own: stored from here, a warp's 16 bytes per lane would touch 32 rows each time (128 x 256 fp32:
      // 11000 cycles, bf16 5000). The rows go through the memory of the key tiles and out in pieces of 512 or 256 bytes.
      const int col0 = set * 128;
      uint8_t* const rows = smem + warp * (32 * kOutPitch);
      if (a.num_splits == 1) {
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 32) {
          uint32_t o[32];
          tmem_ld_x32(lane_addr + kColO + col0 + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(o[q * 8 + 2 * i]) * inv,
                                                              __uint_as_float(o[q * 8 + 2 * i + 1]) * inv);
              w4[i] = *reinterpret_cast<const uint32_t*>(&hh);
            }
            *reinterpret_cast<uint4*>(rows + lane * kOutPitch16 + (c0 + q * 8) * 2) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
          }
        }
        __syncwarp();
        __nv_bfloat16* dst = a.out + ((size_t)b * kHeads + (warp & 3) * 32) * kDimV + half * 256 + col0;
#pragma unroll 8
        for (int r = lane >> 4; r < 32; r += 2)
          *reinterpret_cast<uint4*>(dst + (size_t)r * kDimV + (lane & 15) * 8) =
              *reinterpret_cast<const uint4*>(rows + r * kOutPitch16 + (lane & 15) * 16);
        if (half == 0 && set == 0 && a.lse) a.lse[(size_t)b * kHeads + head] = lse2 * 0.6931471805599453f;
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 32) {
          uint32_t o[32];
          tmem_ld_x32(lane_addr + kColO + col0 + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            *reinterpret_cast<float4*>(rows + lane * kOutPitch + (c0 + q * 4) * 4) =
                make_float4(__uint_as_float(o[q * 4]) * inv, __uint_as_float(o[q * 4 + 1]) * inv,
                            __uint_as_float(o[q * 4 + 2]) * inv, __uint_as_float(o[q * 4 + 3]) * inv);
          }
        }
        __syncwarp();
        float* dst = a.part_o + (((size_t)b * a.num_splits + split) * kHeads + (warp & 3) * 32) * kDimV + half * 256 + col0;
#pragma unroll 8
        for (int r = 0; r < 32; ++r)
          *reinterpret_cast<float4*>(dst + (size_t)r * kDimV + lane * 4) =
              *reinterpret_cast<const float4*>(rows + r * kOutPitch + lane * 16);
        if (half == 0 && set == 0) a.part_lse[((size_t)b * a.num_splits + split) * kHeads + head] = lse2;
      }
    }
  } else if (warp == kMmaWarp) {
    // ===================================== MMA issuer, Q * K^T ==========================================
    cluster_wait();
    if (elect_one()) {
      constexpr uint32_t idesc_qk = umma_idesc(kFmtBF16, kFmtBF16, kHeads, kChunk);
      bool ok = wait_bar<false>(bar_qt, 0, s_abort);
      if (!ok) give_up(UMDK_PH_TMA_FULL, 0);
      const uint64_t k_desc = umma_desc_k_sw128(smem_u32(k_sm));
      const bool dg = a.diag != nullptr && blockIdx.x == 0 && blockIdx.y == 0;
      long long dt[4] = {0, 0, 0, 0};
      const long long t_begin = dg ? clock64() : 0;
      long long t_prev = t_begin;
      auto lap = [&](int i) {
        if (dg) {
          const long long t = clock64();
          dt[i] += t - t_prev;
          t_prev = t;
        }
      };
      for (int c = 0; c < num_chunks && ok; ++c) {
        const int st = c % kStages;
        ok = wait_bar<false>(&bar_full[st], (c / kStages) & 1, s_abort);
        if (!ok) {
          give_up(UMDK_PH_TMA_FULL, 100 + c);
          break;
        }
        lap(0);
        if (c >= 1) ok = step_over(kMlaRead, c - 1);   // S(c) takes the place of S(c-1)
        if (!ok) {
          give_up(UMDK_PH_TMEM_EMPTY, 100 + c);
          break;
        }
        lap(1);
        tc_fence_after();
        // one add per step: everything else about the operands is constant
        const uint64_t bd = k_desc + st * (kStageBytes >> 4);
        const uint32_t q = tmem_base + kColQ;
#pragma unroll
        for (int j = 0; j < kMaxSlabs; ++j) {
          if (j >= slabs_of(c)) break;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ta(tmem_base + kColS, q + j * 32 + k * 8, bd + j * (kKSlabBytes >> 4) + 2 * k, idesc_qk, (j | k) ? 1u : 0u);
        }
        umma_commit(step_bar(kMlaS, c));
        lap(3);
      }
      if (dg) {
        for (int i = 0; i < 4; ++i)
          if (i != 2) a.diag[8 + i] = dt[i];
        a.diag[15] = clock64() - t_begin;
      }
      umma_commit(step_bar(kMlaEnd, 0));   // also where it gave up: see the end of the kernel
    }
  } else if (warp == kPvWarp) {
    // ===================================== MMA issuer, P * V ============================================
    cluster_wait();
    // A thread of its own: S(c+2) can be made while the softmax of chunk c is not through, and neither product waits for what
    // the other one's next step needs.
    if (elect_one()) {
      constexpr uint32_t idesc_pv = umma_idesc(kFmtBF16, kFmtBF16, kHeads, 256, 0, 1);
      const uint64_t v_desc = umma_desc_mn_sw128(smem_u32(k_sm), kKSlabBytes, 1024);
      const bool dg = a.diag != nullptr && blockIdx.x == 0 && blockIdx.y == 0;
      long long dt[2] = {0, 0};
      long long t_prev = dg ? clock64() : 0;
      for (int c = 0; c < num_chunks; ++c) {
        const int st = c % kStages;
        // P(c-1) * V is through: the buffer may take P(c+1)
        if (c >= 1 && !step_over(kMlaO, c - 1)) {
          give_up(UMDK_PH_TMEM_EMPTY, 200 + c);
          break;
        }
        if (c >= 1) mbar_arrive(step_bar(kMlaFree, c - 1));
        if (!wait_bar<false>(&bar_full[st], (c / kStages) & 1, s_abort)) {   // (over: S(c) was made of it)
          give_up(UMDK_PH_TMA_FULL, 200 + c);
          break;
        }
        if (dg) {
          const long long t = clock64();
          dt[1] += t - t_prev;
          t_prev = t;
        }
        if (!step_over(kMlaP, c)) {
          give_up(UMDK_PH_GROUP_READY, 200 + c);
          break;
        }
        if (dg) {
          const long long t = clock64();
          dt[0] += t - t_prev;
          t_prev = t;
        }
        tc_fence_after();
        const uint64_t vd = v_desc + st * (kStageBytes >> 4);
#pragma unroll
        for (int k = 0; k < kChunk / 16; ++k)   // 16 keys per step: A advances 8 columns, B two 8-key groups
          umma_f16_ta(tmem_base + kColO, tmem_base + kColP + (c & 1) * (kChunk / 2) + k * 8, vd + k * (2048 >> 4), idesc_pv,
                      (c | k) ? 1u : 0u);
        if (c + 1 < num_chunks) {   // behind the last chunk one commit, below, is for everybody
          umma_commit(&bar_empty[st]);
          umma_commit(step_bar(kMlaO, c));
        }
      }
      if (dg) {
        a.diag[10] = dt[0];
        a.diag[12] = dt[1];
      }
      umma_commit(step_bar(kMlaEnd, 0));   // also where it gave up
    }
  } else if (warp >= kExchangeWarp && warp < kMmaWarp) {
    // ===================================== exchange (warps 8..11) =======================================
    cluster_wait();
    const int head = (warp & 3) * 32 + lane;   // == TMEM lane
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t peer_x[2] = {map_to_cta(x_buf(0), peer) + static_cast<uint32_t>(head) * 16u,
                                map_to_cta(x_buf(1), peer) + static_cast<uint32_t>(head) * 16u};
    const uint32_t peer_xfull = map_to_cta(bar_xfull, peer);
    const bool dg = a.diag != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && head == 0;
    long long dt[2] = {0, 0};
    long long t_prev = dg ? clock64() : 0;
    for (int c = 0; c < num_chunks; ++c) {
      if (!__all_sync(0xffffffffu, step_over(kMlaS, c))) {
        give_up(UMDK_PH_TMEM_FULL, 3000 + c);
        break;
      }
      tc_fence_after();
      uint32_t sr[kChunk];
      tmem_ld_x16(lane_addr + kColS, sr);
      tmem_ld_x16(lane_addr + kColS + 16, sr + 16);
      tmem_ld_x16(lane_addr + kColS + 32, sr + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(step_bar(kMlaRead, c));
      if (dg) t_prev = clock64();
      // the partner's softmax warps must have read the partial of two chunks ago out of their exchange buffer; the second buffer
      // is Q's memory to begin with
      if (c >= 1 && !__all_sync(0xffffffffu, c == 1 ? wait_bar<false>(bar_xq, 0, s_abort)
                                                    : wait_bar<false>(&bar_xfree[c & 1], ((c >> 1) - 1) & 1, s_abort))) {
        give_up(UMDK_PH_GROUP_READY, c);
        break;
      }
      if (dg) {
        const long long t = clock64();
        dt[0] += t - t_prev;
        t_prev = t;
      }
#pragma unroll
      for (int j4 = 0; j4 < kChunk / 4; ++j4)
        st_async_v4(peer_x[c & 1] + j4 * (kHeads * 16), sr[4 * j4], sr[4 * j4 + 1], sr[4 * j4 + 2], sr[4 * j4 + 3],
                    peer_xfull + (c & 1) * 8);
      if (dg) dt[1] += clock64() - t_prev;
    }
    if (dg) {
      a.diag[2] = dt[0];
      a.diag[3] = dt[1];
    }
  } else {
    // ===================================== gather producers (warps 14..19) ==================================
    bool ok = true;
    const bool dg = a.diag != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && lane == 0 && warp == kProducerWarp;
    long long dt[2] = {0, 0};
    long long t_prev = dg ? clock64() : 0;
    auto lap = [&](int i) {
      if (dg) {
        const long long t = clock64();
        dt[i] += t - t_prev;
        t_prev = t;
      }
    };
    for (int c = 0; c < num_chunks && ok; ++c) {
      const int st = c % kStages, n_slabs = slabs_of(c);
      const int n_inst = (kChunk / 4) * n_slabs;   // gather4 copies per tile
      if (c == kFreeStages) {   // from here on in Q's memory
        cluster_wait();         // the first tiles are on their way without the partner
        ok = __all_sync(0xffffffffu, wait_bar<false>(bar_qt, 0, s_abort));
        if (!ok) {
          if (lane == 0) give_up(UMDK_PH_TMA_EMPTY, 4000);
          break;
        }
      }
      if (c >= kStages) {
        ok = __all_sync(0xffffffffu, wait_bar<false>(&bar_empty[st], ((c / kStages) - 1) & 1, s_abort));
        if (!ok) {
          if (lane == 0) give_up(UMDK_PH_TMA_EMPTY, c);
          break;
        }
      }
      lap(0);
      if (warp == kProducerWarp && lane == 0) mbar_expect_tx(&bar_full[st], static_cast<uint32_t>(n_slabs) * kKSlabBytes);
      __syncwarp();
      uint8_t* stage = k_sm + st * kStageBytes;
      const int4* rows4 = reinterpret_cast<const int4*>(rows_sm + c * kChunk);
      // A warp issues its lanes' copies one after the other, about 80 cycles apart, and different warps issue side by
      // side: the copies of a tile are dealt over all producer warps (nine each) instead of filling two of them.
      for (int u = lane * kProducerWarps + warp - kProducerWarp; u < n_inst; u += 32 * kProducerWarps) {
        const int grp = n_slabs == 4 ? u >> 2 : u / 5, slab = u - grp * n_slabs;
        int4 r = rows4[grp];
        r.x = max(r.x, 0);   // masked keys read row 0: their scores are set to -inf before the softmax
        r.y = max(r.y, 0);
        r.z = max(r.z, 0);
        r.w = max(r.w, 0);
        const int col = slab < 4 ? half * 256 + slab * 64 : 512;
        tma_gather4(stage + slab * kKSlabBytes + grp * 512, &tmKV, &bar_full[st], col, r);
      }
      lap(1);
    }
    if (num_chunks <= kFreeStages) cluster_wait();
    if (dg) {
      for (int i = 0; i < 2; ++i) a.diag[13 + i] = dt[i];
    }
  }
  __syncwarp();
  if (warp >= kSoftWarps) cluster_arrive();
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    // every MMA issued has retired (they read shared memory and write TMEM), also where the softmax warps gave up on them
    mbar_wait_warp(step_bar(kMlaEnd, 0), mla_wait(kMlaEnd, 0).parity);
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  cluster_wait();   // neither CTA leaves while the other may still write into its shared memory
}

// Joins the key-list splits that have keys (the first `live` of num_splits): out = sum_i exp2(lse_i - lse) * o_i. One CTA per
// (sequence, head), four columns per thread; the weights are made once per CTA and eight splits' partials are in flight at a
// time (bound by the latency of reading live x 2 KB per head out of L2).
__global__ void __launch_bounds__(128) mla_merge_kernel(const float* __restrict__ part_o,
                                                        const float* __restrict__ part_lse,
                                                        __nv_bfloat16* __restrict__ out, float* __restrict__ lse,
                                                        int num_splits, int live) {
  extern __shared__ float w_sm[];   // [live]
  const int bh = blockIdx.x;        // b * 128 + head
  const int b = bh / kHeads, head = bh % kHeads;
  const float4* po = reinterpret_cast<const float4*>(part_o + ((size_t)b * num_splits * kHeads + head) * kDimV) + threadIdx.x;
  const size_t step = (size_t)kHeads * kDimV / 4;
  float4 v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (u < live) v[u] = __ldg(po + u * step);
  if (threadIdx.x < 32) {
    const float* pl = part_lse + (size_t)b * num_splits * kHeads + head;
    float mx = -INFINITY;
    for (int s = threadIdx.x; s < live; s += 32) {
      w_sm[s] = pl[(size_t)s * kHeads];
      mx = fmaxf(mx, w_sm[s]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float den = 0.f;
    for (int s = threadIdx.x; s < live; s += 32) {
      w_sm[s] = w_sm[s] == -INFINITY ? 0.f : exp2f(w_sm[s] - mx);
      den += w_sm[s];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    for (int s = threadIdx.x; s < live; s += 32) w_sm[s] = den > 0.f ? w_sm[s] / den : 0.f;
    if (threadIdx.x == 0 && lse) lse[bh] = den > 0.f ? (mx + log2f(den)) * 0.6931471805599453f : -INFINITY;
  }
  __syncthreads();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < live; s0 += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (s0 + u >= live) break;
      if (s0 > 0) v[u] = __ldg(po + (s0 + u) * step);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (s0 + u >= live) break;
      const float w = w_sm[s0 + u];
      acc.x = fmaf(w, v[u].x, acc.x);
      acc.y = fmaf(w, v[u].y, acc.y);
      acc.z = fmaf(w, v[u].z, acc.z);
      acc.w = fmaf(w, v[u].w, acc.w);
    }
  }
  __nv_bfloat162 o2[2] = {__floats2bfloat162_rn(acc.x, acc.y), __floats2bfloat162_rn(acc.z, acc.w)};
  *reinterpret_cast<uint2*>(out + (size_t)bh * kDimV + threadIdx.x * 4) = *reinterpret_cast<const uint2*>(o2);
}

}  // namespace
}  // namespace umdk

using namespace umdk;

// Smallest num_splits the kernel accepts for a key list of `topk` entries (umdk_b200/ops/attention.py works it out itself; a test
// compares the two).
UMDK_API int umdk_sparse_mla_min_splits(int topk) { return (topk + kMaxKeys - 1) / kMaxKeys; }

// q: [B, 128, 576] bf16; kv: [num_pages, 64, 576] bf16; block_table: [B, max_pages]; indices: [B, topk];
// out: [B, 128, 512] bf16; lse: [B, 128] fp32 (may be null). part_o / part_lse: scratch for num_splits > 1
// ([B, splits, 128, 512] and [B, splits, 128] fp32).
UMDK_API int umdk_sparse_mla_decode(const void* q, const void* kv, const int* block_table, const int* indices,
                                    const int* seq_lens, void* out, float* lse, float* part_o, float* part_lse,
                                    int B, int topk, int max_pages, int num_pages, int num_splits, float sm_scale,
                                    int* status, void* stream, long long* diag) {
  if (B < 1 || topk < 1 || max_pages < 1 || num_pages < 1 || num_splits < 1) return -UMDK_ERR_BAD_ARG;
  if (num_splits > 1 && (part_o == nullptr || part_lse == nullptr)) return -UMDK_ERR_BAD_ARG;
  // one CTA pair resolves at most kMaxKeys rows of the key list up front (see umdk_sparse_mla_min_splits)
  const int per_split = ((topk + num_splits - 1) / num_splits + kChunk - 1) / kChunk * kChunk;   // as in the kernel
  if (per_split > kMaxKeys) return -UMDK_ERR_BAD_ARG;
  const int live = (topk + per_split - 1) / per_split;   // whole chunks: the last splits may be left without keys
  if ((size_t)num_pages * kPage > 0x7fffffffull) return -UMDK_ERR_BAD_ARG;
  CUtensorMap tmQ, tmKV;
  if (make_tmap_2d(&tmQ, TMAP_BF16, q, kDim, (uint64_t)B * kHeads, kDim * 2, 64, kHeads, TMAP_SW_128B))
    return -UMDK_ERR_BAD_ARG;
  // the cache as a matrix of token rows; box = one 128-byte piece of one row (tile::gather4 takes four of them)
  if (make_tmap_2d(&tmKV, TMAP_BF16, kv, kDim, (uint64_t)num_pages * kPage, kDim * 2, 64, 1, TMAP_SW_128B))
    return -UMDK_ERR_BAD_ARG;
  static bool attr = false;
  if (!attr) {
    UMDK_CUDA_CHECK(cudaFuncSetAttribute(sparse_mla_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kSmemBytes));
    attr = true;
  }
  MlaArgs a;
  a.kv = static_cast<const __nv_bfloat16*>(kv);
  a.block_table = block_table;
  a.indices = indices;
  a.seq_lens = seq_lens;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.lse = lse;
  a.part_o = part_o;
  a.part_lse = part_lse;
  a.B = B;
  a.topk = topk;
  a.max_pages = max_pages;
  a.num_pages = num_pages;
  a.num_splits = num_splits;
  a.scale_log2 = sm_scale * 1.4426950408889634f;
  a.status = status;
  a.diag = diag;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 grid(2 * live, B);
  sparse_mla_decode_kernel<<<grid, kThreads, kSmemBytes, s>>>(tmQ, tmKV, a);
  UMDK_CUDA_CHECK(cudaGetLastError());
  if (num_splits > 1) {
    const size_t smem = sizeof(float) * live;
    if (smem > 48 * 1024)
      UMDK_CUDA_CHECK(cudaFuncSetAttribute(mla_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    mla_merge_kernel<<<B * kHeads, 128, smem, s>>>(part_o, part_lse, static_cast<__nv_bfloat16*>(out), lse, num_splits, live);
    UMDK_CUDA_CHECK(cudaGetLastError());
  }
  return 0;
}

// Barrier and parity (2 * barrier + parity) of a wait of the kernel's: for the test that walks through the roles' orders.
UMDK_API int umdk_sparse_mla_wait(int step, int c) {
  if (step < kMlaS || step > kMlaMax || c < 0) return -UMDK_ERR_BAD_ARG;
  const MlaWait w = mla_wait(static_cast<MlaStep>(step), c);
  return 2 * w.bar + static_cast<int>(w.parity);
}
