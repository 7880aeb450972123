// Argument blocks of the expert-parallel entry points that the Python call path (csrc/pycalls/calls.cpp) uses too.
#pragma once
#include <stdint.h>

constexpr int kUmdkMaxRanks = 32;

struct UmdkEpDispatchParams {
  int R, rank, E, K, H, cap, quant, T;
  int n_cap, a_cap, num_ctas, phase_mask;
  void* peers[kUmdkMaxRanks];
  const void* x;
  const int64_t* topk_idx;
  const float* topk_w;
  const int* send_idx;
  const int* rank_slot;
  const int* num_per_expert;
  const int* num_per_rank;
  void* recv_x;
  float* recv_scales;
  int* expand_idx;
  int* recv_count;
  int64_t* recv_per_expert;
  int* recv_meta;
  int* counts_dev;
  int* counts_host;
  uint32_t* ctrl;
  int* status;
  long long* diag;   // optional [R] per-source wait times in ns (diagnose mode), else null
  int64_t* row_expert;        // optional [n_cap] local expert per row (-1 behind the received rows), with
  float* row_weight;          // [n_cap] routing weight per row (0 behind them)
  int64_t* per_expert_host;   // optional [E/R] copy of recv_per_expert in mapped host memory
  int* status_host;           // optional [4] copy of the status record in mapped host memory, written with the tag
  int host_tag;               // one rank: counts_host[6] becomes this when the counts are in host memory, [5] when everything the call
                              // writes is in memory (0: neither)
};

struct UmdkEpCombineParams {
  int R, rank, E, K, H, cap, T;
  int mode, apply_weights, n_rows, num_ctas, phase_mask;
  void* peers[kUmdkMaxRanks];
  const void* y;
  const int* recv_meta;
  const int* counts_dev;
  const int* src_idx;
  const uint8_t* in_rank;
  const int64_t* topk_idx;
  const float* topk_w;
  void* out;
  uint32_t* ctrl;
  int* status;
  long long* diag;   // optional [R] per-source wait times in ns (diagnose mode), else null
  int a_cap;         // mode 0: arrivals that recv_meta has room for
};

struct UmdkEpLLDispatchParams {
  int R, rank, E, K, H, T_cap, T, num_ctas, phase_mask;
  void* peers[kUmdkMaxRanks];
  const void* x;
  const int64_t* topk_idx;
  const int* send_idx;         // null: the dispatch derives positions and sizes itself
  const int* num_per_expert;
  int* group_off;
  int64_t* recv_per_expert;
  uint32_t* ctrl;
  int* status;
};

struct UmdkEpLLCombineParams {
  int R, rank, E, K, H, T_cap, T, num_ctas, phase_mask;
  void* peers[kUmdkMaxRanks];
  const void* y;
  const int* group_off;
  const int64_t* topk_idx;
  const float* topk_w;
  void* out;
  uint32_t* ctrl;
  int* status;
};
