// Host interface of the attention core inside the library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksb {
namespace attn {

struct Call {
  const void* q8;   // operands as the C ABI's ksb_sage_attn takes them
  const float* qs;
  const void* k8;
  const float* ks;
  const void* vt;
  const float* vs;
  int64_t H, Lq, Lk;
  const int32_t* tile_offsets;  // per Q block, or per pair of Q blocks with pair_lists
  const int32_t* tile_entries;
  const int32_t* order;
  bool pair_lists;
  // output row l of head h: out + (h / heads_per_batch) * out_bs + l * out_ts + (h % heads_per_batch) * out_hs elements
  void* out;
  int64_t out_ts, out_hs, out_bs;
  int64_t heads_per_batch;  // 0: all heads belong to one sample
  void* const* peer_out;
  int n_peers;
  int64_t rows_per_peer;
};

int run(const Call& c, int dtype, bool chained, cudaStream_t st);

}  // namespace attn
}  // namespace ksb
