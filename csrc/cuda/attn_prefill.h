// Flash attention for many query rows (attn_prefill.cu): grouped-query prefill and materialised latent-attention prefill.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace plow {

struct PrefillArgs {
  const void* q;            // bf16 [rows][nq][hdq]
  const void* k;            // bf16: keys; for latent attention [tokens][heads][256] = [key part | value]
  const void* v;            // bf16: values (= k for latent attention)
  const void* kr;           // latent attention: rotary key part [tokens][64], shared by the heads; else null
  const int* page_table;    // [slots][max_pages]: 64-token pages
  const int* seq;           // [rows]
  const int* pos;           // [rows], < 0: inactive
  void* chunks;             // scratch: 8 ints per chunk
  int chunk_cap;            // chunks it holds
  int* counters;            // scratch: [0] number of chunks
  int* claim;               // scratch: work counter
  void* out;                // bf16 [rows][nq * 128]
  int* status;
  int64_t n_tokens;         // cached tokens the keys / values cover
  int rows, nq, nkv, max_pages, window;
  float scale;
};

// Head dim 128 (keys 128 or, with `kr`, 192 wide).  Returns 0 or an error code.
int launch_attn_prefill(const PrefillArgs& a, cudaStream_t stream);

}  // namespace plow
