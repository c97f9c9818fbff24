// GEMM of prefill sizes on pairs of SMs (gemm_pair.cu), for the launchers of gemm_sm100.cu.
#pragma once
#include <cuda_runtime.h>

namespace sglb {

// Row groups of a grouped product, device memory: [count + 1] row offsets, group and first row of each token tile, number of tiles.
struct GemmGroups {
  const int *offsets, *tile_group, *tile_row0, *num_tiles;
  int count;
};

// Whether a dense product of more than 256 tokens is faster here than in tiles of 128 x `single_bn` on single SMs.
bool gemm_pair_pays(int T, int N, int K, int single_bn);

int gemm_pair(const void* x, long long ldx, const void* w, const void* bias, void* out, int T, int N, int K, bool gated,
              const GemmGroups* groups, int bt, cudaStream_t stream);

}  // namespace sglb
