// The launchers of the decode kernels, whose source files are compiled side by side: bhi_gemv_huffman.cu, bhi_gemv_ans.cu,
// bhi_tiles.cu.  Each returns kStagedDeclined for what it does not serve.
#pragma once

#include "bhi_staged.cuh"

namespace bhi {

template <class Codec>
int gemv_launch(const Layer &L, const typename Codec::Args &targs, const uint8_t *prepared, const uint16_t *X, const uint16_t *bias,
                uint16_t *Y, const PeerSet *peers, int B, bool pair_complete, cudaStream_t st);
template <class Codec>
int tile_launch(const Layer &L, const typename Codec::Args &targs, const uint8_t *prepared, const uint16_t *X, uint16_t *Y, int B,
                cudaStream_t st);
template <class Codec>
int tileq_launch(const Layer &L, const typename Codec::Args &targs, const uint8_t *prepared, const uint16_t *X, uint16_t *Y, int B,
                 cudaStream_t st);

// each reads and clears the status word of its source file
cudaError_t take_gemv_huffman_status(int *out);
cudaError_t take_gemv_ans_status(int *out);
cudaError_t take_tiles_status(int *out);

}  // namespace bhi
