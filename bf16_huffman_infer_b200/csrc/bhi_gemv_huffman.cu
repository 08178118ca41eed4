// The fused decode + product of Huffman-coded layers.
#include "bhi_gemv.cuh"

namespace bhi {

template int gemv_launch<HuffCodec>(const Layer &, const HuffArgs &, const uint8_t *, const uint16_t *, const uint16_t *, uint16_t *,
                                    const PeerSet *, int, bool, cudaStream_t);

cudaError_t take_gemv_huffman_status(int *out) { return take_status(out); }

}  // namespace bhi
