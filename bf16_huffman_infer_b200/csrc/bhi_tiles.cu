// The fused products that keep their sums in tensor memory.
#include "bhi_tile.cuh"
#include "bhi_tileq.cuh"
#include "bhi_launch.cuh"

namespace bhi {

template int tile_launch<HuffCodec>(const Layer &, const HuffArgs &, const uint8_t *, const uint16_t *, uint16_t *, int, cudaStream_t);
template int tile_launch<AnsCodec>(const Layer &, const AnsArgs &, const uint8_t *, const uint16_t *, uint16_t *, int, cudaStream_t);
template int tileq_launch<HuffCodec>(const Layer &, const HuffArgs &, const uint8_t *, const uint16_t *, uint16_t *, int, cudaStream_t);
template int tileq_launch<AnsCodec>(const Layer &, const AnsArgs &, const uint8_t *, const uint16_t *, uint16_t *, int, cudaStream_t);

cudaError_t take_tiles_status(int *out) { return take_status(out); }

}  // namespace bhi
