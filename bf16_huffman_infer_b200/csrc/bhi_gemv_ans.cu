// The fused decode + product of rANS-coded layers.
#include "bhi_gemv.cuh"

namespace bhi {

template int gemv_launch<AnsCodec>(const Layer &, const AnsArgs &, const uint8_t *, const uint16_t *, const uint16_t *, uint16_t *,
                                    const PeerSet *, int, bool, cudaStream_t);

cudaError_t take_gemv_ans_status(int *out) { return take_status(out); }

}  // namespace bhi
