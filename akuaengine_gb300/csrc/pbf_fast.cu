// The walk and the pair kernels in default (fast) math.
#include "pbf_passes.cuh"

namespace akua {

void enqueue_pairs_fast(akua_pbf* s, cudaStream_t st, Marker& mark) {
    enqueue_pairs<false>(s, st, mark);
}

}  // namespace akua
