// The walk and the pair kernels in exact math.
#include "pbf_passes.cuh"

namespace akua {

void enqueue_pairs_exact(akua_pbf* s, cudaStream_t st, Marker& mark) {
    enqueue_pairs<true>(s, st, mark);
}

}  // namespace akua
