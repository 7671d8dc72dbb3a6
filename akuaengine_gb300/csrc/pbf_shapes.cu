// The walk at the tile shapes that akua_pbf_set_search_shape and the autotuner may choose instead of
// the default.
#include "pbf_passes.cuh"

namespace akua {
namespace {

static_assert(kSearchBlock == 128 && kListStage == 32, "the shape left out here");

template <bool EXACT>
void launch_shape(akua_pbf* s, cudaStream_t st, int density, float* feat) {
    const int b = s->search_block, g = s->search_stage;
    if (g == 48) {  // 64 or 128 threads (akua_pbf_set_search_shape refuses 256)
        if (b == 64) launch_search_shape<EXACT, 64, 48>(s, st, density, feat);
        else launch_search_shape<EXACT, 128, 48>(s, st, density, feat);
    } else if (g == 16) {
        if (b == 64) launch_search_shape<EXACT, 64, 16>(s, st, density, feat);
        else if (b == 256) launch_search_shape<EXACT, 256, 16>(s, st, density, feat);
        else launch_search_shape<EXACT, 128, 16>(s, st, density, feat);
    } else {
        if (b == 64) launch_search_shape<EXACT, 64, 32>(s, st, density, feat);
        else launch_search_shape<EXACT, 256, 32>(s, st, density, feat);
    }
}

}  // namespace

void launch_search_other(akua_pbf* s, cudaStream_t st, bool exact, int density, float* feat) {
    if (exact) launch_shape<true>(s, st, density, feat);
    else launch_shape<false>(s, st, density, feat);
}

}  // namespace akua
