// sort_k32v32.cu -- every shape of the sort's tuning grid for uint32_t keys with uint32_t payloads.
#include "sort_kernels.cuh"

namespace gprtcu {
const std::array<SortRunFn, kSortGridSize> kSortTableK32V32 =
    make_sort_table<uint32_t, uint32_t>(std::make_index_sequence<kSortGridSize>{});
const SortSmallFn kSortSmallK32V32 = &sort_small_run<uint32_t, uint32_t>;
}  // namespace gprtcu
