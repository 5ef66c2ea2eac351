// sort_k64v64.cu -- every shape of the sort's tuning grid for uint64_t keys with uint64_t payloads.
#include "sort_kernels.cuh"

namespace gprtcu {
const std::array<SortRunFn, kSortGridSize> kSortTableK64V64 =
    make_sort_table<uint64_t, uint64_t>(std::make_index_sequence<kSortGridSize>{});
const SortSmallFn kSortSmallK64V64 = &sort_small_run<uint64_t, uint64_t>;
}  // namespace gprtcu
