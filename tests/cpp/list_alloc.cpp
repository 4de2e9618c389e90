// The tile lists' allocation arithmetic, as the list scan uses it: one group of
// 1,024 tiles, four to a thread, placed at `before`.
#include "cudaraster/detail/list_alloc.h"

extern "C" {

uint64_t group_entries(const int32_t* counts) {
    uint64_t sum = 0;
    for (int t = 0; t < 256; t++) sum += cr::entriesOf4(counts + 4 * t);
    return sum;
}
int32_t group_fits(const int32_t* counts, uint64_t before, int64_t capacity) {
    return cr::listsFit(before + group_entries(counts), capacity) ? 1 : 0;
}
int32_t reported(uint64_t total) { return cr::reportedEntries(total); }
int32_t holds(int32_t index, int64_t capacity) { return cr::listHolds(index, capacity) ? 1 : 0; }

}
