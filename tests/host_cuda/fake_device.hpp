// What a test sets and reads of the device that is not there.
#pragma once

#include <cstddef>
#include <cstdint>
#include <map>

namespace fake {
extern size_t total, used;                   // device memory
extern int fail_pinned;                      // page-locked allocations to refuse
extern size_t used_after_failed_pinned;      // device memory held when the next one is made
extern std::map<uint32_t, int> permutations; // gather passes by width
extern int small_runs, overlaps;             // one-launch programs; those whose workspace others hold
}  // namespace fake
