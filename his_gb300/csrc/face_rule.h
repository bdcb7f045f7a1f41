// When a float64 grid set keeps face planes (swe2d_tile64.cuh) for the two-kernel step.
#pragma once
#include <cstddef>

namespace his {

// Sets of fewer cells than FACES_LEAST do without: two launches more cost what the faces saved
// would (100 x 81: 120 us per call with its CFL rate fused, 131 split; 163 x 201 even;
// 400 x 325 331 against 309).  So do sets whose faces would take more than FACES_MOST, or more than
// a sixteenth of the free device memory: the planes buy a tenth of a step's time, and what a
// caller still has to allocate, or another set of its program, would miss the room.
constexpr size_t FACES_MOST = (size_t)4 << 30, FACES_LEAST = 40000;
inline bool faces_taken(size_t bytes, size_t cells, size_t free_bytes) {
    return cells >= FACES_LEAST && bytes <= FACES_MOST && bytes <= free_bytes / 16;
}

}  // namespace his
