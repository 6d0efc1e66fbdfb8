// list_form.h -- which form of the DEM list step the library runs (dem.cu dem_list_pick; host only).
#pragma once

#include <cstdint>

namespace peb {

// A scene counts as in contact from 2 list entries a sphere on, and then until they fall below 1.75:
// the count moves by a few per cent from one rebuild to the next, and every change of form costs a
// step outside the captured graph and a new capture.
inline bool list_dense(bool was, int64_t n, int64_t entries) {
    return was ? 4 * entries >= 7 * n : entries >= 2 * n;
}

// The overlapped form (2) or the plain one (0); all give the same results.  Overlapping pays once
// the contact kernel, which then integrates its spheres too, is long enough beside the integration
// of the others, and costs a longer start (its release and the last block's wait).  One scene of one
// material, us per step (plain / overlapped): FP64 mostly apart 100,000 spheres 6.6 / 6.3, 200,000
// 9.2 / 7.7, 700,000 21.7 / 19.1, 30,000 5.2 / 5.9; FP64 in contact 2,197 11.5 / 10.9, 97,336 23.8 /
// 22.5, 704,969 108 / 100; mixed mostly apart 400,000 10.5 / 10.3, 700,000 16.1 / 15.6, 200,000 8.3 /
// 10.0; mixed in contact 29,791 11.9 / 10.8, 195,112 27.7 / 24.4, 1,048,576 134 / 107, 8,000 10.3 /
// 10.5.  Batches of scenes stay plain (1.0M spheres in 64: 42.5 / 46.3).
// one: one scene of one material under the linear law, no orientations.
inline int list_form_rule(bool one, bool fp64, int64_t n, bool dense) {
    const bool over = dense ? fp64 || n >= 25000 : n >= (fp64 ? 100000 : 400000);
    return one && over ? 2 : 0;
}

}  // namespace peb
