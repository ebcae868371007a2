// The walk of the device SAH build's swap partition (sah_build.cuh), shared with a host-side
// test.
#pragma once

#include "common.cuh"

namespace gr {

// Where the swap partition leaves a non-match, R less.  T (`moved`) holds the positions of
// the matches after the first non-match p1, in order; pos starts at the non-match's own
// distance from p1 and steps to T[pos] - p1 until it is R or more.
//
// A step is as long as the number g of non-matches from p1 up to T[pos], which only grows
// with pos.  So where a position s steps of g ahead has the same g, all positions between
// have it too and the s steps are taken at once; s doubles while that holds and halves once
// it does not.  With g counting the runs of matches passed, a walk meets at most sqrt(2 R) of
// them and takes about 2 log2 of each one's steps.  Step by step, a few non-matches ahead of
// all matches (a small light listed before a large mesh) made one thread follow a chain as
// long as the scene.  Creation with a two-triangle light first, step by step and now: 20,000
// triangles 2.13 / 1.36 ms, 102,400 5.67 / 1.67, 400,000 18.3 / 2.34, 1,000,000 44.2 / 3.8;
// with the light last, where no walk is long, 1.33 / 1.36, 1.62 / 1.67, 2.40 / 2.35, 3.9 / 3.8.
template <class M>
GR_HD uint32_t sah_back(const M& moved, uint32_t pos, uint32_t R, uint32_t p1) {
    if (pos >= R) return pos;
    uint32_t g = static_cast<uint32_t>(moved[pos]) - p1 - pos, s = 1;
    bool grow = true;
    while (g - 1u < 0x80000000u) {  // (0 or negative cannot be: the walk would not end)
        const uint64_t to = pos + static_cast<uint64_t>(s) * g;
        const uint32_t ahead = to < R ? static_cast<uint32_t>(moved[to]) - p1 - static_cast<uint32_t>(to) : 0u;
        if (to < R && (s == 1 || ahead == g)) {
            const bool same = ahead == g;
            pos = static_cast<uint32_t>(to);
            g = ahead;
            if (!same) grow = true;  // another run
            if (same && grow) s *= 2;
            else if (s > 1) s /= 2;
        } else if (s == 1) {
            return static_cast<uint32_t>(to);
        } else {
            grow = false;
            s /= 2;
        }
    }
    return pos;
}

}  // namespace gr
