// The order in which a group's camera paths enter the queue, shared by the path tracer's
// kernels and a host-side test.
//
// A group is `passes` passes over a width x height image; sample `slot` = pass * npix +
// row * width + col is where the film gather finds it.  Entry q of the camera-ray queue
// is not sample q: the queue runs through the image in patches, every pass of a few
// neighbouring pixels together.  A warp's camera rays then cover a patch of 4 pixels x 8
// passes instead of 32 pixels of a row, and the rays of a shading chunk (6,144 entries of
// 768 threads: 12 x 8 pixels x 64 passes) leave from one small part of the scene, so both
// they and the rays they continue as share nodes and primitives in L1.
// Which entry a path has changes no result.
//
//   quads   runs of ORDER_QUAD pixels of the pixel order, all passes of a quad together,
//           pass by pass
//   bands   the pixel order takes bands of ORDER_BAND rows, each in column groups
//           ORDER_QUAD wide, row by row; a remainder of the width is one narrower group
#pragma once

#include "common.cuh"

namespace gr {

#ifndef GR_ORDER_QUAD
#define GR_ORDER_QUAD 4
#endif
#ifndef GR_ORDER_BAND
#define GR_ORDER_BAND 8
#endif
constexpr uint32_t ORDER_QUAD = GR_ORDER_QUAD;
constexpr uint32_t ORDER_BAND = GR_ORDER_BAND;

struct PathOrder {
    uint32_t width = 0, height = 0, npix = 0, passes = 0;
    uint32_t quad_paths = 0;  // paths in full quads
    uint32_t full_bands = 0, last_rows = 0;
    FastDiv by_quad_paths;  // passes of one quad
    FastDiv by_band;        // pixels of a full band
    FastDiv by_last;        // pixels of a column group of the last band
    FastDiv by_npix, by_width;
};

struct PathSample {
    uint32_t pass, row, col, slot;
};

// At most 2^31 - 1 paths.
inline PathOrder make_path_order(uint32_t width, uint32_t height, uint32_t passes) {
    PathOrder o;
    o.width = width;
    o.height = height;
    o.npix = width * height;
    o.passes = passes;
    const uint32_t quads = o.npix / ORDER_QUAD;
    o.quad_paths = quads * ORDER_QUAD * passes;
    o.full_bands = height / ORDER_BAND;
    o.last_rows = height % ORDER_BAND;
    o.by_quad_paths = make_fastdiv(quads ? ORDER_QUAD * passes : 1u);
    o.by_band = make_fastdiv(width * ORDER_BAND);
    o.by_last = make_fastdiv(o.last_rows ? ORDER_QUAD * o.last_rows : 1u);
    o.by_npix = make_fastdiv(o.npix);
    o.by_width = make_fastdiv(width);
    return o;
}

// The sample of queue entry q < npix * passes.
GR_HD PathSample path_sample(const PathOrder& o, uint32_t q) {
    PathSample s;
    uint32_t i;  // position in the pixel order
    if (q < o.quad_paths) {
        const uint32_t quad = fast_div(q, o.by_quad_paths);
        const uint32_t r = q - quad * (ORDER_QUAD * o.passes);
        s.pass = r / ORDER_QUAD;
        i = quad * ORDER_QUAD + r % ORDER_QUAD;
    } else {
        const uint32_t left = o.npix % ORDER_QUAD, r = q - o.quad_paths;
        s.pass = r / left;
        i = o.npix - left + r % left;
    }
    const uint32_t band = fast_div(i, o.by_band);
    const uint32_t b = i - band * (o.width * ORDER_BAND);  // position in the band
    const bool full = band < o.full_bands;
    const uint32_t rows = full ? ORDER_BAND : o.last_rows;
    const uint32_t groups = o.width / ORDER_QUAD;
    const uint32_t g = full ? b / (ORDER_QUAD * ORDER_BAND) : fast_div(b, o.by_last);
    uint32_t row;
    if (g < groups) {
        const uint32_t r = b - g * (ORDER_QUAD * rows);
        row = r / ORDER_QUAD;
        s.col = g * ORDER_QUAD + r % ORDER_QUAD;
    } else {
        const uint32_t w = o.width % ORDER_QUAD, r = b - groups * (ORDER_QUAD * rows);
        row = r / w;
        s.col = groups * ORDER_QUAD + r % w;
    }
    s.row = band * ORDER_BAND + row;
    s.slot = s.pass * o.npix + s.row * o.width + s.col;
    return s;
}

}  // namespace gr
