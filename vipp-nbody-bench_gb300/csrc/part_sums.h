// Scratch of an M2L whose tiles are shared out among work units (m2l_tc.cu,
// m2l_fp64.cu): the units' partial sums and a counter per tile.
#pragma once

#include <cstddef>

namespace gb {

template <typename T>
struct PartSums {
    T *part = nullptr;
    unsigned *cnt = nullptr;  // [tiles] finished units of a tile
    unsigned tiles = 0;       // tiles the two are sized for
    int p = 0;                // and the expansion order
    bool holds(unsigned t, int q) const { return part && cnt && t <= tiles && q <= p; }
};

// Tiles the scratch has to hold: those of the cell buffers (`bound`), up to `limit`, beyond
// which tiles run whole; none when no tree of these n particles can have as few as
// `limit` tiles of `rows` targets (its leaves hold at most `leaf` particles each, and
// at most 8 cells of each of the nsys trees are above level 2 and no targets).
inline unsigned split_tiles_held(std::size_t n, std::size_t leaf, std::size_t nsys, unsigned rows, unsigned bound, unsigned limit) {
    const std::size_t leaves = (n + leaf - 1) / leaf, targets = leaves > 8 * nsys ? leaves - 8 * nsys : 0;
    return targets / rows > limit ? 0 : bound < limit ? bound : limit;
}

// Both buffers anew; alloc(pointer, count) frees what the pointer held, sets it (null
// when it fails) and returns 0 or an error, which is passed on. Nothing is recorded as
// held before both are there, so that after a failure no smaller request passes for met.
template <typename T, class Alloc>
auto resize(PartSums<T> &s, unsigned tiles, int p, std::size_t values, Alloc &&alloc) -> decltype(alloc(s.cnt, values)) {
    s.tiles = 0, s.p = 0;
    auto e = alloc(s.part, values);
    if (e == decltype(e){}) e = alloc(s.cnt, static_cast<std::size_t>(tiles));
    if (e == decltype(e){}) s.tiles = tiles, s.p = p;
    return e;
}

}  // namespace gb
