// The level schedule of SLRIter's in-place passes (src/MutoSLRIter.cpp:40-71).
//
// Muon i's level is one more than the highest level that an earlier muon
// left on any voxel of i's path.  A voxel's muons then have strictly
// increasing levels in index order, and two muons of one level share no
// voxel: running the muons of a level at once, level after level, gives
// every muon the image state of the muon-after-muon loop.  One ordered sweep
// over the pairs; the recurrence is sequential in the muon index.  Plain C++
// (host code, no CUDA types).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace muto {

// off[0..nt]: each muon's pairs vox[off[i] .. off[i+1]); voxels >= V are
// ignored.  Fills level[0..nt) (1-based) and returns the number of levels.
inline uint32_t slr_levels(const uint64_t* off, const uint32_t* vox, uint64_t nt, uint64_t V, uint32_t* level) {
    std::vector<uint32_t> last(V, 0);
    uint32_t levels = 0;
    for (uint64_t i = 0; i < nt; ++i) {
        uint32_t lv = 0;
        for (uint64_t k = off[i]; k < off[i + 1]; ++k)
            if (vox[k] < V) lv = std::max(lv, last[vox[k]]);
        ++lv;
        for (uint64_t k = off[i]; k < off[i + 1]; ++k)
            if (vox[k] < V) last[vox[k]] = lv;
        level[i] = lv;
        levels = std::max(levels, lv);
    }
    return levels;
}

// The steps that a schedule runs in: a level, or part of one, of at most `muons`
// muons (fewer than 256) and, unless it is one muon, at most `pairs` pairs, so that a
// pair's place in its step is a 32-bit number.  Level l's muons (1-based) are places
// start[l] .. start[l+1] of the level order, the pairs of place q are fo[q] ..
// fo[q+1].  Fills sstart with the steps' first places and the end, place[q] with the
// muon's place in its step; returns the number of steps.
inline uint32_t slr_steps(const std::vector<uint32_t>& start, uint32_t levels, const uint64_t* fo, uint32_t muons,
                          uint64_t pairs, std::vector<uint32_t>& sstart, std::vector<uint8_t>& place) {
    sstart.clear();
    place.assign(start[levels + 1], 0);
    for (uint32_t l = 1; l <= levels; ++l) {
        uint32_t first = start[l];
        for (uint32_t q = first; q < start[l + 1]; ++q) {
            if (q == start[l] || q - first == muons || fo[q + 1] - fo[first] > pairs) {
                first = q;
                sstart.push_back(q);
            }
            place[q] = static_cast<uint8_t>(q - first);
        }
    }
    sstart.push_back(start[levels + 1]);
    return static_cast<uint32_t>(sstart.size() - 1);
}

}  // namespace muto
