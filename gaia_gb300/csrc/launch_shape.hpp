// Host rules on the shape of a launch.
#pragma once
#include <algorithm>

namespace gaia {

constexpr int kWarp = 32;
constexpr int kMinBlock = 64;  // threads of the smallest block that a sweep runs

// About half as many threads, in whole warps, at least kMinBlock: every warp of a block owns a
// part of the staging area and runs full-warp shuffles.
inline int smaller_block(int B) { return std::max(kMinBlock, B / 2 / kWarp * kWarp); }

}  // namespace gaia
