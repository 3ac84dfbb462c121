// Row ranges of the budget network's weight gradients (host only).
#pragma once

#include <algorithm>
#include <cstddef>

namespace hrnn {

constexpr int kTileK = 16;  // rows a weight-gradient block stages at a time

// The row ranges of a batch of B: for the 256 x 256 layers sixteen of at least 64 rows
// (their 32 tiles times the ranges fill the device twice or three times), for the
// output layer 32 rows each.
struct Ranges {
    int per, per3 = 32;
    size_t n, n3;
    explicit Ranges(int B)
        : per(std::max(64, ((B + 15) / 16 + kTileK - 1) / kTileK * kTileK)),
          n((size_t)(B + per - 1) / per),
          n3((size_t)(B + 31) / 32) {}
};

// The most ranges a batch of up to B rows has: what a workspace made for B rows and kept
// for smaller batches needs room for.  Ranges(B).n does not grow with B (16 at 1024
// rows, 13 of 80 rows at 1025), but it is at most 16 and at most one per 64 rows.
struct MostRanges {
    size_t n, n3;
    explicit MostRanges(int B) : n(std::min<size_t>(16, (size_t)(B + 63) / 64)), n3((size_t)(B + 31) / 32) {}
};

}  // namespace hrnn
