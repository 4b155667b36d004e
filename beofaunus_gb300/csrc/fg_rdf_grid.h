// Blocks of the g(r) histogram kernel (host code without CUDA, so that it is
// tested as it is).
#pragma once
#include <algorithm>
#include <cstdint>

namespace fg {

constexpr int kRdfThreads = 128;
constexpr int kRdfTile = 128;        // j positions staged per pass

// Tiles of kRdfThreads x kRdfTile pairs of N particles spread over eight blocks
// per SM, and over more where a block's 32-bit counters could not hold all its
// pairs in one bin (from 3.3 million particles on 152 SMs).
inline int64_t rdf_blocks(int64_t N, int sms) {
    const int64_t nt = (N + kRdfThreads - 1) / kRdfThreads, tiles = nt * nt;
    const int64_t per_block = (int64_t)0xFFFFFFFF / (kRdfThreads * kRdfTile);
    return std::min(tiles, std::max((int64_t)8 * sms, (tiles + per_block - 1) / per_block));
}

}  // namespace fg
