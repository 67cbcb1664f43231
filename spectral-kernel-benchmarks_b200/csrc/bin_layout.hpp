// Sizes of the plans' bin arrays (row-transformed planes, [block][ky][kx][plane]).
#pragma once

#include <cstdint>

namespace skb {

// Blocks of 16 planes keep a CTA's pieces of one kx column keep * 16 values apart and
// on 128-byte lines whatever the plane count; the last block costs up to 15 planes
// (17 planes store 32).  An array of fewer than 16 planes is one block of just those:
// a whole block would take up to 16 times its size (1024^2, FP64, one plane: 134 MB
// for 8) and ran 1 % slower (geometric mean over 64^2 to 1024^2, both precisions).
// One block of 17 to 31 planes ran up to 4 % slower than two of 16.
constexpr int kBinBlockShift = 4;
constexpr std::uint64_t kBinBlock = std::uint64_t(1) << kBinBlockShift;

// Planes that an array for `planes` planes stores.
constexpr std::uint64_t stored_planes(std::uint64_t planes) {
    return planes < kBinBlock ? planes : (planes + kBinBlock - 1) / kBinBlock * kBinBlock;
}

// Bytes of an array for `planes` planes of ny rows with kx < keep.
constexpr std::uint64_t bin_array_bytes(std::uint64_t ny, std::uint64_t keep, std::uint64_t planes,
                                        std::uint64_t elementBytes) {
    return ny * keep * stored_planes(planes) * 2 * elementBytes;
}

}  // namespace skb
