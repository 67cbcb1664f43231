// Column addressing shared by the grouped vertical GEMM kernels.
#pragma once

#include "vertical.hpp"

namespace skb {

// Element offset of plan column `col` (member * memberColumns + mode * fields
// + field) in a cell-addressed operand, with its partner (or -1) and
// conjugation.
__device__ __forceinline__ void bin_column(const BinBoundary& bb, int col, long long& base, long long& partner,
                                           bool& conj) {
    // Plan column = member * memberColumns + mode * fields + plan field.
    long long member = 0;
    int rest = col;
    if (bb.memberColumns > 0) {
        member = col / bb.memberColumns;
        rest = static_cast<int>(col - member * bb.memberColumns);
    }
    const int mode = rest / bb.fields;
    const int sub = rest - mode * bb.fields;
    const int field = bb.fieldMap != nullptr ? __ldg(bb.fieldMap + sub) : sub;
    const long long memberStride =
        bb.memberStride != 0 ? bb.memberStride : static_cast<long long>(bb.fields) * bb.zStride;
    const long long off = member * memberStride + static_cast<long long>(field) * bb.zStride;
    base = __ldg(bb.cell + mode) + off;
    const long long p = bb.partner != nullptr ? __ldg(bb.partner + mode) : -1;
    partner = p >= 0 ? p + off : -1;
    conj = bb.conj != nullptr && __ldg(bb.conj + mode) != 0;
}

}  // namespace skb
