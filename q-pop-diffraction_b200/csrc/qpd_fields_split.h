// How the layers of a stack are shared out among the blocks of the field preparation (qpd_fields.cu).  Plain C++, so
// that the split can be checked without a GPU.
#pragma once

#include <algorithm>

namespace qpd {

constexpr int kFieldsLayers = 32;  // layers of a chunk

// Chunks first .. first + chunks - 1 hold the crop; group g takes the `per` of them from first + g per on, and sums the
// ramp over the layers below its first chunk by itself.
struct FieldsSplit {
    long long first, chunks, per, groups;
};

// A film is cut into as many groups as it takes to have `blocks` blocks: the sum over the layers below is short beside
// an idle device.  A plane of many columns fills the device anyway and takes one group, which sums every layer once,
// except that a group per chunk is left where that sums no layer more than 1.5 times on average (two chunks from layer 0).
inline FieldsSplit fields_split(long long column_blocks, long long z0, long long nz, long long blocks) {
    FieldsSplit s;
    s.first = z0 / kFieldsLayers;
    s.chunks = (z0 + nz + kFieldsLayers - 1) / kFieldsLayers - s.first;
    // chunks summed by a group per chunk, against those of the stack
    const long long sums = s.chunks * s.first + s.chunks * (s.chunks + 1) / 2, stack = s.first + s.chunks;
    long long want = std::min(s.chunks, std::max<long long>(1, (blocks + column_blocks - 1) / column_blocks));
    if (2 * sums <= 3 * stack) want = s.chunks;
    s.per = (s.chunks + want - 1) / want;
    s.groups = (s.chunks + s.per - 1) / s.per;
    return s;
}

}  // namespace qpd
