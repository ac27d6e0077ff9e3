// Loading packed tensors: file streams -> device records on the GPU.
#pragma once
#include <memory>
#include <vector>

#include "common.h"
#include "cuda_util.h"
#include "nint_blayout.h"

namespace mfqb {

// Device memory of one tensor in the byte-lane layout: records, anchors and row constants in one allocation.
struct PackedDev {
    DevBuf mem;
    NintDevB d{};
    uint64_t bytes = 0;   // records + anchors + row constants
    void alloc(size_t extra = 0);               // geometry in d is set; `extra` more bytes at extra_at()
    void* extra_at() const { return static_cast<char*>(mem.p) + extra_off; }
    size_t extra_off = 0;
};

// Rows [row0, row0 + n) and groups [group0, ...) of a parsed tensor; every unit of `ope` file rows becomes `padded` device rows
// (expert records pad to whole row-blocks; a plain tensor is one unit).  `units`: file positions of the units, ascending.
struct LoadRows {
    int64_t row0, ope, padded;
    std::vector<int> units;
};

// Fills p (geometry and memory set) from the file streams and returns when the device holds the tensor.
void load_nint(const NintView& t, int64_t group0, const LoadRows& rows, int device, PackedDev& p);
void load_nvq(const HostNvq& t, const NvqStreams& s, int64_t row0, int64_t group0, int device, PackedDev& p);

// Geometry of a device tensor of n rows x k columns (n: device rows).
NintDevB nint_geometry(const NintView& t, int64_t n, int64_t k);

}  // namespace mfqb
