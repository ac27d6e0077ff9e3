// Loading packed tensors: file streams -> device records on the GPU.
#pragma once
#include <memory>
#include <vector>

#include "common.h"
#include "cuda_util.h"
#include "nint_blayout.h"

namespace mfqb {

// Device memory of a tensor.  Mapping and unmapping 52 MB takes 0.7 to 5 ms, up to twice what loading it takes (1.5 ms with
// decoding and freeing), so the blocks of freed tensors are parked and taken again by tensors of about their size: at most
// kParkedBytes in kParkedBlocks of each device, given back when newer ones push them out, when an allocation of the library
// finds no room, or by mfqb_memory_trim.
//
// A block is parked after all work of its device has ended, so whatever stream takes it next may write at once.  What waits for
// that work is cudaFree, of a few bytes that every tensor has beside its block: where a stream is being captured
// (cudaStreamCaptureModeRelaxed, or by another thread) freeing is allowed, and synchronising the device would end the capture.
constexpr size_t kParkedBytes = 256u << 20;
constexpr int kParkedBlocks = 16;

struct TensorBuf {
    void* p = nullptr;
    size_t bytes = 0;   // asked for; the block may be larger
    TensorBuf() = default;
    TensorBuf(const TensorBuf&) = delete;
    TensorBuf& operator=(const TensorBuf&) = delete;
    TensorBuf(TensorBuf&& o) noexcept : p(o.p), bytes(o.bytes), fence_(o.fence_), block_(o.block_), device_(o.device_) { o.p = o.fence_ = nullptr; }
    void alloc(size_t n);   // on the current device
    void release();
    ~TensorBuf() { release(); }

private:
    void* fence_ = nullptr;   // freed before the block is parked
    size_t block_ = 0;
    int device_ = 0;
};
bool give_back_parked(int device);   // true where the device got memory back

// Device memory of one tensor in the byte-lane layout: records, anchors and row constants in one allocation.
struct PackedDev {
    TensorBuf mem;
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
