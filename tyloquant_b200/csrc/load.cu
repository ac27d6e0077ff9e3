// Loading packed tensors.  The file holds one LSB-first bitstream per field over the whole tensor; the streams are copied to
// the device as they are and re-laid there, a warp per (row-block, chunk) record, so the host neither unpacks nor packs
// anything (doing that took 5 ns per weight on one core: 280 ms for 14336 x 4096; the copy over PCIe is what is left).
//
// Worker threads share a load: each takes pieces of a few MB of rows, copies their stretches of the streams into pinned memory
// of its own, and queues the transfer and the re-layout kernel on a stream of its own, two pieces deep, so that the
// pageable-memory copies of several cores, PCIe and the kernels overlap.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "lane_unit.h"
#include "load.h"
#include "nvq_blayout.h"
#include "tile_tc.h"

namespace mfqb {

// ---- re-layout kernels ---------------------------------------------------------------------------------------------------
struct PackArgs {
    const uint32_t* stream[5];   // staged bytes, 16-byte aligned, readable a few words past their end
    uint32_t bit0[5];            // bit of the piece's first value in them
    int width[5];
    // device row r of the piece: unit r / padded, row r % padded of it; file row (of the piece) unit * ope + row when row < ope
    int rows, padded, ope, src_rows;
    int ng_file, group0, ng, gs, nchunks, wc, rec_words;
    int nvec_file, nsign_file, nvec, index_bits, bits;   // lattice: vectors and sign blocks per file row; scalar: code width
    uint32_t bankmap;
    uint32_t *items, *anchors;   // of the piece's first row
    uint4* rowc;
};

__device__ __forceinline__ uint32_t stream_bits(const uint32_t* s, uint32_t bit, int n) {   // n <= 32
    const uint32_t v = __funnelshift_r(__ldg(s + (bit >> 5)), __ldg(s + (bit >> 5) + 1), bit & 31);
    return n == 32 ? v : v & ((1u << n) - 1u);
}
// Where a file row of a stream begins (64 bits: a row-block can be as wide as an int says), for values counted inside the row.
struct RowBits {
    const uint32_t* p;
    uint32_t bit;
    __device__ __forceinline__ RowBits(const PackArgs& a, int k, int src, uint32_t per_row) {
        const uint64_t b = a.bit0[k] + (uint64_t)max(src, 0) * per_row * (uint32_t)a.width[k];
        p = a.stream[k] + (b >> 5);
        bit = (uint32_t)b & 31u;
    }
    __device__ __forceinline__ uint32_t get(uint64_t first_bit, int n) const {
        const uint64_t b = bit + first_bit;
        return stream_bits(p + (b >> 5), (uint32_t)b & 31u, n);
    }
};
__device__ __forceinline__ int pack_src_row(const PackArgs& a, int r) {   // file row of a device row, -1: padding
    if (r >= a.rows) return -1;
    const int u = r / a.padded, o = r - u * a.padded, src = u * a.ope + o;
    return o < a.ope && src < a.src_rows ? src : -1;
}

// Streams: 0 neuron scales, 1 neuron minima (16 bits), 2 sub-scales, 3 sub-minima, 4 codes.
template <int BITS, int T>
__global__ void __launch_bounds__(256) pack_nint_kernel(const __grid_constant__ PackArgs a) {
    using BU = ByteUnit<BITS>;
    constexpr int WC = BU::words_for(8 * T);
    const int lane = threadIdx.x & 31, q = lane >> 2, c = lane & 3, nrb = (a.rows + 15) / 16;
    for (long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); item < (long long)nrb * a.nchunks; item += (long long)gridDim.x * 8) {
        const int rb = (int)(item / a.nchunks), ch = (int)(item - (long long)rb * a.nchunks);
        const int src[2] = {pack_src_row(a, rb * 16 + q), pack_src_row(a, rb * 16 + q + 8)};
        const uint32_t per_row = (uint32_t)a.ng_file;
        const RowBits code[2] = {{a, 4, src[0], per_row * a.gs}, {a, 4, src[1], per_row * a.gs}};
        uint32_t w[WC];
#pragma unroll
        for (int i = 0; i < WC; ++i) w[i] = 0u;
#pragma unroll
        for (int r = 0; r < 8 * T; ++r) {   // register r: the coordinates of nint_reg_coord
            const int hi = r & 1, ft = r >> 2, f = ft / T, t = ft % T, slot = 8 * t + 4 * (c & 1);
            const int grp = ch * kChunkGroupsB + 4 * f + 2 * ((r >> 1) & 1) + (c >> 1);
            uint32_t v = 0u;
            if (src[hi] >= 0 && grp < a.ng && slot < a.gs) {
                const int wq = a.width[4], cnt = min(4, a.gs - slot);
                const uint32_t four = code[hi].get(((uint64_t)(a.group0 + grp) * a.gs + slot) * wq, 4 * wq);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < cnt) v |= ((four >> (i * wq)) & ((1u << BITS) - 1u)) << (8 * i);
            }
            BU::put(w, r, v);
        }
        uint32_t* rec = a.items + item * a.rec_words;
#pragma unroll
        for (int i = 0; i < WC; ++i) rec[i * 32 + lane] = w[i];
        uint32_t s0 = 0u, s1 = 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int grp = ch * kChunkGroupsB + 2 * c + (i & 1);
            if (src[i >> 1] < 0 || grp >= a.ng) continue;
            const uint64_t at = (uint64_t)(a.group0 + grp);
            s0 |= RowBits(a, 2, src[i >> 1], per_row).get(at * a.width[2], a.width[2]) << (8 * i);
            s1 |= RowBits(a, 3, src[i >> 1], per_row).get(at * a.width[3], a.width[3]) << (8 * i);
        }
        rec[WC * 32 + lane] = s0;
        rec[(WC + 1) * 32 + lane] = s1;
    }
}

// Streams: 0 anchors (16 bits), 1 sub-scales / states, 2 indices, 3 sign masks (7 bits).
template <int IB>
__global__ void __launch_bounds__(256) pack_nvq_kernel(const __grid_constant__ PackArgs a) {
    constexpr int FB = IB + 4, WC = (24 * FB + 31) / 32;
    const int lane = threadIdx.x & 31, q = lane >> 2, c = lane & 3, nrb = (a.rows + 15) / 16;
    for (long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); item < (long long)nrb * a.nchunks; item += (long long)gridDim.x * 8) {
        const int rb = (int)(item / a.nchunks), ch = (int)(item - (long long)rb * a.nchunks);
        const int src[2] = {pack_src_row(a, rb * 16 + q), pack_src_row(a, rb * 16 + q + 8)};
        const RowBits sub[2] = {{a, 1, src[0], (uint32_t)a.ng_file}, {a, 1, src[1], (uint32_t)a.ng_file}};
        const RowBits index[2] = {{a, 2, src[0], (uint32_t)a.nvec_file}, {a, 2, src[1], (uint32_t)a.nvec_file}};
        const RowBits sign[2] = {{a, 3, src[0], (uint32_t)a.nsign_file}, {a, 3, src[1], (uint32_t)a.nsign_file}};
        auto state = [&](int hi, int grp) {
            if (src[hi] < 0 || grp >= a.ng) return 0u;
            return sub[hi].get((uint64_t)(a.group0 + grp) * a.width[1], a.width[1]);
        };
        uint32_t w[WC + 1], sword = 0u;
#pragma unroll
        for (int i = 0; i <= WC; ++i) w[i] = 0u;
#pragma unroll
        for (int r = 0; r < 24; ++r) {
            const int hi = r & 1, ft = r >> 2, f = ft / 3, t = ft % 3;
            const int grp = ch * kChunkGroupsB + 4 * f + 2 * ((r >> 1) & 1) + (c >> 1), vec = grp * 6 + 2 * t + (c & 1);
            if (src[hi] < 0 || grp >= a.ng || vec >= a.nvec) continue;
            const uint32_t idx = index[hi].get((uint64_t)(a.group0 * 6 + vec) * IB, IB);
            const uint32_t mask = sign[hi].get((uint64_t)(a.group0 * 3 + (vec >> 1)) * 7u, 7);
            const uint32_t full = mask | ((uint32_t)(__popc(mask) & 1) << 7);   // the eighth sign is the parity of the seven stored ones
            const uint32_t field = ((full >> ((vec & 1) * 4)) & 15u) | (idx << 4);
            const int pos = r * FB, wi = pos >> 5, sh = pos & 31;
            w[wi] |= field << sh;
            if (sh + FB > 32) w[wi + 1] |= field >> (32 - sh);
            if (t == 0) {   // the codebook bank of pair i = f * 4 + a
                const int i = f * 4 + (r & 3);
                sword |= ((a.bankmap >> (2 * (state(hi, grp) & 15u))) & 3u) << (8 * (i >> 1) + 4 + 2 * (i & 1));
            }
        }
        uint32_t* rec = a.items + item * a.rec_words;
#pragma unroll
        for (int i = 0; i < WC; ++i) rec[i * 32 + lane] = w[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) sword |= (state(i >> 1, ch * kChunkGroupsB + 2 * c + (i & 1)) & 15u) << (8 * i);
        rec[WC * 32 + lane] = sword;
    }
}

// Anchors and row constants, a thread per device row.  minima = 0: lattice rows have none.
__global__ void pack_rows_kernel(const __grid_constant__ PackArgs a, int minima) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= (a.rows + 15) / 16 * 16) return;
    const int src = pack_src_row(a, r);
    uint32_t v = 0u;
    if (src >= 0) {
        v = stream_bits(a.stream[0], a.bit0[0] + (uint32_t)src * 16u, 16);
        if (minima) v |= stream_bits(a.stream[1], a.bit0[1] + (uint32_t)src * 16u, 16) << 16;
    }
    a.anchors[r] = v;
    a.rowc[r] = tile_row_const(v, a.bits);
}

// ---- worker pool ---------------------------------------------------------------------------------------------------------
namespace {
constexpr size_t kSlotBytes = 2u << 20;   // staging of one piece; large enough that a transfer outlasts its launch
constexpr int kLoadWorkers = 8;

struct Slot {
    char *host = nullptr, *dev = nullptr;
    cudaEvent_t done = nullptr;
    bool used = false;
    void alloc(size_t bytes) {   // all three, or none: a slot outlives the load that could not have it
        try {
            MFQB_CUDA(cudaHostAlloc((void**)&host, bytes, cudaHostAllocDefault));
            MFQB_CUDA(cudaMalloc((void**)&dev, bytes));
            MFQB_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
        } catch (...) {
            (void)cudaGetLastError();   // the launches of a later load look at it
            release();
            throw;
        }
    }
    void release() {
        if (host) cudaFreeHost(host);
        if (dev) cudaFree(dev);
        if (done) cudaEventDestroy(done);
        *this = Slot{};
    }
};
struct Worker {
    cudaStream_t stream = nullptr;
    Slot slot[2];
};
// Staging of one device, kept between loads (32 MB each of pinned and device memory at most, as far as loads have used
// it); a load holds the lock, so loads to one device come one after the other.
struct LoadPool {
    std::mutex mu;
    Worker worker[kLoadWorkers];
};
LoadPool g_load[64];

struct Piece {
    int64_t dev_row0, src_row0;
    int rows, padded, ope, src_rows;
};
struct StreamSpec {
    const uint8_t* base;
    int64_t per_row;
    int width;
};
size_t up256(size_t v) { return (v + 255) / 256 * 256; }
size_t stage_bytes(const std::vector<StreamSpec>& st, int64_t src_rows) {
    size_t n = 0;
    for (const auto& s : st) n += up256((size_t)((src_rows * s.per_row * s.width + 7) / 8) + 1 + 16);
    return n;
}

// Pieces of at most kSlotBytes of streams: several whole units, or row-blocks of one (at least one row-block).
std::vector<Piece> cut_pieces(const LoadRows& rows, const std::vector<StreamSpec>& st) {
    std::vector<Piece> out;
    auto fits = [&](int64_t r) { return stage_bytes(st, r) <= kSlotBytes; };
    int64_t per = rows.ope;   // rows of a piece inside a unit
    while (per > 16 && !fits(per)) per = std::max<int64_t>(16, (per / 2 + 15) / 16 * 16);
    for (size_t i = 0; i < rows.units.size();) {
        const int64_t dev0 = (int64_t)i * rows.padded, src0 = rows.row0 + rows.units[i] * rows.ope;
        if (per < rows.ope) {
            for (int64_t r = 0; r < rows.ope; r += per) {
                const int64_t src = std::min(per, rows.ope - r), dev = r + per < rows.ope ? per : rows.padded - r;
                out.push_back(Piece{dev0 + r, src0 + r, (int)dev, (int)dev, (int)src, (int)src});
            }
            ++i;
            continue;
        }
        size_t n = 1;
        while (i + n < rows.units.size() && rows.units[i + n] == rows.units[i] + (int)n && fits((int64_t)(n + 1) * rows.ope)) ++n;
        out.push_back(Piece{dev0, src0, (int)(n * rows.padded), (int)rows.padded, (int)rows.ope, (int)(n * rows.ope)});
        i += n;
    }
    return out;
}

// Runs the pieces; `launch` queues the re-layout of one piece (streams, bit offsets and rows of `a` are set).
void run_pieces(const std::vector<Piece>& pieces, const std::vector<StreamSpec>& st, const PackArgs& proto, const PackedDev& p, int device,
                const std::function<void(const PackArgs&, cudaStream_t)>& launch) {
    if (device < 0 || device >= 64) fail(MFQB_ERR_ARG, "device index %d out of range", device);
    LoadPool& pool = g_load[device];
    std::lock_guard<std::mutex> lock(pool.mu);
    size_t need = 0;
    for (const Piece& pc : pieces) need = std::max(need, stage_bytes(st, pc.src_rows));
    const bool big = need > kSlotBytes;   // a row-block of a very wide tensor: staging of this load only
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    const int workers = big ? 1 : (int)std::min<size_t>(std::min(kLoadWorkers, hw), pieces.size());
    Slot big_slot;
    std::atomic<size_t> next{0};
    std::atomic<bool> stop{false};
    std::mutex err_mu;
    std::exception_ptr err;
    auto work = [&](int wi) {
        Worker& w = pool.worker[wi];
        try {
            MFQB_CUDA(cudaSetDevice(device));
            if (!w.stream) MFQB_CUDA(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
            for (int turn = 0; !stop; ++turn) {
                const size_t i = next.fetch_add(1);
                if (i >= pieces.size()) break;
                const Piece& pc = pieces[i];
                Slot& sl = big ? big_slot : w.slot[turn & 1];
                if (!sl.host) sl.alloc(big ? need : kSlotBytes);
                if (sl.used) MFQB_CUDA(cudaEventSynchronize(sl.done));
                PackArgs a = proto;
                size_t off = 0;
                for (size_t k = 0; k < st.size(); ++k) {
                    const uint64_t bit = (uint64_t)pc.src_row0 * st[k].per_row * st[k].width, end = bit + (uint64_t)pc.src_rows * st[k].per_row * st[k].width;
                    const size_t b0 = bit / 8, n = (size_t)((end + 7) / 8 - b0);
                    memcpy(sl.host + off, st[k].base + b0, n);
                    a.stream[k] = reinterpret_cast<const uint32_t*>(sl.dev + off);
                    a.bit0[k] = (uint32_t)(bit & 7);
                    a.width[k] = st[k].width;
                    off += up256(n + 16);
                }
                a.rows = pc.rows;
                a.padded = pc.padded;
                a.ope = pc.ope;
                a.src_rows = pc.src_rows;
                a.items = const_cast<uint32_t*>(p.d.items) + (size_t)(pc.dev_row0 / 16) * p.d.nchunks * p.d.rec_words;
                a.anchors = const_cast<uint32_t*>(p.d.anchors) + pc.dev_row0;
                a.rowc = const_cast<uint4*>(p.d.rowc) + pc.dev_row0;
                MFQB_CUDA(cudaMemcpyAsync(sl.dev, sl.host, off, cudaMemcpyHostToDevice, w.stream));
                launch(a, w.stream);
                MFQB_CUDA(cudaGetLastError());
                MFQB_CUDA(cudaEventRecord(sl.done, w.stream));
                sl.used = true;
            }
        } catch (...) {
            stop = true;
            std::lock_guard<std::mutex> g(err_mu);
            if (!err) err = std::current_exception();
        }
        if (w.stream && cudaStreamSynchronize(w.stream) != cudaSuccess) {
            std::lock_guard<std::mutex> g(err_mu);
            if (!err) err = std::make_exception_ptr(Error(MFQB_ERR_CUDA, std::string("loading a tensor: ") + cudaGetErrorString(cudaGetLastError())));
        }
    };
    std::vector<std::thread> threads;
    try {
        for (int i = 1; i < workers; ++i) threads.emplace_back(work, i);
    } catch (const std::system_error&) {   // no more threads to be had: the ones there are do the work
    }
    work(0);
    for (auto& t : threads) t.join();
    big_slot.release();
    for (auto& w : pool.worker) w.slot[0].used = w.slot[1].used = false;   // all streams are idle
    if (err) std::rethrow_exception(err);
}

template <int BITS>
void launch_pack_nint(const PackArgs& a, int t8, unsigned grid, cudaStream_t s) {
    auto go = [&](auto t) {
        constexpr int T = decltype(t)::value;
        if constexpr (nint_bl_in_catalog(BITS, T)) pack_nint_kernel<BITS, T><<<grid, 256, 0, s>>>(a);
    };
    switch (t8) {
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 3: go(std::integral_constant<int, 3>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 5: go(std::integral_constant<int, 5>{}); break;
        case 6: go(std::integral_constant<int, 6>{}); break;
        case 8: go(std::integral_constant<int, 8>{}); break;
    }
}
unsigned pack_grid(const PackArgs& a) { return (unsigned)std::min<long long>(((long long)(a.rows + 15) / 16 * a.nchunks + 7) / 8, 148 * 8); }
}  // namespace

NintDevB nint_geometry(const NintView& t, int64_t n, int64_t k) {
    NintDevB d{};
    d.n = (int)n;
    d.k = (int)k;
    d.ng = (int)((k + t.gs - 1) / t.gs);
    d.bits = t.bits;
    d.gs = t.gs;
    d.sub_bits = t.sub_bits;
    d.t8 = (t.gs + 7) / 8;
    d.nrb = (d.n + 15) / 16;
    d.nchunks = (d.ng + kChunkGroupsB - 1) / kChunkGroupsB;
    d.wc = byte_unit_words(d.bits, 8 * d.t8);
    d.rec_words = (d.wc + 2) * 32;
    d.tile_terms = t.gs % 8 ? 2 : 1;
    return d;
}

namespace {
struct Parked {
    void* p;
    size_t bytes;
};
struct ParkedList {   // oldest first
    std::mutex mu;
    std::vector<Parked> blocks;
};
ParkedList& parked(int device) {
    static ParkedList* lists = new ParkedList[64];   // outlives tensors that are freed while the process ends
    return lists[device];
}
}  // namespace

void TensorBuf::alloc(size_t n) {
    release();
    bytes = n;
    if (!n) return;
    MFQB_CUDA(cudaGetDevice(&device_));
    if (device_ >= 64) fail(MFQB_ERR_ARG, "device index %d out of range", device_);
    device_malloc(&fence_, 256);
    {
        ParkedList& l = parked(device_);
        std::lock_guard<std::mutex> lock(l.mu);
        auto best = l.blocks.end();   // the smallest that fits and wastes no more than an eighth
        for (auto it = l.blocks.begin(); it != l.blocks.end(); ++it)
            if (it->bytes >= n && it->bytes - n <= n / 8 && (best == l.blocks.end() || it->bytes < best->bytes)) best = it;
        if (best != l.blocks.end()) {
            p = best->p;
            block_ = best->bytes;
            l.blocks.erase(best);
            return;
        }
    }
    device_malloc(&p, n);
    block_ = n;
}

void TensorBuf::release() {
    bytes = 0;
    if (!p && !fence_) return;
    void *const mem = p, *const fence = fence_;
    p = fence_ = nullptr;
    int prev = device_;
    cudaGetDevice(&prev);
    if (prev != device_) cudaSetDevice(device_);
    const bool idle = cudaFree(fence) == cudaSuccess;   // waits for the device, see above
    std::vector<Parked> out;
    if (idle && mem && block_ <= kParkedBytes) {
        ParkedList& l = parked(device_);
        std::lock_guard<std::mutex> lock(l.mu);
        l.blocks.push_back(Parked{mem, block_});
        size_t total = 0;
        for (const Parked& b : l.blocks) total += b.bytes;
        while (total > kParkedBytes || l.blocks.size() > kParkedBlocks) {
            total -= l.blocks.front().bytes;
            out.push_back(l.blocks.front());
            l.blocks.erase(l.blocks.begin());
        }
    } else if (mem) {
        out.push_back(Parked{mem, block_});
    }
    for (const Parked& b : out) cudaFree(b.p);
    if (prev != device_) cudaSetDevice(prev);
}

bool give_back_parked(int device) {
    if (device < 0 || device >= 64) return false;
    std::vector<Parked> out;
    {
        ParkedList& l = parked(device);
        std::lock_guard<std::mutex> lock(l.mu);
        out.swap(l.blocks);
    }
    for (const Parked& b : out) cudaFree(b.p);
    return !out.empty();
}

void device_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    int device = -1;
    if (e == cudaErrorMemoryAllocation && cudaGetLastError() == e && cudaGetDevice(&device) == cudaSuccess && give_back_parked(device))
        e = cudaMalloc(p, bytes);
    MFQB_CUDA(e);
}

void PackedDev::alloc(size_t extra) {
    const size_t items = up256((size_t)d.nrb * d.nchunks * d.rec_words * 4), anchors = up256((size_t)d.nrb * 16 * 4), rowc = (size_t)d.nrb * 16 * sizeof(uint4);
    extra_off = items + anchors + up256(rowc);
    mem.alloc(extra_off + extra);
    d.items = static_cast<const uint32_t*>(mem.p);
    d.anchors = reinterpret_cast<const uint32_t*>(static_cast<char*>(mem.p) + items);
    d.rowc = reinterpret_cast<const uint4*>(static_cast<char*>(mem.p) + items + anchors);
    bytes = (uint64_t)d.nrb * d.nchunks * d.rec_words * 4 + (uint64_t)d.nrb * 16 * (4 + sizeof(uint4));
}

void load_nint(const NintView& t, int64_t group0, const LoadRows& rows, int device, PackedDev& p) {
    const std::vector<StreamSpec> st = {{t.ns, 1, 16}, {t.nm, 1, 16}, {t.ss, t.ng, t.sub_width}, {t.sm, t.ng, t.sub_width}, {t.q, t.ng * t.gs, t.q_width}};
    PackArgs a{};
    a.ng_file = (int)t.ng;
    a.group0 = (int)group0;
    a.ng = p.d.ng;
    a.gs = t.gs;
    a.nchunks = p.d.nchunks;
    a.wc = p.d.wc;
    a.rec_words = p.d.rec_words;
    a.bits = t.bits;
    const int t8 = p.d.t8;
    run_pieces(cut_pieces(rows, st), st, a, p, device, [t8](const PackArgs& b, cudaStream_t s) {
        pack_rows_kernel<<<(b.rows + 15 + 255) / 256, 256, 0, s>>>(b, 1);
        switch (b.bits) {
            case 2: launch_pack_nint<2>(b, t8, pack_grid(b), s); break;
            case 3: launch_pack_nint<3>(b, t8, pack_grid(b), s); break;
            case 4: launch_pack_nint<4>(b, t8, pack_grid(b), s); break;
            case 5: launch_pack_nint<5>(b, t8, pack_grid(b), s); break;
            case 6: launch_pack_nint<6>(b, t8, pack_grid(b), s); break;
            default: launch_pack_nint<8>(b, t8, pack_grid(b), s); break;
        }
    });
}

void load_nvq(const HostNvq& t, const NvqStreams& sv, int64_t row0, int64_t group0, int device, PackedDev& p) {
    const std::vector<StreamSpec> st = {{sv.anchors, 1, 16}, {sv.sub, t.ng, t.sub_bits}, {sv.idx, t.nvec, t.index_bits}, {sv.signs, t.nsign, 7}};
    PackArgs a{};
    a.ng_file = (int)t.ng;
    a.group0 = (int)group0;
    a.ng = p.d.ng;
    a.gs = 24;
    a.nchunks = p.d.nchunks;
    a.wc = p.d.wc;
    a.rec_words = p.d.rec_words;
    a.nvec_file = (int)t.nvec;
    a.nsign_file = (int)t.nsign;
    a.nvec = (p.d.k + 3) / 4;
    a.index_bits = t.index_bits;
    a.bankmap = p.d.bankmap;
    const LoadRows rows{row0, p.d.n, p.d.n, {0}};
    run_pieces(cut_pieces(rows, st), st, a, p, device, [](const PackArgs& b, cudaStream_t s) {
        pack_rows_kernel<<<(b.rows + 15 + 255) / 256, 256, 0, s>>>(b, 0);
        switch (b.index_bits) {
            case 8: pack_nvq_kernel<8><<<pack_grid(b), 256, 0, s>>>(b); break;
            case 9: pack_nvq_kernel<9><<<pack_grid(b), 256, 0, s>>>(b); break;
            default: pack_nvq_kernel<10><<<pack_grid(b), 256, 0, s>>>(b); break;
        }
    });
}

}  // namespace mfqb
