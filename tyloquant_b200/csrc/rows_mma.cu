// Host side of the few-rows kernel (rows_mma.cuh): which products take it, the split of the work, launches.
#include <algorithm>
#include <mutex>

#include "cuda_util.h"
#include "rows_mma.h"
#include "rows_mma_launch.cuh"

namespace mfqb {

int* device_status_word(int device);

// Whether every weight is an exact f16 integer: |q - mid| ss below 2^11 (rows_mma.cuh).
static bool rows_exact(const NintDevB& w) {
    if (w.bits > 5) return false;
    const int q = w.bits == 5 ? 16 : (1 << w.bits) - 1;
    return q * ((1 << std::min(w.sub_bits, 8)) - 1) <= 2048;
}
static bool rows_takes(const NintDevB& w, int m) {
    if (m < 2 || m > kRowsMax) return false;
    // A look-up per four weights and the table's bank conflicts: NVQ3 17408 x 5120 8 rows 21.1 us, 16 rows 26.0; tile kernel 23.6.
    if (w.table) return w.tile_terms == 1 && m <= 8;
    if (w.bits == 8) return false;   // a record would be 26 to 66 registers: NINT8-48 14336 x 4096 32 us for 8 rows, tile kernel 17
    // Two to four rows, and padded group sizes, have integer kernels (4e-6) or two-term weights as their other path: exact widths
    // only.  Widths up to four bits are not centred and would lose accuracy where they are rounded.
    if (m < 5 || w.gs % 8 || w.bits < 5) return rows_exact(w);
    return true;
}

struct RowsPlan {
    int tiles = 0, slices = 0, pass_rb = 0, passes = 0, rounds = 0;   // rounds: records of the busiest warp
    size_t x_bytes = 0, smem = 0;
};

// Split of the work: slices of K times tiles of row-blocks, one CTA each, at most one per SM.  More slices than one where shared
// memory does not hold all of K, or where rows are few; only as many as divide the SMs evenly: a grid that leaves one to four of
// them free costs the chain up to 3 us (NINT4 4096 x 4096, 16 rows: 148 tiles 9.0 us, 147 11.8, 144 10.8, 128 9.3).
static bool rows_plan(const NintDevB& w, int m, bool glu, int sms, RowsPlan& best) {
    const int nt = m <= 8 ? 1 : 2, unit = glu ? 2 : 1, units = w.nrb / unit;
    const size_t chunk = (size_t)rows_chunk_bytes(w.t8, nt), slot = (size_t)8 * nt * kRowsSlot * 4, ctx = w.table ? (size_t)w.table_words * 4 + 64 : 0;
    double best_cost = 0;
    for (int s = 1; s <= std::min(w.nchunks, kRowsSlices); ++s) {
        if (sms % s) continue;
        const int nch = (w.nchunks + s - 1) / s, tiles = std::min(units, sms / s);
        if (tiles < 1) break;
        const int r = (units + tiles - 1) / tiles * unit;   // row-blocks of the largest tile
        const size_t x = nch * chunk, fixed = x + ctx + kRowsWarps * slot;
        if (fixed + unit * slot > kRowsSmem || nch > kRowsChunks) continue;
        const int fit = std::min(kRowsPass, (int)((kRowsSmem - fixed) / slot) / unit * unit), passes = (r + fit - 1) / fit;
        if (s > 1 && passes > 1) continue;
        const int pass_rb = ((r + passes - 1) / passes + unit - 1) / unit * unit;
        // clocks: a record of every warp, the activations into shared memory, the ends of a pass, the sum over slices
        const int rounds = (pass_rb * nch + kRowsWarps - 1) / kRowsWarps;
        const double cost = (double)passes * (rounds * (nt == 1 ? 2600 : 3100) + 1500) + x / 50.0 + (s > 1 ? 3500 : 0);
        if (best.tiles == 0 || cost < best_cost) {
            best_cost = cost;
            best.tiles = tiles;
            best.slices = s;
            best.pass_rb = pass_rb;
            best.passes = passes;
            best.rounds = passes * rounds;
            best.x_bytes = x;
            best.smem = fixed + pass_rb * slot;
        }
    }
    return best.tiles > 0;
}

// Long lists of records, nine to sixteen rows: the tile kernel's steps cost less than the second activation tile here, the more bits
// the sooner, and passes over row-blocks pay for their ends.  us, 16 rows, here and on the tile kernel:
//   two and three bits at any length: NINT2-16 57344 x 4096 50.6 and 51.9, 128256 x 4096 102.7 and 103.1, NINT3-24 57344 x 4096 47.9
//   and 49.4, 128256 x 4096 96.3 and 96.8;
//   four bits, up to two passes: NINT4-24 45056 x 4096 (22 records a warp) 35.9 and 39.4, 57344 (30) 48.0 and 46.8, NINT4-32 57344
//   (22) 44.7 and 47.4; three: NINT4-24 128256 x 384 (18 octets of a group) 21.5 and 22.2, x 1536 (72) 46.3 and 41.8;
//   five and six bits, one pass: NINT5-24 36864 x 4096 (54 octets) 36.1 and 37.5, 45056 (66) 43.8 and 44.1, NINT6-24 36864 (54) 37.9
//   and 38.1, 45056 (66) 45.1 and 44.5, NINT6-48 28672 (42) 30.4 and 30.5, 45056 (66) 43.7 and 42.6;
//   two: NINT6-24 96000 x 384 (18) 18.7 and 19.4, x 768 (30) 26.6 and 24.5, NINT5-32 57344 x 384 (16) 16.4 and 15.9, x 4096 54.6 and 49.0.
// A padded group size doubles the tile kernel's steps (NINT5-28 28672 x 4096: 32.4 and 72.4).
static bool rows_long(const NintDevB& w, const RowsPlan& p) {
    if (w.bits <= 3 || w.gs % 8) return false;
    const int octets = p.rounds * w.t8;
    if (p.passes > (w.bits == 4 ? 2 : 1) && octets > 20) return true;
    return p.rounds > 25 || (w.bits > 4 && octets > (w.bits == 5 ? 66 : 60));
}

static void launch_rows_x(const RowsXArgs& a, int t8, const TileNorm* norm, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    const int lanes = 8 * rows_x_parts(t8), tokens = 128 / lanes;
    cfg.gridDim = norm ? dim3((unsigned)a.m) : dim3((unsigned)a.nchunks, (unsigned)((a.m + tokens - 1) / tokens));
    cfg.blockDim = dim3(norm ? 1024u : (unsigned)((std::min(a.m, tokens) * lanes + 31) / 32 * 32));
    if (norm) cfg.dynamicSmemBytes = (size_t)(a.k + 7) / 8 * 16;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto go = [&](auto t_c) {
        constexpr int T = decltype(t_c)::value;
        // the same split of the SM's memory as the kernels of the chain, see whole_carveout in tile_tc.cu
        static bool done[64] = {};
        int dev = 0;
        MFQB_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64 || !done[dev]) {
            MFQB_CUDA(cudaFuncSetAttribute(rows_x_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            MFQB_CUDA(cudaFuncSetAttribute(rows_norm_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            if (dev >= 0 && dev < 64) done[dev] = true;
        }
        if (norm) MFQB_CUDA(cudaLaunchKernelEx(&cfg, rows_norm_kernel<T>, a, *norm));
        else MFQB_CUDA(cudaLaunchKernelEx(&cfg, rows_x_kernel<T>, a));
    };
    switch (t8) {
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 3: go(std::integral_constant<int, 3>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 5: go(std::integral_constant<int, 5>{}); break;
        case 6: go(std::integral_constant<int, 6>{}); break;
        default: go(std::integral_constant<int, 8>{}); break;
    }
}

static GrowOnlyScratch g_frags, g_shared;
static size_t rows_frag_bytes(const NintDevB& w) { return (size_t)w.nchunks * rows_chunk_bytes(w.t8, 2); }
// Parts and arrival counts of any plan (slices > 1 have one pass).
static size_t rows_part_bytes(int device) { return (size_t)device_sm_count(device) * kRowsPass * 16 * kRowsMax * 4; }
static size_t rows_shared_bytes(int device) { return rows_part_bytes(device) + (size_t)device_sm_count(device) * 4; }
static const char *kRowsFrags = "mfqb_mul_mat (activation fragments)", *kRowsShared = "mfqb_mul_mat (parts of shared rows)";
void reserve_rows(const NintDevB& w, int device, cudaStream_t s) {
    if (!rows_takes(w, 2) && !rows_takes(w, 5)) return;
    g_frags.reserve(device, rows_frag_bytes(w), s, kRowsFrags);
    g_shared.reserve(device, rows_shared_bytes(device), s, kRowsShared);
}

bool launch_rows_product(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int device, cudaStream_t s, bool glu, const TileNorm* norm) {
    if (!rows_takes(w, m) || (norm && (w.k % 4 || w.k > 20480))) return false;   // the row as bf16 in a CTA's 48 KB
    RowsPlan p;
    if (!rows_plan(w, m, glu, device_sm_count(device), p)) return false;
    if (m > 8 && rows_long(w, p)) return false;
    const int nt = m <= 8 ? 1 : 2;
    RowsArgs a{};
    a.w = w;
    a.undo = 1048576.f;
    if (w.jsc) tile_lattice_scales(w, a.lut16, a.undo);
    a.y = y;
    a.m = m;
    a.ldy = glu ? w.n / 2 : w.n;
    a.y_dtype = y_dtype;
    a.glu = glu;
    a.tiles = p.tiles;
    a.slices = p.slices;
    a.pass_rb = p.pass_rb;
    a.x_bytes = (int)p.x_bytes;
    a.error = device_status_word(device);
    static std::mutex launches[64];   // the two launches belong together: another thread's on the same stream would take the scratch between them
    std::lock_guard<std::mutex> lock(launches[device]);
    // One call with this weight makes room for every smaller batch of it: fragments of 16 rows, parts of any plan.
    unsigned char* frags = static_cast<unsigned char*>(g_frags.get(device, rows_frag_bytes(w), s, kRowsFrags));
    unsigned char* shared = static_cast<unsigned char*>(g_shared.get(device, rows_shared_bytes(device), s, kRowsShared, true));
    a.x = frags;
    a.parts = reinterpret_cast<float*>(shared);
    a.counters = reinterpret_cast<unsigned*>(shared + rows_part_bytes(device));
    RowsXArgs xa{};
    xa.x = static_cast<const __nv_bfloat16*>(x);
    xa.m = m;
    xa.k = w.k;
    xa.gs = w.gs;
    xa.nt = nt;
    xa.nchunks = w.nchunks;
    xa.factor = w.table ? 1.f / 4096.f : rows_x_factor(w.bits);
    xa.out = frags;
    xa.counters = a.counters;
    xa.n_counters = p.slices > 1 ? p.tiles : 0;
    launch_rows_x(xa, w.t8, norm, s);
    cudaError_t e = cudaErrorNotSupported;
    switch (w.table ? 0 : w.bits) {
        case 0: e = launch_rows_nvq(a, p.smem, s); break;
        case 2: e = launch_rows_bits<2>(a, p.smem, s); break;
        case 3: e = launch_rows_bits<3>(a, p.smem, s); break;
        case 4: e = launch_rows_bits<4>(a, p.smem, s); break;
        case 5: e = launch_rows_bits<5>(a, p.smem, s); break;
        case 6: e = launch_rows_bits<6>(a, p.smem, s); break;
        default: break;
    }
    if (e != cudaSuccess)
        fail(MFQB_ERR_CUDA, "%s%d gs=%d few-rows product launch (m = %d, %zu bytes of shared memory): %s", w.table ? "NVQ index bits " : "NINT", w.table ? w.index_bits : w.bits, w.gs,
             m, p.smem, cudaGetErrorString(e));
    return true;
}

}  // namespace mfqb
