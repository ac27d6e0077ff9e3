// Dense weight handles: blob -> device layout -> decode / multiply entry points.
#include <cuda_bf16.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

#include <climits>

#include "cuda_util.h"
#include "nint_blayout.h"
#include "load.h"
#include "nvq.h"
#include "nvq_blayout.h"
#include "rows_mma.h"
#include "tile_tc.h"

namespace mfqb {

int device_sm_count(int device) {
    static std::mutex mu;
    static int cache[64] = {0};
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= 64) fail(MFQB_ERR_ARG, "device index %d out of range", device);
    if (!cache[device]) {
        int v = 0;
        MFQB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device));
        cache[device] = v;
    }
    return cache[device];
}

static bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) (void)cudaGetLastError();
    return st != cudaStreamCaptureStatusNone;
}
static std::mutex g_scratch_mu;   // one lock for every pool: growth is rare
void GrowOnlyScratch::reserve(int device, size_t bytes, cudaStream_t stream, const char* what) {
    {
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        if (device >= 0 && device < 64 && dev_[device].bytes >= bytes) return;
    }
    if (!capturing(stream)) get(device, bytes, stream, what);
}
void* GrowOnlyScratch::get(int device, size_t bytes, cudaStream_t stream, const char* what, bool exact) {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (device < 0 || device >= 64) fail(MFQB_ERR_ARG, "device index %d out of range", device);
    PerDevice& d = dev_[device];
    if (d.bytes >= bytes) return d.p;
    if (capturing(stream))
        fail(MFQB_ERR_ARG,
             "%s needs %zu bytes of library scratch (it holds %zu) while the stream is being captured: "
             "run one call of this size outside the capture first",
             what, bytes, d.bytes);
    void* p = nullptr;
    const size_t want = exact ? bytes : bytes + bytes / 2;
    device_malloc(&p, want);
    MFQB_CUDA(cudaMemsetAsync(p, 0, want, stream));   // some users keep self-resetting counters in their block: they start at zero, in the call's own order
    d.p = p;   // the previous block stays allocated: earlier launches and captured graphs may still use it
    d.bytes = want;
    return p;
}

// Per device a status word that kernels set when a bounded wait runs out (mfqb_device_status).
struct DeviceStatus {
    std::mutex mu;
    int* host[64] = {nullptr};
    int* dev[64] = {nullptr};
};
static DeviceStatus g_status;

int* device_status_word(int device) {   // pinned, mapped: the host can read it without a sync
    std::lock_guard<std::mutex> lock(g_status.mu);
    if (!g_status.host[device]) {
        MFQB_CUDA(cudaHostAlloc((void**)&g_status.host[device], sizeof(int), cudaHostAllocMapped));
        *g_status.host[device] = 0;
        MFQB_CUDA(cudaHostGetDevicePointer((void**)&g_status.dev[device], g_status.host[device], 0));
    }
    return g_status.dev[device];
}

int device_status(int device) {
    std::lock_guard<std::mutex> lock(g_status.mu);
    return g_status.host[device] ? *static_cast<volatile int*>(g_status.host[device]) : 0;
}

}  // namespace mfqb

using namespace mfqb;

namespace mfqb {
void launch_nint_bl_dequant(const NintDevB& w, void* out, int out_dtype, cudaStream_t s);
void launch_bl_gemv(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int ldy, int device, cudaStream_t s, bool swiglu = false, bool glu = false);
bool nint_bl_supported(int bits, int gs);
size_t gemvs_fix_bytes(int device);
void launch_swiglu(const void* gate_up, int in_dtype, int rows, int f, void* hidden, cudaStream_t s);
void reserve_planes(const NintDevB& w, int device, cudaStream_t s);
void launch_bl_gemv_norm(const NintDevB& w, const float* h, const float* delta, const float* gamma, float eps, float* h_out, void* y, int y_dtype,
                         bool glu, int device, cudaStream_t s);
int g_moe_f16_from_x2 = 4;   // see mfqb_tune
void launch_bl_gemv_multi(const NintDevB* ws, void* const* ys, int count, const void* x, int y_dtype, int device, cudaStream_t s);
bool launch_bl_gemvs(const NintDevB& w, const void* x, int x_dtype, void* y, int y_dtype, int device, void* fix, int* error, cudaStream_t s);
}

// Which single-row kernel a plain NINT weight takes: 0 = by shape (default), 1 = always the ring
// kernel, 2 = always the streamed kernel (mfqb_tune("gemv1_kernel", v)).
static int g_gemv1_choice = 0;
static bool gemv1_use_streamed(const NintDevB& w) {
    if (g_gemv1_choice == 1) return false;
    if (g_gemv1_choice == 2) return true;
    (void)w;
    return false;   // measured on B200: the ring kernel is as fast or faster on every shape of the sweep
}

struct mfqb_weight {
    int family = 0, device = 0;
    mfqb_weight_info info{};
    NintDevB nint{};
    PackedDev dev;       // its extra memory: the streamed single-row kernel's partial rows of row-blocks shared by two CTAs, and their counters
    int* status = nullptr;   // the device's host-visible status word
    NvqDevicePtr nvq;
};

namespace mfqb {

void check_nint_supported(const NintView& t) {
    const int b = t.bits;
    if (!(b == 2 || b == 3 || b == 4 || b == 5 || b == 6 || b == 8))
        fail(MFQB_ERR_UNSUPPORTED, "NINT%d is not an executable code width (2,3,4,5,6,8)", b);
    if (!nint_bl_supported(b, t.gs)) fail(MFQB_ERR_UNSUPPORTED, "NINT%d with groupsize %d is outside the runtime catalog", b, t.gs);
}

const NintDevB& weight_device_layout(const mfqb_weight* w);
int weight_device_index(const mfqb_weight* w);

static mfqb_weight* make_nint_weight(const NintView& t, const SliceRange& r, int device) {
    check_nint_supported(t);
    auto w = std::make_unique<mfqb_weight>();
    DeviceGuard guard(device);
    w->family = MFQB_FAMILY_NINT;
    w->device = device;
    w->dev.d = nint_geometry(t, r.n, r.k);
    w->dev.alloc(gemvs_fix_bytes(device));
    MFQB_CUDA(cudaMemset(w->dev.extra_at(), 0, gemvs_fix_bytes(device)));
    load_nint(t, r.group0, LoadRows{r.row0, r.n, r.n, {0}}, device, w->dev);
    w->status = device_status_word(device);
    w->nint = w->dev.d;
    mfqb_weight_info& i = w->info;
    i.family = MFQB_FAMILY_NINT;
    i.bits = t.bits;
    i.groupsize = t.gs;
    i.sub_bits = t.sub_bits;
    i.n = r.n;
    i.k = r.k;
    i.device = device;
    i.jsc_banks = 0;
    i.payload_bytes = nint_payload_bytes(t, r.n, r.ng);
    i.device_bytes = w->dev.bytes;
    return w.release();
}

const NintDevB& weight_device_layout(const mfqb_weight* w) { return w->family == MFQB_FAMILY_NINT ? w->nint : nvq_device_layout(*w->nvq); }

// Rows from which the tile kernel is tried.
static int tile_from(const mfqb_weight* w) { return w->family == MFQB_FAMILY_NINT ? 5 : 2; }
static GrowOnlyScratch g_glu_rows;   // the products of gated rows that no kernel with the gate in its epilogue takes
constexpr const char* kGluRows = "mfqb_mul_mat_glu (gate and up products)";
// A call of m rows makes room for captured calls of fewer, which may take other kernels with scratch of their own: the integer
// one below tile_from rows, the few-rows kernel below the tile kernel.  (Every kernel's own block holds all that it takes.)
void reserve_fewer_rows(const mfqb_weight* w, int m, bool glu, cudaStream_t s) {
    const int from = tile_from(w);
    if (m < from) return;
    const NintDevB& dev = weight_device_layout(w);
    if (w->family == MFQB_FAMILY_NINT) reserve_planes(dev, w->device, s);
    reserve_rows(dev, w->device, s);
    if (glu) g_glu_rows.reserve(w->device, (size_t)(from - 1) * w->info.n * 4, s, kGluRows);
}
int weight_device_index(const mfqb_weight* w) { return w->device; }

}  // namespace mfqb

// prod [rows, n] float32 whose columns come in 16-wide blocks alternating gate and up -> y [rows, n / 2] = up * silu(gate)
__global__ void glu_blocks_kernel(const float* __restrict__ prod, int rows, int n, void* __restrict__ y, int y_dtype) {
    const int half = n >> 1;
    const size_t total = (size_t)rows * half;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / half;
        const int j = (int)(i % half), blk = j >> 4, lane = j & 15;
        const float g = prod[r * n + blk * 32 + lane], u = prod[r * n + blk * 32 + 16 + lane];
        const float v = u * g / (1.0f + expf(-g));
        if (y_dtype == MFQB_F32) static_cast<float*>(y)[i] = v;
        else static_cast<__nv_bfloat16*>(y)[i] = __float2bfloat16_rn(v);
    }
}

extern "C" {
#pragma GCC visibility push(default)

int mfqb_weight_from_blob_slice(const char* dtype, const void* blob, uint64_t nbytes, int axis, int64_t begin,
                                int64_t end, int device, mfqb_weight** out) {
    return guarded([&] {
        if (!dtype || !blob || !out) fail(MFQB_ERR_ARG, "mfqb_weight_from_blob: null argument");
        const std::string d(dtype);
        const bool whole = begin == 0 && end < 0;
        if (dtype_is_nint(d)) {
            const NintView t = parse_nint_view(blob, nbytes);
            if (d[4] - '0' != t.bits) fail(MFQB_ERR_FORMAT, "MFQ dtype/blob mismatch: %s contains NINT%d", dtype, t.bits);
            *out = make_nint_weight(t, whole ? SliceRange{0, t.n, 0, t.k, t.ng} : slice_nint(t, axis, begin, end), device);
        } else if (dtype_is_nvq(d)) {
            NvqStreams streams;
            const HostNvq t = parse_nvq_header(blob, nbytes, &streams);
            check_nvq_dtype(d, t);
            auto w = std::make_unique<mfqb_weight>();
            w->family = MFQB_FAMILY_NVQ;
            w->device = device;
            w->nvq = make_nvq_device(t, streams, whole ? SliceRange{0, t.n, 0, t.k, t.ng} : slice_nvq(t, axis, begin, end), device, &w->info);
            *out = w.release();
        } else {
            fail(MFQB_ERR_UNSUPPORTED, "dtype '%s' is outside the packed-weight execution path", dtype);
        }
    });
}

int mfqb_weight_from_blob(const char* dtype, const void* blob, uint64_t nbytes, int device, mfqb_weight** out) {
    return mfqb_weight_from_blob_slice(dtype, blob, nbytes, 0, 0, -1, device, out);
}

int mfqb_weight_info_get(const mfqb_weight* w, mfqb_weight_info* info) {
    return guarded([&] {
        if (!w || !info) fail(MFQB_ERR_ARG, "mfqb_weight_info_get: null argument");
        *info = w->info;
    });
}

int mfqb_weight_clone(const mfqb_weight* src, mfqb_weight** out) {
    return guarded([&] {
        if (!src || !out) fail(MFQB_ERR_ARG, "mfqb_weight_clone: null argument");
        if (src->family != MFQB_FAMILY_NINT) fail(MFQB_ERR_UNSUPPORTED, "mfqb_weight_clone: only scalar-quantised (NINT) weights");
        DeviceGuard guard(src->device);
        auto w = std::make_unique<mfqb_weight>();
        w->family = src->family;
        w->device = src->device;
        w->info = src->info;
        w->dev.d = src->dev.d;
        const size_t fix = src->dev.mem.bytes - src->dev.extra_off;
        w->dev.alloc(fix);
        MFQB_CUDA(cudaMemcpy(w->dev.mem.p, src->dev.mem.p, src->dev.extra_off, cudaMemcpyDeviceToDevice));
        MFQB_CUDA(cudaMemset(w->dev.extra_at(), 0, fix));
        w->status = src->status;
        w->nint = w->dev.d;
        *out = w.release();
    });
}

int mfqb_weight_free(mfqb_weight* w) {
    return guarded([&] {
        if (!w) return;
        DeviceGuard guard(w->device);
        delete w;
    });
}

int mfqb_dequant(const mfqb_weight* w, void* out, int out_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!w || !out) fail(MFQB_ERR_ARG, "mfqb_dequant: null argument");
        if (out_dtype != MFQB_F32 && out_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_dequant: bad output dtype");
        DeviceGuard guard(w->device);
        if (w->family == MFQB_FAMILY_NINT) launch_nint_bl_dequant(w->nint, out, out_dtype, stream);
        else nvq_dequant(*w->nvq, out, out_dtype, stream);
    });
}

int mfqb_mul_mat(const mfqb_weight* w, const void* x, int m, void* y, int y_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!w || !x || !y) fail(MFQB_ERR_ARG, "mfqb_mul_mat: null argument");
        if (m < 1) fail(MFQB_ERR_ARG, "mfqb_mul_mat: m must be >= 1, got %d", m);
        if (y_dtype != MFQB_F32 && y_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_mul_mat: bad output dtype");
        DeviceGuard guard(w->device);
        const int64_t n = w->info.n, k = w->info.k;
        const size_t ysz = y_dtype == MFQB_F32 ? 4 : 2;
        reserve_fewer_rows(w, m, false, stream);
        if (w->family == MFQB_FAMILY_NINT) {
            if (m >= 2 && launch_rows_product(w->nint, x, m, y, y_dtype, w->device, stream)) return;
            if (m >= 5 && launch_tile_product(w->nint, x, m, y, y_dtype, w->device, stream)) return;
            if (m == 1 && gemv1_use_streamed(w->nint) &&
                launch_bl_gemvs(w->nint, x, MFQB_BF16, y, y_dtype, w->device, w->dev.extra_at(), w->status, stream))
                return;
            constexpr int per_launch = 8;   // batch rows one GEMV launch covers
            for (int m0 = 0; m0 < m; m0 += per_launch) {
                const int mm = std::min(per_launch, m - m0);
                launch_bl_gemv(w->nint, static_cast<const char*>(x) + (size_t)m0 * k * 2, mm,
                                    static_cast<char*>(y) + (size_t)m0 * n * ysz, y_dtype, (int)n, w->device, stream);
            }
        } else {
            nvq_mul_mat(*w->nvq, x, m, y, y_dtype, stream);
        }
    });
}

int mfqb_mul_mat_swiglu(const mfqb_weight* w, const void* gate_up, int m, void* y, int y_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!w || !gate_up || !y) fail(MFQB_ERR_ARG, "mfqb_mul_mat_swiglu: null argument");
        if (m < 1) fail(MFQB_ERR_ARG, "mfqb_mul_mat_swiglu: m must be >= 1, got %d", m);
        if (y_dtype != MFQB_F32 && y_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_mul_mat_swiglu: bad output dtype");
        if (w->info.k > INT_MAX) fail(MFQB_ERR_ARG, "mfqb_mul_mat_swiglu: row length out of range");
        DeviceGuard guard(w->device);
        if (m == 1 && w->family == MFQB_FAMILY_NINT) {   // activation computed as the down projection loads its row
            launch_bl_gemv(w->nint, gate_up, 1, y, y_dtype, (int)w->info.n, w->device, stream, true);
            return;
        }
        static GrowOnlyScratch pool;
        void* act = pool.get(w->device, (size_t)m * w->info.k * 2, stream, "mfqb_mul_mat_swiglu (activation rows)");
        launch_swiglu(gate_up, MFQB_F32, m, (int)w->info.k, act, stream);
        const int rc = mfqb_mul_mat(w, act, m, y, y_dtype, stream);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
    });
}

int mfqb_mul_mat_rmsnorm(const mfqb_weight* w, const float* h, const float* delta, const float* gamma, float eps, float* h_out, void* y,
                         int y_dtype, int gated, mfqb_stream_t stream) {
    return guarded([&] {
        if (!w || !h || !gamma || !y) fail(MFQB_ERR_ARG, "mfqb_mul_mat_rmsnorm: null argument");
        if (y_dtype != MFQB_F32 && y_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_mul_mat_rmsnorm: bad output dtype");
        if (h_out == h) fail(MFQB_ERR_ARG, "mfqb_mul_mat_rmsnorm: h_out must not be h (other CTAs still read h)");
        if (w->family != MFQB_FAMILY_NINT || w->nint.table) fail(MFQB_ERR_UNSUPPORTED, "mfqb_mul_mat_rmsnorm: scalar-quantised (NINT) weights only");
        DeviceGuard guard(w->device);
        launch_bl_gemv_norm(w->nint, h, delta, gamma, eps, h_out, y, y_dtype, gated != 0, w->device, stream);
    });
}

int mfqb_mul_mat_glu(const mfqb_weight* w, const void* x, int m, void* y, int y_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!w || !x || !y) fail(MFQB_ERR_ARG, "mfqb_mul_mat_glu: null argument");
        if (m < 1) fail(MFQB_ERR_ARG, "mfqb_mul_mat_glu: m must be >= 1, got %d", m);
        if (y_dtype != MFQB_F32 && y_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_mul_mat_glu: bad output dtype");
        if (w->info.n % 32) fail(MFQB_ERR_ARG, "mfqb_mul_mat_glu: the weight needs whole (gate, up) pairs of 16-row blocks, n = %lld", (long long)w->info.n);
        DeviceGuard guard(w->device);
        if (m == 1 && w->family == MFQB_FAMILY_NINT) {   // activation applied where the kernel writes its rows
            launch_bl_gemv(w->nint, x, 1, y, y_dtype, (int)w->info.n, w->device, stream, false, true);
            return;
        }
        const NintDevB& dev = weight_device_layout(w);
        reserve_fewer_rows(w, m, true, stream);
        if (m >= 2 && launch_rows_product(dev, x, m, y, y_dtype, w->device, stream, true)) return;
        if (m >= tile_from(w) && launch_tile_product(dev, x, m, y, y_dtype, w->device, stream, true)) return;
        float* prod = static_cast<float*>(g_glu_rows.get(w->device, (size_t)m * w->info.n * 4, stream, kGluRows));
        const int rc = mfqb_mul_mat(w, x, m, prod, MFQB_F32, stream);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
        const size_t total = (size_t)m * (w->info.n / 2);
        glu_blocks_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, 148 * 8), 256, 0, stream>>>(prod, m, (int)w->info.n, y, y_dtype);
        MFQB_CUDA(cudaGetLastError());
    });
}

int mfqb_mul_mat_multi(const mfqb_weight* const* ws, int count, const void* x, void* const* ys, int y_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!ws || !x || !ys) fail(MFQB_ERR_ARG, "mfqb_mul_mat_multi: null argument");
        if (count < 1 || count > 8) fail(MFQB_ERR_ARG, "mfqb_mul_mat_multi: 1 to 8 weights per call, got %d", count);
        if (y_dtype != MFQB_F32 && y_dtype != MFQB_BF16) fail(MFQB_ERR_ARG, "mfqb_mul_mat_multi: bad output dtype");
        NintDevB devs[8];
        for (int i = 0; i < count; ++i) {
            if (!ws[i] || !ys[i]) fail(MFQB_ERR_ARG, "mfqb_mul_mat_multi: null weight or output");
            if (ws[i]->family != MFQB_FAMILY_NINT) fail(MFQB_ERR_UNSUPPORTED, "mfqb_mul_mat_multi: scalar-quantised (NINT) weights only");
            if (ws[i]->device != ws[0]->device) fail(MFQB_ERR_ARG, "mfqb_mul_mat_multi: weights live on different devices");
            devs[i] = ws[i]->nint;
        }
        DeviceGuard guard(ws[0]->device);
        launch_bl_gemv_multi(devs, ys, count, x, y_dtype, ws[0]->device, stream);
    });
}

// Copies `words` 32-bit words (activations in mapped pinned host memory -> device staging).
__global__ void host_to_device_words_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, size_t words) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) dst[i] = src[i];
}

// The same for up to 32 buffers in one launch (blockIdx.y picks the buffer): one trip over PCIe for all of them.
struct HostGatherTable {
    const uint32_t* src[32];
    uint32_t* dst[32];
    unsigned words[32];
};
__global__ void host_gather_words_kernel(const __grid_constant__ HostGatherTable t) {
    const uint32_t* src = t.src[blockIdx.y];
    uint32_t* dst = t.dst[blockIdx.y];
    const unsigned words = t.words[blockIdx.y];
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

// Device staging of the host-buffer entry point: per device one stream and two buffers that grow on
// demand and are then reused, so a call costs two copies, the kernel and one synchronisation.
namespace {
struct HostCallState {
    std::mutex mu[64];
    cudaStream_t stream[64] = {nullptr};
    cudaEvent_t done[64] = {nullptr};
    DevBuf x[64], y[64];
};
HostCallState g_host_call;
}  // namespace

// Host-buffer products: `count` weights of one device, each with its own x and y in host memory.
// Everything is enqueued on the device's staging stream and the call waits once, at the end.
static void mul_mat_host_impl(const mfqb_weight* const* ws, int count, const void* const* xs, int m, void* const* ys, int y_dtype) {
    const mfqb_weight* w0 = ws[0];
    if (w0->device < 0 || w0->device >= 64) fail(MFQB_ERR_ARG, "device index %d out of range", w0->device);
    const int device = w0->device;
    DeviceGuard guard(device);
    const size_t ysz = y_dtype == MFQB_F32 ? 4 : 2;
    size_t x_total = 0, y_total = 0;
    for (int i = 0; i < count; ++i) {
        if (!ws[i] || !xs[i] || !ys[i]) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host: null argument");
        if (ws[i]->device != device) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host_multi: weights live on different devices");
        x_total += ((size_t)m * ws[i]->info.k * 2 + 255) / 256 * 256;
        y_total += ((size_t)m * ws[i]->info.n * ysz + 255) / 256 * 256;
    }
    std::lock_guard<std::mutex> lock(g_host_call.mu[device]);   // per device: calls on different GPUs do not serialise
    cudaStream_t& s = g_host_call.stream[device];
    if (!s) MFQB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaEvent_t& ev = g_host_call.done[device];
    if (!ev) MFQB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    DevBuf& dx = g_host_call.x[device];
    DevBuf& dy = g_host_call.y[device];
    if (dx.bytes < x_total) dx.alloc(x_total + x_total / 2);   // nothing of this stream is in flight between calls
    size_t x_off = 0, y_off = 0;
    bool any_copy_back = false;
    // Pinned, mapped host buffers (cudaHostAlloc / cudaHostRegister, which is what a caller that
    // cares about latency passes): a small kernel pulls x over PCIe into the staging buffer and the
    // product kernel writes y straight into host memory -- no copy-engine round trips.  Pageable
    // buffers take the two cudaMemcpyAsync.
    std::vector<std::pair<size_t, int>> copy_back;   // (offset in dy, index)
    // First every activation buffer is staged (the mapped ones 32 per launch), then the products run
    // back to back: consecutive product kernels overlap through programmatic dependent launch, which
    // a staging kernel between them would break.
    std::vector<char*> xd(count);
    std::vector<void*> yd(count);
    HostGatherTable table{};
    int pending = 0;
    unsigned max_words = 0;
    auto flush = [&]() {
        if (!pending) return;
        const dim3 grid(std::max(1u, std::min((max_words + 255) / 256, 16u)), (unsigned)pending);
        host_gather_words_kernel<<<grid, 256, 0, s>>>(table);
        MFQB_CUDA(cudaGetLastError());
        pending = 0;
        max_words = 0;
    };
    for (int i = 0; i < count; ++i) {
        const size_t xb = (size_t)m * ws[i]->info.k * 2, yb = (size_t)m * ws[i]->info.n * ysz;
        void *x_map = nullptr, *y_map = nullptr;
        const bool mapped = (xb % 4 == 0) && xb / 4 <= 0xFFFFFFFFull && (reinterpret_cast<uintptr_t>(xs[i]) % 4 == 0) &&
                            cudaHostGetDevicePointer(&x_map, const_cast<void*>(xs[i]), 0) == cudaSuccess &&
                            cudaHostGetDevicePointer(&y_map, ys[i], 0) == cudaSuccess;
        if (!mapped) (void)cudaGetLastError();   // not an error: the buffers are simply pageable
        if (i > 0 && xs[i] == xs[i - 1] && ws[i]->info.k == ws[i - 1]->info.k) {   // the same host rows as the previous product: staged once
            xd[i] = xd[i - 1];
            if (!mapped) {
                if (!any_copy_back && dy.bytes < y_total) dy.alloc(y_total + y_total / 2);
                any_copy_back = true;
                copy_back.emplace_back(y_off, i);
            }
            yd[i] = mapped ? y_map : static_cast<void*>(static_cast<char*>(dy.p) + y_off);
            y_off += (yb + 255) / 256 * 256;
            continue;
        }
        xd[i] = static_cast<char*>(dx.p) + x_off;
        if (mapped) {
            table.src[pending] = static_cast<const uint32_t*>(x_map);
            table.dst[pending] = reinterpret_cast<uint32_t*>(xd[i]);
            table.words[pending] = (unsigned)(xb / 4);
            max_words = std::max(max_words, (unsigned)(xb / 4));
            if (++pending == 32) flush();
        } else {
            MFQB_CUDA(cudaMemcpyAsync(xd[i], xs[i], xb, cudaMemcpyHostToDevice, s));
            if (!any_copy_back && dy.bytes < y_total) dy.alloc(y_total + y_total / 2);
            any_copy_back = true;
            copy_back.emplace_back(y_off, i);
        }
        yd[i] = mapped ? y_map : static_cast<void*>(static_cast<char*>(dy.p) + y_off);
        x_off += (xb + 255) / 256 * 256;
        y_off += (yb + 255) / 256 * 256;
    }
    flush();
    // consecutive single-row products of one shape class on the same activations (q, k, v of a block) share a launch
    auto same_class = [](const mfqb_weight* a, const mfqb_weight* b) {
        return a->family == MFQB_FAMILY_NINT && b->family == MFQB_FAMILY_NINT && !a->nint.table && !b->nint.table && a->nint.bits == b->nint.bits &&
               a->nint.gs == b->nint.gs && a->nint.k == b->nint.k && a->nint.rec_words == b->nint.rec_words;
    };
    for (int i = 0; i < count;) {
        int run = 1;
        if (m == 1)
            while (i + run < count && run < 8 && xs[i + run] == xs[i] && same_class(ws[i], ws[i + run])) ++run;
        const int rc = run > 1 ? mfqb_mul_mat_multi(ws + i, run, xd[i], yd.data() + i, y_dtype, s) : mfqb_mul_mat(ws[i], xd[i], m, yd[i], y_dtype, s);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
        i += run;
    }
    for (const auto& cb : copy_back)
        MFQB_CUDA(cudaMemcpyAsync(ys[cb.second], static_cast<char*>(dy.p) + cb.first, (size_t)m * ws[cb.second]->info.n * ysz,
                                  cudaMemcpyDeviceToHost, s));
    // wait by polling an event: the answer comes back a few microseconds sooner than through a blocking synchronise
    MFQB_CUDA(cudaEventRecord(ev, s));
    for (;;) {
        const cudaError_t q = cudaEventQuery(ev);
        if (q == cudaSuccess) break;
        if (q != cudaErrorNotReady) MFQB_CUDA(q);
    }
}

int mfqb_mul_mat_host(const mfqb_weight* w, const void* x_host, int m, void* y_host, int y_dtype) {
    return guarded([&] {
        if (!w || !x_host || !y_host) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host: null argument");
        if (m < 1) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host: m must be >= 1");
        mul_mat_host_impl(&w, 1, &x_host, m, &y_host, y_dtype);
    });
}

int mfqb_mul_mat_host_multi(const mfqb_weight* const* ws, int count, const void* const* xs_host, int m, void* const* ys_host, int y_dtype) {
    return guarded([&] {
        if (!ws || !xs_host || !ys_host) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host_multi: null argument");
        if (count < 1 || m < 1) fail(MFQB_ERR_ARG, "mfqb_mul_mat_host_multi: count and m must be >= 1");
        mul_mat_host_impl(ws, count, xs_host, m, ys_host, y_dtype);
    });
}

int mfqb_tune(const char* key, int value) {
    return guarded([&] {
        if (!key) fail(MFQB_ERR_ARG, "mfqb_tune: null key");
        if (std::string(key) == "gemv1_kernel" && value >= 0 && value <= 2) g_gemv1_choice = value;
        else if (std::string(key) == "moe_f16_tiles_from_x2" && value >= 2 && value <= 1000000) g_moe_f16_from_x2 = value;
        else if (std::string(key) == "gemm_plan" && value >= 0 && value <= 1) {}   // had two tile plans to choose from; callers may still name it
        else fail(MFQB_ERR_ARG, "mfqb_tune: unknown key '%s' or value %d out of range", key, value);
    });
}

int mfqb_memory_trim(int device) {
    return guarded([&] {
        if (device < 0 || device >= 64) fail(MFQB_ERR_ARG, "mfqb_memory_trim: bad device index %d", device);
        DeviceGuard guard(device);
        give_back_parked(device);
    });
}

int mfqb_device_status(int device, int* status) {
    return guarded([&] {
        if (!status || device < 0 || device >= 64) fail(MFQB_ERR_ARG, "mfqb_device_status: bad argument");
        *status = device_status(device);
    });
}

int mfqb_selfcheck_layout(const char* dtype, const void* blob, uint64_t nbytes, uint64_t* mismatches) {
    return guarded([&] {
        if (!dtype || !blob || !mismatches) fail(MFQB_ERR_ARG, "mfqb_selfcheck_layout: null argument");
        const std::string d(dtype);
        if (dtype_is_nint(d)) {
            check_nint_supported(parse_nint_view(blob, nbytes));
            HostNint t = parse_nint(blob, nbytes);
            *mismatches = selfcheck_nint_bytes(t);
        } else if (dtype_is_nvq(d)) {
            *mismatches = selfcheck_nvq_bytes(parse_nvq(blob, nbytes));
        } else {
            fail(MFQB_ERR_UNSUPPORTED, "dtype '%s' is outside the packed-weight execution path", dtype);
        }
    });
}

#pragma GCC visibility pop
}  // extern "C"
