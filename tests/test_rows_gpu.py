"""The few-rows kernel (two to sixteen activation rows) against the decoded weights in float64, at the edges of its tiles, slices, passes and formats."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from tyloquant_b200 import QuantWeight, encode  # noqa: E402
from test_gemm_gpu import _status  # noqa: E402
from test_tile_gpu import _kernel_nodes, _kernels  # noqa: E402

# bits, group size, sub-scale bits; bound on the error over what the products add up to without cancellation.  Exact weights leave the float32 sums (some tens of roundings of 2^-24, and the two
# terms of the group sums, 2^-22, which uncentred widths subtract from sums a few times as large); width six takes one f16 rounding of the integers above 2^11, at most 2^-11 of each and
# 1.3e-4 in the mean square of many groups; a row of one group has the largest sub-scale in every place, where all odd codes beyond 16 are off by the whole 1 of 2048 to 4064.
EXACT, ROUNDED, ONE_GROUP = 5e-6, 2.0 ** -12, 2.0 ** -11
PROFILES = [((2, 16, 5), EXACT), ((3, 24, 5), EXACT), ((4, 24, 6), EXACT), ((4, 32, 6), EXACT), ((4, 48, 7), EXACT), ((5, 28, 7), EXACT), ((5, 32, 7), EXACT), ((5, 64, 6), EXACT),
            ((6, 24, 7), ROUNDED), ((6, 40, 7), ROUNDED), ((6, 64, 7), ROUNDED)]


def _x(m, k, seed, offset=0):
    gen = torch.Generator("cuda").manual_seed(seed)
    flat = torch.randn(m * k + offset, device="cuda", generator=gen).to(torch.bfloat16)
    return flat[offset:].view(m, k)


def _check(w, x, bound, **kw):
    got = w.matmul(x, out_dtype=torch.float32, **kw)
    ref = w.dequantize().double()
    err, size = got.double() - x.double() @ ref.T, (x.double().square() @ ref.T.square()).sqrt()
    assert (err.norm() / size.norm()).item() <= bound, (x.shape, ref.shape, (err.norm() / size.norm()).item())
    assert torch.equal(got, w.matmul(x, out_dtype=torch.float32, **kw))   # the same bits in every call
    return got


@pytest.mark.parametrize("profile,bound", PROFILES)
def test_scalar_weights(profile, bound):
    bits, gs, sub = profile
    # rows: less than a row-block, ragged, more than one per CTA; columns: one group and less, ragged, odd, more than a slice
    for n, k in ((1, gs), (17, gs - 3), (100, 1000), (333, 777), (2400, 1030), (48, 12000)):
        w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(n, k, bits, gs, sub, seed=n + k, device="cuda"))
        for m in (5, 8, 9, 16) if bits == 6 else (2, 3, 8, 9, 16):
            _check(w, _x(m, k, m), bound)
        w.free()
    assert _status() == 0


def test_many_row_blocks_per_cta():
    """More row-blocks than a CTA adds up at a time."""
    w = QuantWeight.from_blob("NINT3", encode.random_nint_blob(148 * 16 * 30 + 5, 200, 3, 24, 5, seed=3, device="cuda"))
    for m in (3, 16):
        _check(w, _x(m, 200, m), EXACT)
    w.free()


@pytest.mark.parametrize("dtype,entries,n_banks", [("NVQ3", 256, 1), ("NVQ3J", 256, 2), ("NVQ3J", 256, 4), ("NVQ3J-512", 512, 2), ("NVQ3J-512", 512, 4), ("NVQ3J-L", 1024, 1), ("NVQ3J-L", 1024, 2)])
def test_lattice_weights(dtype, entries, n_banks):
    for n, k in ((9, 20), (300, 2399), (640, 5120)):
        wt = np.random.default_rng(n).standard_normal((n, k), dtype=np.float32) * np.float32(0.02)
        banks = encode.d4_256_codebook()[None] if dtype == "NVQ3" else encode.synthetic_d4_banks(entries, n_banks, seed=9)
        w = QuantWeight.from_blob(dtype, encode.nvq_blob(encode.quantize_nvq3(wt, banks, jsc=dtype != "NVQ3", device="cuda")))
        for m in (2, 5, 8):
            x = _x(m, k, m)
            assert any("rows_mma_kernel" in name for name in _kernels(lambda: w.matmul(x)))
            _check(w, x, EXACT)
        w.free()
    assert _status() == 0


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_unaligned_rows(offset):
    """Activation rows that start on 2, 4 and 8 bytes."""
    for k, gs in ((1000, 24), (1004, 28), (1001, 24)):
        bits = 5 if gs == 28 else 4
        w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(130, k, bits, gs, 6, seed=k, device="cuda"))
        _check(w, _x(11, k, 1, offset), EXACT)
        w.free()


def test_gated_epilogue_and_non_finite_rows():
    n, k = 32 * 37, 1500
    w = QuantWeight.from_blob("NINT4", encode.random_nint_blob(n, k, 4, 24, 6, seed=8, device="cuda"))
    for m in (2, 7, 16):
        x = _x(m, k, m)
        p = (x.double() @ w.dequantize().double().T).view(m, n // 32, 2, 16)
        want = (p[:, :, 1] * p[:, :, 0] / (1 + torch.exp(-p[:, :, 0]))).reshape(m, n // 2)
        got = w.matmul_glu(x, out_dtype=torch.float32).double()
        assert ((got - want).norm() / want.norm()).item() <= 2e-5
        bad = x.clone()
        bad[0, 3], bad[1, k - 1] = float("inf"), float("nan")
        y = w.matmul(bad, out_dtype=torch.float32)
        assert not torch.isfinite(y[:2]).any() and torch.isfinite(y[2:]).all()
    assert _status() == 0
    w.free()


@pytest.mark.parametrize("dtype", ["NINT4", "NINT5", "NINT6", "NVQ3", "NVQ3J-512"])
def test_non_finite_values_make_all_outputs_of_their_row_nan(dtype):
    n, k = 200, 1500
    if dtype.startswith("NINT"):
        blob = encode.random_nint_blob(n, k, int(dtype[4]), 24, 6, seed=4, device="cuda")
    else:
        wt = np.random.default_rng(3).standard_normal((n, k), dtype=np.float32) * np.float32(0.02)
        banks = encode.d4_256_codebook()[None] if dtype == "NVQ3" else encode.synthetic_d4_banks(512, 2, seed=9)
        blob = encode.nvq_blob(encode.quantize_nvq3(wt, banks, jsc=dtype != "NVQ3", device="cuda"))
    w = QuantWeight.from_blob(dtype, blob)
    for m in (5, 8, 16) if dtype == "NINT6" else (2, 5, 8) if dtype.startswith("NVQ") else (2, 5, 8, 16):
        for at in (0, 700, k - 1):
            for value in (float("inf"), -float("inf"), float("nan")):
                x = _x(m, k, m)
                x[m - 1, at] = value
                y = w.matmul(x, out_dtype=torch.float32)
                assert torch.isnan(y[m - 1]).all() and torch.isfinite(y[:m - 1]).all(), (dtype, m, at, value)
    assert _status() == 0
    w.free()


WIDE = [((4, 48, 6), EXACT), ((5, 48, 6), EXACT), ((6, 32, 7), ROUNDED), ((6, 48, 7), ROUNDED), ((4, 44, 6), EXACT), ((5, 44, 6), EXACT), ((5, 60, 6), EXACT)]


@pytest.mark.parametrize("profile,bound", WIDE)
def test_wide_records(profile, bound):
    """Records that come into registers by halves, groups that two threads write; rows that start on 2, 4, 8 and 16 bytes."""
    bits, gs, sub = profile
    for n, k in ((1, gs), (100, 1000), (333, 777), (2400, 1032), (48, 12000)):
        w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(n, k, bits, gs, sub, seed=n + k, device="cuda"))
        for m, offset in ((5, 0), (8, 1), (9, 2), (15, 4), (16, 8)):
            _check(w, _x(m, k, m, offset), ONE_GROUP if bound == ROUNDED and n == 1 else bound)
        w.free()
    assert _status() == 0


class _FuncAttributes(ctypes.Structure):   # cudaFuncAttributes, its first members
    _fields_ = [("shared", ctypes.c_size_t), ("const", ctypes.c_size_t), ("local", ctypes.c_size_t), ("max_threads", ctypes.c_int), ("regs", ctypes.c_int),
                ("rest", ctypes.c_byte * 256)]


@pytest.mark.parametrize("profile", [p for p, _ in PROFILES + WIDE])
def test_the_next_products_activations_fit_beside_a_product(profile):
    """Each of an SM's four schedulers has 16,384 registers.  What a product's warps leave of them holds the CTA that writes the
    next product's activations, which is then there when the product ends; and no product keeps more than a few words of a
    thread in local memory."""
    bits, gs, sub = profile
    w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(64, 3 * gs, bits, gs, sub, seed=1, device="cuda"))
    rt = ctypes.CDLL("libcudart.so.12")
    for m in (8, 16):
        x, kernels = _x(m, 3 * gs, 1), {}
        for name, params in _kernel_nodes(lambda: w.matmul(x)):
            attr = _FuncAttributes()
            assert rt.cudaFuncGetAttributes(ctypes.byref(attr), ctypes.c_void_p(params.func)) == 0
            kernels["x" if "rows_x" in name else "product" if "rows_mma" in name else name] = (attr, params.block[0])
        (write, write_threads), (product, threads) = kernels["x"], kernels["product"]
        rounded = lambda regs: (regs + 7) // 8 * 8   # noqa: E731
        left = 16384 - rounded(product.regs) * threads // 4
        assert rounded(write.regs) * 32 * -(-write_threads // 128) <= left, (m, write.regs, write_threads, product.regs, threads)
        assert product.local <= 128, (m, product.local)
    w.free()


@pytest.mark.parametrize("profile,n,k,here", [((2, 16, 5), 57344, 4096, True), ((3, 24, 5), 100000, 1030, True), ((4, 24, 6), 57344, 2048, True), ((4, 24, 6), 57344, 4096, False),
                                              ((4, 24, 6), 128256, 768, False), ((5, 24, 7), 36864, 2048, True), ((5, 32, 7), 57344, 768, True), ((5, 32, 7), 57344, 2048, False),
                                              ((6, 24, 7), 57344, 768, True), ((6, 24, 7), 57344, 1536, False), ((5, 28, 7), 70000, 1536, True)])
def test_long_lists(profile, n, k, here):
    """Sixteen rows through many row-blocks, one to three passes of them, on the side of the line that is the faster one (148 SMs).
    Bound of the tile kernel: two f16 roundings, as its own tests have it."""
    bits, gs, sub = profile
    w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(n, k, bits, gs, sub, seed=n, device="cuda"))
    x = _x(16, k, 1)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert any("rows_mma_kernel" in name for name in _kernels(lambda: w.matmul(x))) == here
    _check(w, x, 3.6e-4 if not here else ROUNDED if bits == 6 else EXACT)
    w.free()
    assert _status() == 0
