"""Edges of the tensor-memory tile kernel behind batched products: token tiles, row tiles, shared tiles, both f16 forms of
lattice weights."""

import ctypes
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import mfq_oracle as O  # noqa: E402
from tyloquant_b200 import QuantWeight, encode  # noqa: E402
from test_gemm_gpu import _status  # noqa: E402
from test_nint_gpu import bf16_tensor, REL_L2  # noqa: E402

SHAPES = [(1, 24), (127, 200), (129, 1001), (272, 4104), (1000, 776)]   # rows around 16 and 128, one chunk to many, ragged columns
TOKENS = [5, 16, 17, 33, 128, 129, 255, 257, 520]


@pytest.mark.parametrize("profile", [(2, 16, 5), (3, 24, 5), (4, 24, 6), (4, 48, 6), (5, 28, 7), (6, 24, 7), (8, 22, 7), (8, 64, 7)])
def test_scalar_weights(profile):
    bits, gs, sb = profile
    for n, k in SHAPES:
        blob = encode.random_nint_blob(n, k, bits, gs, sb, seed=n + k + gs, device="cuda")
        ref = O.dequant_nint(O.unpack_nint(blob))
        w = QuantWeight.from_blob(f"NINT{bits}", blob)
        for m in TOKENS:
            x = encode.bf16_round(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32))
            x[0] *= np.float32(2.0 ** 100)   # every row has its own scale
            x[-1] *= np.float32(2.0 ** -66)
            y = w.matmul(bf16_tensor(x), out_dtype=torch.float32).cpu().numpy()
            assert _status() == 0
            # against what the products add up to without cancellation (a single output can cancel to nearly nothing)
            err = y.astype(np.float64) - x.astype(np.float64) @ ref.astype(np.float64).T
            size = np.sqrt(np.square(x, dtype=np.float64) @ np.square(ref, dtype=np.float64).T)
            for rows in (slice(0, 1), slice(1, m - 1), slice(m - 1, m)):
                assert np.linalg.norm(err[rows]) <= REL_L2 * np.linalg.norm(size[rows]), (profile, n, k, m, rows)
        w.free()


@pytest.mark.parametrize("form", ["plain", "joint, exact scales", "joint, two terms"])
def test_lattice_weights(form):
    jsc = form != "plain"
    banks = encode.synthetic_d4_banks(512, 2, seed=5) if jsc else O.d4_256_codebook()[None]
    for n, k in SHAPES:
        wt = encode.bf16_round(np.random.default_rng(n + k).standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
        blob = encode.nvq_blob(encode.quantize_nvq3(wt, banks, jsc=jsc, device="cuda"))
        if form.endswith("two terms"):   # state scales with eleven significant bits: their products with the codes are no f16 numbers
            at = blob.index(bytes([1, 2, 16, 1]), 36) + 4   # the metadata header: version, banks, states, mode, then the scales
            lut = (np.frombuffer(blob[at:at + 32], dtype="<f2").astype(np.float32) * np.float32(1.2373)).astype("<f2")
            blob = blob[:at] + lut.tobytes() + blob[at + 32:]
        ref = O.dequant_nvq(O.unpack_nvq(blob))
        w = QuantWeight.from_blob("NVQ3J-512" if jsc else "NVQ3", blob)
        for m in [2, 3] + TOKENS:
            x = encode.bf16_round(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32))
            y = w.matmul(bf16_tensor(x), out_dtype=torch.float32).cpu().numpy()
            assert _status() == 0
            err = y.astype(np.float64) - x.astype(np.float64) @ ref.astype(np.float64).T
            size = np.sqrt(np.square(x, dtype=np.float64) @ np.square(ref, dtype=np.float64).T)
            assert np.linalg.norm(err) <= 1e-5 * np.linalg.norm(size), (form, n, k, m)   # exact weights and activations: float32 sums
        w.free()


def test_shared_tiles_are_left_clean():
    """Tiles that several CTAs share are summed in a buffer that has to be zero again after every call, whatever the shapes."""
    ws = {}
    for n, k in ((200, 4200), (4096, 1536), (512, 9000)):
        blob = encode.random_nint_blob(n, k, 4, 24, 6, seed=n, device="cuda")
        ws[n] = (QuantWeight.from_blob("NINT4", blob), k, torch.from_numpy(O.dequant_nint(O.unpack_nint(blob))).cuda())
    gen = torch.Generator("cuda").manual_seed(1)
    for i in range(30):
        n = (200, 4096, 512)[i % 3]
        w, k, ref = ws[n]
        x = torch.randn((7, 300, 21, 130)[i % 4], k, device="cuda", generator=gen).to(torch.bfloat16)
        y_ref = x.double() @ ref.double().T
        assert ((w.matmul(x, out_dtype=torch.float32).double() - y_ref).norm() / y_ref.norm()).item() <= REL_L2, i
    assert _status() == 0


@pytest.mark.parametrize("n,k", [(32, 24), (160, 1000), (4128, 2600)])
def test_gated_epilogue(n, k):
    """Whole and shared tiles, the last row tile short of 128 rows."""
    blob = encode.random_nint_blob(n, k, 6, 24, 7, seed=n, device="cuda")
    w = QuantWeight.from_blob("NINT6", blob)
    ref = torch.from_numpy(O.dequant_nint(O.unpack_nint(blob))).cuda().double().reshape(n // 32, 2, 16, k)
    gen = torch.Generator("cuda").manual_seed(2)
    for m in (5, 16, 17, 130, 300):
        x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
        g, u = (torch.einsum("mk,brk->mbr", x.double(), ref[:, i]).reshape(m, -1) for i in range(2))
        want = u * g / (1 + torch.exp(-g))
        for dtype, bound in ((torch.float32, 2 * REL_L2), (torch.bfloat16, 4e-3)):
            got = w.matmul_glu(x, out_dtype=dtype).double()
            assert ((got - want).norm() / want.norm()).item() <= bound, (n, m, dtype)
    assert _status() == 0


@pytest.mark.parametrize("m", [65535, 65536, 70000])
def test_more_rows_than_a_grid_dimension(m):
    n, k = 40, 72
    wt = np.random.default_rng(1).standard_normal((n, k)).astype(np.float32) * np.float32(0.02)
    for dtype, blob, bound in (("NINT4", encode.random_nint_blob(n, k, 4, 24, 6, seed=3, device="cuda"), REL_L2),
                               ("NVQ3", encode.nvq_blob(encode.quantize_nvq3(wt, O.d4_256_codebook()[None], jsc=False, device="cuda")), 1e-5)):
        w = QuantWeight.from_blob(dtype, blob)
        x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(m)).to(torch.bfloat16)
        want = x.double() @ w.dequantize().double().T
        got = w.matmul(x, out_dtype=torch.float32).double()
        assert ((got - want).norm() / want.norm()).item() <= bound, dtype
        assert ((got[-64:] - want[-64:]).norm() / want[-64:].norm()).item() <= bound, dtype
        w.free()
    assert _status() == 0


# Shared tiles: two parts and whole tiles between them, one part of one tile per CTA, three parts, more parts than are added at once
SHARED = [(14336, 4096, 4, 32, 6, 512), (4096, 14336, 6, 24, 7, 16), (5000, 2888, 4, 24, 6, 77), (520, 9000, 3, 24, 5, 33), (100, 24000, 2, 16, 5, 16),
          (100, 24000, 2, 16, 5, 250), (300, 14336, 8, 48, 7, 8)]


@pytest.mark.parametrize("n,k,bits,gs,sb,m", SHARED)
def test_shared_tiles_have_the_same_bits_in_every_call(n, k, bits, gs, sb, m):
    w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(n, k, bits, gs, sb, seed=n, device="cuda"))
    other = QuantWeight.from_blob("NINT4", encode.random_nint_blob(700, 3000, 4, 24, 6, seed=1, device="cuda"))
    gen = torch.Generator("cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
    xo = torch.randn(50, 3000, device="cuda", generator=gen).to(torch.bfloat16)
    first = w.matmul(x, out_dtype=torch.float32)
    want = x.double() @ w.dequantize().double().T
    assert ((first.double() - want).norm() / want.norm()).item() <= REL_L2
    for _ in range(20):
        other.matmul(xo)
        assert torch.equal(first, w.matmul(x, out_dtype=torch.float32))
    if n % 32 == 0:
        glu = w.matmul_glu(x, out_dtype=torch.float32)
        for _ in range(5):
            assert torch.equal(glu, w.matmul_glu(x, out_dtype=torch.float32))
    assert _status() == 0


@pytest.mark.parametrize("bits,n,k,m,grid", [(2, 5000, 2888, 20, 120), (2, 5000, 2888, 512, 80), (4, 4960, 2888, 40, 117), (8, 5120, 2900, 128, 120), (2, 14336, 4096, 60, 148)])
def test_chunks_of_two_octets_are_shared_out_by_whole_parts(bits, n, k, m, grid):
    """Their sums over CTAs weigh more than their chunks: parts of one tile per CTA, unless that makes the longest CTA much longer (148 SMs)."""
    w = QuantWeight.from_blob(f"NINT{bits}", encode.random_nint_blob(n, k, bits, 16, 5, seed=n, device="cuda"))
    x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(m)).to(torch.bfloat16)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert [params.grid[0] for name, params in _kernel_nodes(lambda: w.matmul(x)) if "tile_tc_kernel" in name] == [grid]
    got, want = w.matmul(x, out_dtype=torch.float32), x.double() @ w.dequantize().double().T
    assert ((got.double() - want).norm() / want.norm()).item() <= 3.6e-4   # as below
    assert torch.equal(got, w.matmul(x, out_dtype=torch.float32))
    assert _status() == 0


GROWING_CALL = """
import ctypes, sys, torch
sys.path.insert(0, %r)
from tyloquant_b200 import QuantWeight, encode, moe
w, small = (QuantWeight.from_blob("NINT6", encode.random_nint_blob(n, k, 6, 24, 7, seed=1, device="cuda")) for n, k in ((4096, 14336), (100, 400)))
gen = torch.Generator("cuda").manual_seed(1)
x, xe = (torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16) for m, k in ((16, 14336), (3, 256)))
want = x.double() @ w.dequantize().double().T
gu, dn = (moe.MoeWeight(encode.quantize_expertwise(torch.randn(shape, device="cuda", generator=gen) * 0.02, [4] * 8, device="cuda"))
          for shape in ((8, 192, 256), (8, 256, 96)))
ids, wts = moe.moe_topk(torch.randn(3, 8, device="cuda", generator=gen), 2)
gw, dw = (torch.stack([m.dequantize_expert(i) for i in range(8)]).double()[ids.long()] for m in (gu, dn))   # [token, route, out, in]
h = torch.einsum("troi,ti->tro", gw, xe.double())
act = h[..., 96:] * h[..., :96] / (1 + torch.exp(-h[..., :96]))
ffn = (torch.einsum("trho,tro->trh", dw, act) * wts.double()[..., None]).sum(1)
y, z = small.matmul(x[:, :400].contiguous()), moe.moe_ffn(gu, dn, xe[:1], ids[:1], wts[:1])   # the kernels' code is loaded, the scratch small
rt, blocks = ctypes.CDLL("libcudart.so.12"), []
for size in [1 << i for i in range(8, 20) for _ in range(48)]:
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0 and rt.cudaMemset(p, 0x3f, ctypes.c_size_t(size)) == 0
    blocks.append(p)
torch.cuda.synchronize()
for p in blocks:
    assert rt.cudaFree(p) == 0
y, z = torch.zeros(16, 4096, device="cuda"), None
side = torch.cuda.Stream()
torch.cuda.synchronize()
torch.cuda._sleep(400_000_000)   # the default stream is busy for a fifth of a second
with torch.cuda.stream(side):
    w.matmul(x, out=y)
    z = moe.moe_ffn(gu, dn, xe, ids, wts)
side.synchronize()
busy = not torch.cuda.default_stream().query()
err = [((a.double() - b).norm() / b.norm()).item() for a, b in ((y, want), (z, ffn))]
print(busy, err)
assert max(err) <= 1e-3, err
"""


WARM_CALL = """
import sys, torch
sys.path.insert(0, %r)
from tyloquant_b200 import QuantWeight, encode
ws = [QuantWeight.from_blob("NINT4", encode.random_nint_blob(14336, 4096, 4, 32, 6, seed=1, device="cuda")),
      QuantWeight.from_blob("NINT6", encode.random_nint_blob(14336, 4096, 6, 24, 7, seed=1, device="cuda")),
      QuantWeight.from_blob("NVQ3", encode.nvq_blob(encode.quantize_nvq3(torch.randn(640, 4096).numpy(), encode.d4_256_codebook()[None], jsc=False, device="cuda")))]
x = torch.randn(600, 4096, device="cuda").to(torch.bfloat16)
for w in ws:
    for warm, later in %s:
        for fn in (lambda m, w=w: w.matmul(x[:m]), lambda m, w=w: w.matmul_glu(x[:m])):
            fn(warm)
            torch.cuda.synchronize()
            for m in later:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    y = fn(m)
                graph.replay()
                torch.cuda.synchronize()
                assert torch.isfinite(y.float()).all() and ((fn(m).float() - y.float()).norm() / y.float().norm()).item() < 1e-3, m
"""


@pytest.mark.parametrize("calls", [((8, (2, 3, 5)), (257, (256, 40, 16, 3)), (512, (300, 8, 1))),
                                   ((257, (256, 40, 16, 9, 8, 5, 4, 3, 2, 1)),)])   # the second: nothing but the tile kernel has run before the captures
def test_one_call_makes_room_for_captures_of_smaller_batches(calls):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", WARM_CALL % (root, calls)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


def test_call_that_grows_the_scratch_while_the_default_stream_is_busy():
    """New scratch, in memory that held something else, is cleared in the order of the call's own stream (here a non-blocking one)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", GROWING_CALL % root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


@pytest.mark.parametrize("rows,kernel", [((33, 40), "tile_tc_kernel"), ((16, 9), "rows_mma_kernel")])
def test_overlapping_calls_spoil_no_later_ones(rows, kernel):
    """Calls on one device share scratch and have to be ordered by their streams.  Two of the same kernel that overlap all the same
    may be wrong, but leave nothing behind: arrival counts belong to one call (tiles shared by CTAs, rows in slices of K)."""
    ws = [QuantWeight.from_blob("NINT6", encode.random_nint_blob(n, k, 6, 24, 7, seed=n, device="cuda")) for n, k in ((4096, 14336), (1000, 9000))]
    gen = torch.Generator("cuda").manual_seed(1)
    xs = [torch.randn(m, w.k, device="cuda", generator=gen).to(torch.bfloat16) for m, w in zip(rows, ws)]
    for w, x in zip(ws, xs):
        assert any(kernel in name for name in _kernels(lambda: w.matmul(x)))
    want = [w.matmul(x, out_dtype=torch.float32) for w, x in zip(ws, xs)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(40):
        for s, w, x in zip(streams, ws, xs):
            with torch.cuda.stream(s):
                w.matmul(x)
    torch.cuda.synchronize()
    for _ in range(3):
        for w, x, y in zip(ws, xs, want):
            assert torch.equal(w.matmul(x, out_dtype=torch.float32), y)


@pytest.mark.parametrize("rows", [8, 16, 40])
def test_two_threads_on_one_stream(rows):
    """A product is two launches over scratch of the device (of the few-rows kernel, of the tile kernel): those of two threads on
    the same stream do not mix."""
    w = QuantWeight.from_blob("NINT4", encode.random_nint_blob(256, 512, 4, 32, 6, seed=1, device="cuda"))
    gen = torch.Generator("cuda").manual_seed(1)
    xs = [torch.randn(rows, 512, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(4)]
    want = [w.matmul(x) for x in xs]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(stream):
            for _ in range(20):
                ys = [w.matmul(xs[i]) for _ in range(100)]
                stream.synchronize()
                wrong.extend(i for y in ys if not torch.equal(y, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, len(wrong)


class _NodeParams(ctypes.Structure):   # cudaKernelNodeParams
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("smem", ctypes.c_uint), ("args", ctypes.c_void_p),
                ("extra", ctypes.c_void_p)]


def _kernel_nodes(fn):
    """Name and parameters of the kernels that a call launches: those of its captured graph."""
    rt = ctypes.CDLL("libcudart.so.12")
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert rt.cudaGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    for node in nodes:
        kind, params, name = ctypes.c_int(-1), _NodeParams(), ctypes.c_char_p()
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:   # a kernel
            assert rt.cudaGraphKernelNodeGetParams(ctypes.c_void_p(node), ctypes.byref(params)) == 0
            assert rt.cudaFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
            yield name.value.decode(), params


def _kernels(fn):
    return [name for name, _ in _kernel_nodes(fn)]


@pytest.mark.parametrize("dtype,entries,banks", [("NVQ3J-512", 512, 4), ("NVQ3J-L", 1024, 2)])
def test_codebooks_that_fill_shared_memory(dtype, entries, banks):
    """Wide batches take narrower token tiles where the tables leave no room for 256 columns, not passes of a few rows."""
    n, k = 300, 1000
    wt = np.random.default_rng(1).standard_normal((n, k), dtype=np.float32) * np.float32(0.02)
    w = QuantWeight.from_blob(dtype, encode.nvq_blob(encode.quantize_nvq3(wt, encode.synthetic_d4_banks(entries, banks, seed=5), jsc=True, device="cuda")))
    ref = w.dequantize().double()
    gen = torch.Generator("cuda").manual_seed(1)
    for m in (208, 224, 240, 256, 257, 500, 512):
        x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
        want = x.double() @ ref.T
        got = w.matmul(x, out_dtype=torch.float32).double()
        assert ((got - want).norm() / want.norm()).item() <= 1e-5, m
        names = _kernels(lambda: w.matmul(x))
        assert len(names) == 2 and any("tile_tc_kernel" in name for name in names), (m, names)
    assert _status() == 0


@pytest.mark.parametrize("profile", [(5, 28, 7), (8, 22, 7), (4, 27, 6), (4, 12, 6), (6, 36, 7), (8, 44, 8), (8, 60, 7)])
def test_padded_groups_keep_the_integer_kernels_accuracy(profile):
    """Group sizes that are no multiple of eight: two f16 terms per weight (the last one: the integer kernels), within the 1e-5 of
    the paths with fewer rows; rows whose minimum dwarfs their scale among them."""
    bits, gs, sb = profile
    for n, k in ((1, 24), (129, 1001), (272, 4104), (1000, 776)):
        t = encode.quantize_nint(np.random.default_rng(n).standard_normal((n, k)).astype(np.float32), bits, gs, sb)
        scale, minimum = (np.array(t[name], dtype=np.float16) for name in ("neuron_scale", "neuron_min"))
        scale[3::7] *= np.float16(2.0 ** -9)
        scale[5::11] = 0
        minimum[6::13] = 0
        t["neuron_scale"], t["neuron_min"] = scale, minimum
        blob = encode.nint_blob(t)
        w = QuantWeight.from_blob(f"NINT{bits}", blob)
        ref = O.dequant_nint(O.unpack_nint(blob))
        for m in (4, 5, 16, 17, 64, 65, 129, 257, 520):
            x = encode.bf16_round(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32))
            y = w.matmul(bf16_tensor(x), out_dtype=torch.float32).cpu().numpy()
            err = y.astype(np.float64) - x.astype(np.float64) @ ref.astype(np.float64).T
            size = np.sqrt(np.square(x, dtype=np.float64) @ np.square(ref, dtype=np.float64).T)
            assert np.linalg.norm(err) <= 1e-5 * np.linalg.norm(size), (profile, n, k, m)
        w.free()
    assert _status() == 0


def test_state_scales_far_apart():
    """State scales that are no f16 numbers side by side: rows that only have small ones keep their accuracy."""
    n, k = 100, 400
    wt = np.random.default_rng(1).standard_normal((n, k), dtype=np.float32) * np.float32(0.02)
    t = encode.quantize_nvq3(wt, encode.synthetic_d4_banks(512, 2, seed=5), jsc=True, device="cuda")
    t["sub"][:n // 2] = t["sub"][:n // 2] % 4            # states 0 .. 3 for the first rows
    t["sub"][n // 2:] = 12 + t["sub"][n // 2:] % 4
    blob = encode.nvq_blob(t)
    at = blob.index(bytes([1, 2, 16, 1]), 36) + 4
    lut = np.where(np.arange(16) < 4, 1.37 * 2.0 ** -18, 2.0 ** 14).astype("<f2")
    blob = blob[:at] + lut.tobytes() + blob[at + 32:]
    ref = O.dequant_nvq(O.unpack_nvq(blob)).astype(np.float64)
    w = QuantWeight.from_blob("NVQ3J-512", blob)
    for m in (2, 40, 300):
        x = encode.bf16_round(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32))
        y = w.matmul(bf16_tensor(x), out_dtype=torch.float32).cpu().numpy()
        err, size = y - x.astype(np.float64) @ ref.T, np.sqrt(np.square(x, dtype=np.float64) @ np.square(ref).T)
        for rows in (slice(0, n // 2), slice(n // 2, n)):
            assert np.linalg.norm(err[:, rows]) <= 1e-5 * np.linalg.norm(size[:, rows]), (m, rows)
    assert _status() == 0


@pytest.mark.parametrize("profile", [(2, 16, 5), (3, 24, 5), (4, 24, 6), (4, 32, 6), (6, 24, 7), (8, 48, 7)])
def test_accuracy_of_one_term_weights(profile):
    """Two f16 roundings a weight, of its group's offset and of the whole, each up to 2^-12 of its size's power of two, 1.4e-4 to
    2.8e-4 of the size in the mean square: 2.3e-4 to 2.9e-4 together on these weights, asserted with a quarter more."""
    bits, gs, sb = profile
    k = 2888
    gen = torch.Generator("cuda").manual_seed(bits)
    wt = (torch.randn(1000, k, device="cuda", generator=gen) * 0.02).to(torch.bfloat16).float()
    w = QuantWeight.from_blob(f"NINT{bits}", encode.nint_blob(encode.quantize_nint(wt, bits, gs, sb, device="cuda")))
    ref = w.dequantize().double()
    for m in (5, 33, 600):
        x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
        want = x.double() @ ref.T
        got = w.matmul(x, out_dtype=torch.float32).double()
        assert ((got - want).norm() / want.norm()).item() <= 3.6e-4, m
    w.free()
