"""Edges of loading: pieces, slices, whole-byte storage, padded experts -- decoded bit for bit."""

import os
import struct
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import mfq_oracle as O  # noqa: E402
from tyloquant_b200 import QuantWeight, _capi, encode, moe  # noqa: E402


def _same(a, b):
    return np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))


@pytest.mark.parametrize("profile", [(2, 16, 5), (3, 24, 5), (4, 32, 6), (5, 28, 7), (6, 24, 7), (8, 48, 7), (8, 22, 7)])
def test_scalar_tensors_of_one_and_many_pieces(profile):
    bits, gs, sb = profile
    for n, k in [(1, 1), (17, 333), (1500, 5000), (40, 1 << 19)]:   # the last: a row-block alone exceeds a staging piece
        blob = encode.random_nint_blob(n, k, bits, gs, sb, seed=n + bits, device="cuda")
        ref = O.dequant_nint(O.unpack_nint(blob))
        w = QuantWeight.from_blob(f"NINT{bits}", blob)
        assert _same(w.dequantize().cpu().numpy(), ref), (profile, n, k)
        w.free()
        if n > 16 and k < 1 << 19:
            cut = min(n, 1201)
            rows = QuantWeight.from_blob(f"NINT{bits}", blob, axis=0, begin=13, end=cut)
            assert _same(rows.dequantize().cpu().numpy(), ref[13:cut])
            lo, hi = 3 * gs, (k // gs - 2) * gs
            cols = QuantWeight.from_blob(f"NINT{bits}", blob, axis=1, begin=lo, end=hi)
            assert _same(cols.dequantize().cpu().numpy(), ref[:, lo:hi])


def test_whole_byte_storage_of_older_writers():
    t = encode.quantize_nint(np.random.default_rng(1).standard_normal((33, 250)).astype(np.float32), 4, 24, 6)
    legacy = b"".join([struct.pack("<BBiii", 4, 6, 24, 0, 250), struct.pack("<I", 2), struct.pack("<2q", 33, 250), struct.pack("<II", 33, t["ng"]),
                       t["neuron_scale"].astype("<f2").tobytes(), t["neuron_min"].astype("<f2").tobytes(), t["sub_scale"].numpy().tobytes(),
                       t["sub_min"].numpy().tobytes(), t["q"].numpy().tobytes()])
    a, b = QuantWeight.from_blob("NINT4", legacy), QuantWeight.from_blob("NINT4", encode.nint_blob(t))
    assert _same(a.dequantize().cpu().numpy(), b.dequantize().cpu().numpy())


@pytest.mark.parametrize("jsc", [False, True])
def test_lattice_tensors(jsc):
    banks = encode.synthetic_d4_banks(512, 2, seed=5) if jsc else O.d4_256_codebook()[None]
    for n, k in [(1, 5), (50, 1003), (3000, 4800)]:
        wt = np.random.default_rng(n).standard_normal((n, k), dtype=np.float32)
        blob = encode.nvq_blob(encode.quantize_nvq3(wt, banks, jsc=jsc, device="cuda"))
        ref = O.dequant_nvq(O.unpack_nvq(blob))
        w = QuantWeight.from_blob("NVQ3J-512" if jsc else "NVQ3", blob)
        assert _same(w.dequantize().cpu().numpy(), ref), (n, k)
        if n > 2000:
            part = QuantWeight.from_blob("NVQ3J-512" if jsc else "NVQ3", blob, axis=0, begin=1001, end=2900)
            assert _same(part.dequantize().cpu().numpy(), ref[1001:2900])


def test_experts_with_padded_rows_and_a_shard():
    e, out, k = 12, 100, 300   # 100 rows: padded to 112 on the device
    w = (np.random.default_rng(3).standard_normal((e, out, k)) * 0.02).astype(np.float32)
    bits = [2, 3, 4, 6, 2, 3, 4, 6, 5, 5, 8, 8]
    blob = encode.quantize_expertwise(w, bits, device="cuda")
    whole, shard = moe.MoeWeight(blob), moe.MoeWeight(blob, 0, 3, 9)
    for i in range(e):
        b, gs, sb = encode.CANONICAL_NINT[bits[i]]
        ref = O.dequant_nint(O.unpack_nint(encode.nint_blob(encode.quantize_nint(w[i], b, gs, sb, device="cuda"))))
        assert _same(whole.dequantize_expert(i).cpu().numpy(), ref), i
        if 3 <= i < 9:
            assert _same(shard.dequantize_expert(i).cpu().numpy(), ref), i


def test_memory_of_freed_tensors_is_taken_again_only_when_idle():
    """Tensors loaded into the blocks of freed ones, with work on the freed ones still queued on another stream."""
    side = torch.cuda.Stream()
    x = torch.randn(1, 4096, device="cuda", dtype=torch.bfloat16)
    last = None
    for i, n in enumerate([2048, 2048, 1950, 2048, 300, 2048]):   # the same size, a little smaller, much smaller
        blob = encode.random_nint_blob(n, 4096, 4, 24, 6, seed=i, device="cuda")
        ref = O.dequant_nint(O.unpack_nint(blob))
        w = QuantWeight.from_blob("NINT4", blob)
        assert _same(w.dequantize().cpu().numpy(), ref), (i, n)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(50):
                y = w.matmul(x)
        w.free()
        if last is not None and last.shape == y.shape:
            assert not torch.equal(last, y)
        got = y.float().cpu().numpy()
        want = x.float().cpu().numpy() @ ref.T
        assert np.allclose(got, want, atol=2e-2 * np.abs(want).max()), (i, n)
        last = y


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_a_weight_freed_beside_a_capture_does_not_end_it(mode):
    """Freeing is allowed there: in the capturing thread in the relaxed mode, and in other threads in both."""
    w, other, third = (QuantWeight.from_blob("NINT4", encode.random_nint_blob(512, 512, 4, 24, 6, seed=i, device="cuda")) for i in range(3))
    x = torch.randn(1, 512, device="cuda").to(torch.bfloat16)
    want, out = w.matmul(x), torch.empty(1, 512, device="cuda", dtype=torch.bfloat16)
    w.matmul(x, out=out)
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode=mode)
        w.matmul(x, out=out)
        t = threading.Thread(target=other.free)
        t.start()
        t.join()
        if mode == "relaxed":
            third.free()
        w.matmul(x, out=out)
        graph.capture_end()
    out.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("replay", [False, True])
def test_freeing_waits_for_work_on_any_stream(replay):
    """A freed tensor's block may be written by the next load, so freeing returns after kernels and graphs that could read it."""
    ws = [QuantWeight.from_blob("NINT4", encode.random_nint_blob(512, 512, 4, 24, 6, seed=i, device="cuda")) for i in range(4)]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    if replay:
        with torch.cuda.graph(graph):
            torch.cuda._sleep(100_000_000)
    for w in ws:
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay() if replay else torch.cuda._sleep(100_000_000)
        done = stream.record_event()
        w.free()
        assert done.query()


def test_parked_memory_is_given_back():
    _capi.check(_capi.lib.mfqb_memory_trim(0))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    w = QuantWeight.from_blob("NINT4", encode.random_nint_blob(8192, 8192, 4, 24, 6, seed=1, device="cuda"))
    torch.cuda.empty_cache()
    w.free()
    kept = before - torch.cuda.mem_get_info()[0]
    _capi.check(_capi.lib.mfqb_memory_trim(0))
    assert kept > 30 << 20 and before - torch.cuda.mem_get_info()[0] < kept - (30 << 20)


NO_ROOM = """
import ctypes, os, sys
sys.path.insert(0, %r)
import numpy as np, torch
from oracle import mfq_oracle as O
from tyloquant_b200 import QuantWeight, encode
shim = ctypes.CDLL(os.environ["LD_PRELOAD"])
blob = encode.random_nint_blob(8000, 4000, 4, 24, 6, seed=1, device="cuda")
torch.cuda.synchronize()
shim.fail_next(%d)
try:
    QuantWeight.from_blob("NINT4", blob)
except Exception as e:
    assert "memory" in str(e), e
else:
    raise SystemExit("the load should have failed")
shim.fail_next(0)
w = QuantWeight.from_blob("NINT4", blob)
assert np.array_equal(w.dequantize().cpu().numpy(), O.dequant_nint(O.unpack_nint(blob)))
"""

SHIM = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int at;
void fail_next(int n) { at = n; }
int cudaMalloc(void** p, size_t n) {
    int (*real)(void**, size_t) = (int (*)(void**, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
    if (n == (2u << 20) && at && --at == 0) return 2;
    return real(p, n);
}
"""


@pytest.mark.parametrize("block", [1, 3])
def test_load_after_one_that_found_no_room(tmp_path, block):
    """Staging survives between loads; a block (the first, or one of several) whose device half could not be allocated is not taken
    for complete."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", NO_ROOM % (root, block)], env={**os.environ, "LD_PRELOAD": str(lib)}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


def test_experts_larger_than_a_staging_piece():
    """Experts are cut by row-blocks; 100 and 500 rows are padded to whole ones, the last piece with them."""
    for e, out, k in ((3, 100, 40000), (5, 500, 9000)):
        w = torch.randn(e, out, k, device="cuda", generator=torch.Generator("cuda").manual_seed(out)) * 0.02
        bits = [(6, 4, 8, 6, 6)[i] for i in range(e)]
        blob = encode.quantize_expertwise(w, bits, device="cuda")
        whole, shard = moe.MoeWeight(blob), moe.MoeWeight(blob, 0, 1, 3)
        for i in range(e):
            b, gs, sb = encode.CANONICAL_NINT[bits[i]]
            ref = O.dequant_nint(O.unpack_nint(encode.nint_blob(encode.quantize_nint(w[i], b, gs, sb, device="cuda"))))
            assert _same(whole.dequantize_expert(i).cpu().numpy(), ref), i
            if 1 <= i < 3:
                assert _same(shard.dequantize_expert(i).cpu().numpy(), ref), i
