"""GPU parity for the mixture-of-experts rows of the path: router, route plan, NINTM weights,
routed expert matmul, expert FFN and expert-range shards, against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import mfq_oracle as O  # noqa: E402
from tyloquant_b200 import encode, moe  # noqa: E402
from test_nint_gpu import rel_l2, bf16_tensor, REL_L2  # noqa: E402
from test_tile_gpu import _kernels  # noqa: E402


@pytest.mark.parametrize("tokens,experts,k", [(1, 128, 8), (33, 128, 8), (7, 256, 6), (5, 16, 16), (9, 384, 12), (3, 100, 8), (64, 4096, 4)])
def test_router_ids_are_bit_exact(tokens, experts, k):
    rng = np.random.default_rng(tokens + experts)
    z = rng.standard_normal((tokens, experts)).astype(np.float32)
    z[0, :4] = z[0, 4]          # ties resolve to the smaller expert id
    if tokens > 1:
        z[1, 3] = np.nan        # NaN ranks last
    zt = torch.from_numpy(z).cuda()
    for mode in (O.ROUTER_DELAYED_SOFTMAX, O.ROUTER_SOFTMAX, O.ROUTER_SIGMOID, O.ROUTER_SQRT_SOFTPLUS):
        ids, w = moe.moe_topk(zt, k, mode=mode, normalize=(mode != O.ROUTER_DELAYED_SOFTMAX), norm_floor=1e-20, scale=1.5)
        rid, rw = O.moe_topk(z, k, mode=mode, normalize=(mode != O.ROUTER_DELAYED_SOFTMAX), norm_floor=1e-20, scale=1.5)
        if mode in (O.ROUTER_DELAYED_SOFTMAX, O.ROUTER_SIGMOID):
            # selection on monotone functions of the raw logits: exact
            assert np.array_equal(ids.cpu().numpy(), rid), mode
            np.testing.assert_allclose(w.cpu().numpy(), rw, rtol=2e-6, atol=1e-7)
        else:
            # scores pass through expf / log1pf, whose last bits may differ between the device and
            # numpy: an id may differ from the oracle's only where the two scores involved are
            # within 2 float32 units of each other (a numerical tie)
            got = ids.cpu().numpy()
            scores = O.router_scores(z, mode)
            for t, r in zip(*np.nonzero(got != rid)):
                a, b = scores[t, got[t, r]], scores[t, rid[t, r]]
                assert abs(a - b) <= 2 * np.spacing(max(abs(a), abs(b)).astype(np.float32)), (mode, t, r, a, b)
    bias = torch.from_numpy(rng.standard_normal(experts).astype(np.float32)).cuda()
    ids, w = moe.moe_topk(zt, k, bias=bias)
    rid, rw = O.moe_topk(z, k, bias=bias.cpu().numpy())
    assert np.array_equal(ids.cpu().numpy(), rid)
    np.testing.assert_allclose(w.cpu().numpy(), rw, rtol=2e-6, atol=1e-7)


def test_router_matches_torch_topk():
    z = torch.randn(256, 128, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    ids, w = moe.moe_topk(z, 8)
    tv, ti = torch.topk(z, 8, dim=1)
    assert torch.equal(ids.long(), ti)
    assert torch.allclose(w, torch.softmax(tv, dim=1), rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("tokens,experts,k", [(1, 128, 8), (40, 128, 8), (300, 64, 4), (3, 7, 2), (700, 128, 8)])
def test_route_plan_matches_oracle(tokens, experts, k):
    rng = np.random.default_rng(tokens)
    ids = np.stack([rng.choice(experts, k, replace=False) for _ in range(tokens)]).astype(np.int32)
    eb, tb, order = moe.route_plan(torch.from_numpy(ids).cuda(), experts, tile_m=8)
    reb, rtb, _, rorder = O.route_plan(ids, experts, 8)
    assert np.array_equal(eb.cpu().numpy(), reb)
    assert np.array_equal(tb.cpu().numpy(), rtb)
    assert np.array_equal(order.cpu().numpy(), rorder)   # ascending pair index inside every expert segment


def _moe_case(e_count, h, f, bits, seed):
    rng = np.random.default_rng(seed)
    wgu = encode.bf16_round(rng.standard_normal((e_count, 2 * f, h), dtype=np.float32) * np.float32(0.02))
    wdn = encode.bf16_round(rng.standard_normal((e_count, h, f), dtype=np.float32) * np.float32(0.02))
    return encode.quantize_expertwise(wgu, bits, device="cuda"), encode.quantize_expertwise(wdn, bits, device="cuda")


def test_golden_nintm_experts_decode_bit_exact(golden):
    for key in ("nintm_gate_up", "nintm_down"):
        blob = golden[key + "__blob"].tobytes()
        ref = golden[key + "__w"]
        w = moe.MoeWeight(blob)
        assert (w.info.n_experts, w.info.out_per_expert, w.info.k) == ref.shape
        for e in range(ref.shape[0]):
            got = w.dequantize_expert(e).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), ref[e].view(np.uint32)), (key, e)
        w.free()


def test_golden_nintm_ffn_matches_oracle(golden):
    gu_ref, dn_ref = golden["nintm_gate_up__w"], golden["nintm_down__w"]
    gu = moe.MoeWeight(golden["nintm_gate_up__blob"].tobytes())
    dn = moe.MoeWeight(golden["nintm_down__blob"].tobytes())
    e_count, _, h = gu_ref.shape
    rng = np.random.default_rng(8)
    for tokens in (1, 5):
        x = encode.bf16_round(rng.standard_normal((tokens, h), dtype=np.float32))
        z = rng.standard_normal((tokens, e_count)).astype(np.float32)
        ids, wts = moe.moe_topk(torch.from_numpy(z).cuda(), 2)
        rid, rw = O.moe_topk(z, 2)
        assert np.array_equal(ids.cpu().numpy(), rid)
        out = gu.matmul_id(bf16_tensor(x), ids, out_dtype=torch.float32).cpu().numpy()
        want = np.stack([[gu_ref[rid[t, r]] @ x[t] for r in range(2)] for t in range(tokens)])
        assert rel_l2(out, want) <= REL_L2
        y = moe.moe_ffn(gu, dn, bf16_tensor(x), ids, wts).cpu().numpy()
        y_ref = O.moe_ffn(x, gu_ref, dn_ref, rid, rw)
        # nothing is rounded between the two matmuls (the activation stays float32, or is never
        # stored at all at decode sizes): the stated bound holds against the all-float32 oracle
        assert rel_l2(y, y_ref) <= REL_L2
    gu.free()
    dn.free()


@pytest.mark.parametrize("tokens", [1, 32, 101])
def test_mixed_precision_layer_and_expert_shards(tokens):
    """A scaled-down config-4 layer: 16 experts, bits drawn from {2,3,4,6}, top-4."""
    e_count, h, f, k = 16, 256, 96, 4
    bits = np.random.default_rng(4003).choice([2, 3, 4, 6], e_count)
    gu_blob, dn_blob = _moe_case(e_count, h, f, bits, seed=4001)
    gu_ref = O.dequant_nintm(O.unpack_nintm(gu_blob))
    dn_ref = O.dequant_nintm(O.unpack_nintm(dn_blob))
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    rng = np.random.default_rng(4002)
    x = encode.bf16_round(rng.standard_normal((tokens, h), dtype=np.float32))
    z = rng.standard_normal((tokens, e_count)).astype(np.float32)
    ids, wts = moe.moe_topk(torch.from_numpy(z).cuda(), k)
    rid, rw = O.moe_topk(z, k)
    assert np.array_equal(ids.cpu().numpy(), rid)
    y = moe.moe_ffn(gu, dn, bf16_tensor(x), ids, wts).cpu().numpy()
    assert rel_l2(y, O.moe_ffn(x, gu_ref, dn_ref, rid, rw)) <= REL_L2
    assert sum(gu.expert_bytes(e) for e in range(e_count)) == gu.info.payload_bytes
    # expert-parallel shards: each holds a contiguous expert range; their outputs add up
    parts = []
    for b, e in ((0, 6), (6, 16)):
        sgu, sdn = moe.MoeWeight(gu_blob, expert_begin=b, expert_end=e), moe.MoeWeight(dn_blob, expert_begin=b, expert_end=e)
        parts.append(moe.moe_ffn(sgu, sdn, bf16_tensor(x), ids, wts))
        sgu.free()
        sdn.free()
    assert rel_l2((parts[0] + parts[1]).cpu().numpy(), y) <= 1e-5
    gu.free()
    dn.free()


@pytest.mark.parametrize("tokens", [16, 40, 400])
def test_route_plan_tiles_and_grouped_tile_kernel(tokens):
    """48 experts, top-4, the four canonical precisions in one launch: 16 tokens give integer tiles of two pairs, 40 tokens
    (3.3 pairs per expert) and 400 (33) go to the tensor-memory tile kernel.  Also through an expert shard."""
    e_count, h, f, k = 48, 256, 96, 4
    bits = np.random.default_rng(5003).choice([2, 3, 4, 6], e_count)
    gu_blob, dn_blob = _moe_case(e_count, h, f, bits, seed=5001)
    gu_ref = O.dequant_nintm(O.unpack_nintm(gu_blob))
    dn_ref = O.dequant_nintm(O.unpack_nintm(dn_blob))
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    rng = np.random.default_rng(5002 + tokens)
    x = encode.bf16_round(rng.standard_normal((tokens, h), dtype=np.float32))
    z = rng.standard_normal((tokens, e_count)).astype(np.float32)
    ids, wts = moe.moe_topk(torch.from_numpy(z).cuda(), k)
    rid, rw = O.moe_topk(z, k)
    out = gu.matmul_id(bf16_tensor(x), ids, out_dtype=torch.float32).cpu().numpy()
    want = np.stack([[gu_ref[rid[t, r]] @ x[t] for r in range(k)] for t in range(tokens)])
    assert rel_l2(out, want) <= REL_L2
    y = moe.moe_ffn(gu, dn, bf16_tensor(x), ids, wts).cpu().numpy()
    assert rel_l2(y, O.moe_ffn(x, gu_ref, dn_ref, rid, rw)) <= REL_L2
    parts = []
    for b, e in ((0, 20), (20, 48)):
        sgu, sdn = moe.MoeWeight(gu_blob, expert_begin=b, expert_end=e), moe.MoeWeight(dn_blob, expert_begin=b, expert_end=e)
        parts.append(moe.moe_ffn(sgu, sdn, bf16_tensor(x), ids, wts))
        sgu.free()
        sdn.free()
    assert rel_l2((parts[0] + parts[1]).cpu().numpy(), y) <= 1e-5
    gu.free()
    dn.free()


def test_one_token_calls_back_to_back_past_the_expert_table():
    """514 experts, two of them past the table a CTA keeps at hand; calls with other routes follow one another without a wait."""
    e_count, h, f, k = 514, 72, 48, 4
    gu_blob, dn_blob = _moe_case(e_count, h, f, np.random.default_rng(5).choice([3, 4, 6], e_count), seed=6)
    gu_ref, dn_ref = O.dequant_nintm(O.unpack_nintm(gu_blob)), O.dequant_nintm(O.unpack_nintm(dn_blob))
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    rng = np.random.default_rng(7)
    x = encode.bf16_round(rng.standard_normal((1, h), dtype=np.float32))
    zs = [rng.standard_normal((1, e_count)).astype(np.float32) for _ in range(12)]
    for i, z in enumerate(zs):
        z[0, [512, 513, i, 511]] += 9.0
    xt, zt = bf16_tensor(x), [torch.from_numpy(z).cuda() for z in zs]
    torch.cuda.synchronize()
    ys = []
    for z in zt:
        ids, wts = moe.moe_topk(z, k)
        ys.append(moe.moe_ffn(gu, dn, xt, ids, wts))
    for y, z in zip(ys, zs):
        rid, rw = O.moe_topk(z, k)
        assert rel_l2(y.cpu().numpy(), O.moe_ffn(x, gu_ref, dn_ref, rid, rw)) <= REL_L2
    gu.free()
    dn.free()


@pytest.mark.parametrize("tokens", [2, 6, 64])
def test_gate_up_shard_beside_a_whole_down_weight(tokens):
    """Routes to experts that only the down weight holds add nothing, whatever earlier calls left in the scratch: the single-row
    kernels, the integer tiles and the tensor-memory tiles."""
    e_count, h, f, k = 8, 256, 96, 2
    gu_blob, dn_blob = _moe_case(e_count, h, f, [4, 6] * 4, seed=31)
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    gu_shard, dn_shard = moe.MoeWeight(gu_blob, 0, 2, 5), moe.MoeWeight(dn_blob, 0, 2, 5)
    rng = np.random.default_rng(32)
    x = bf16_tensor(encode.bf16_round(rng.standard_normal((tokens, h), dtype=np.float32)))
    ids, wts = moe.moe_topk(torch.from_numpy(rng.standard_normal((tokens, e_count)).astype(np.float32)).cuda(), k)
    moe.moe_ffn(gu, dn, 64.0 * x, ids, wts)
    got = moe.moe_ffn(gu_shard, dn, x, ids, wts)
    want = moe.moe_ffn(gu_shard, dn_shard, x, ids, wts)
    assert (got - want).abs().max().item() <= 1e-5 * want.abs().max().item()   # float32 sums in another order
    for w in (gu, dn, gu_shard, dn_shard):
        w.free()


def test_more_pairs_than_a_grid_dimension():
    """8200 tokens of 8 routes: 65,600 pairs through the routed product and the FFN."""
    e_count, h, f, tokens, routes = 8, 48, 24, 8200, 8
    gu_blob, dn_blob = _moe_case(e_count, h, f, [4, 6] * 4, seed=41)
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    gen = torch.Generator("cuda").manual_seed(42)
    x = torch.randn(tokens, h, device="cuda", generator=gen).to(torch.bfloat16)
    ids, wts = moe.moe_topk(torch.randn(tokens, e_count, device="cuda", generator=gen), routes)
    gw, dw = (torch.stack([w.dequantize_expert(e) for e in range(e_count)]).double() for w in (gu, dn))
    every = torch.einsum("th,eoh->teo", x.double(), gw)
    want = torch.gather(every, 1, ids.long()[:, :, None].expand(-1, -1, 2 * f))
    got = gu.matmul_id(x, ids, out_dtype=torch.float32).double()
    assert ((got - want).norm() / want.norm()).item() <= REL_L2
    act = every[..., f:] * every[..., :f] / (1 + torch.exp(-every[..., :f]))
    out = torch.gather(torch.einsum("tef,ehf->teh", act, dw), 1, ids.long()[:, :, None].expand(-1, -1, h))
    want = (out * wts.double()[:, :, None]).sum(1)
    got = moe.moe_ffn(gu, dn, x, ids, wts).double()
    assert ((got - want).norm() / want.norm()).item() <= REL_L2
    gu.free()
    dn.free()


@pytest.mark.parametrize("tokens", [4, 8, 11, 12, 16, 100, 260, 400])
def test_records_with_padded_groups_keep_the_integer_kernels_accuracy(tokens):
    """NINT5's groups of 28 are padded to 32: such a record's products stay within 1e-5 at every batch size (two f16 terms for
    weights and float32 activations on the tile kernel), and the FFN within what its activations' 16 bits cost at fewer pairs."""
    e_count, h, f, k = 8, 520, 200, 2
    gu_blob, dn_blob = _moe_case(e_count, h, f, [3, 4, 5, 8] * 2, seed=51)
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    gen = torch.Generator("cuda").manual_seed(52)
    x = torch.randn(tokens, h, device="cuda", generator=gen).to(torch.bfloat16)
    ids, wts = moe.moe_topk(torch.randn(tokens, e_count, device="cuda", generator=gen), k)
    gw, dw = (torch.stack([w.dequantize_expert(e) for e in range(e_count)]).double() for w in (gu, dn))
    every = torch.einsum("th,eoh->teo", x.double(), gw)
    pick = lambda t: torch.gather(t, 1, ids.long()[:, :, None].expand(-1, -1, t.shape[2]))
    want = pick(every)
    got = gu.matmul_id(x, ids, out_dtype=torch.float32).double()
    assert ((got - want).norm() / want.norm()).item() <= 1e-5
    act = every[..., f:] * every[..., :f] / (1 + torch.exp(-every[..., :f]))
    want = (pick(torch.einsum("tef,ehf->teh", act, dw)) * wts.double()[:, :, None]).sum(1)
    got = moe.moe_ffn(gu, dn, x, ids, wts).double()
    assert ((got - want).norm() / want.norm()).item() <= (2e-5 if tokens * k >= 3 * e_count else 2e-4)
    gu.free()
    dn.free()


@pytest.mark.parametrize("cohorts,tokens", [(9, 400), (16, 400), (16, 2100)])
def test_records_of_many_cohorts(cohorts, tokens):
    """Up to sixteen cohorts take the tile kernel, however many experts share one."""
    e_count, h, f, k = 16, 72, 48, 8
    gen = torch.Generator("cuda").manual_seed(cohorts)
    blobs = []
    for shape in ((e_count, 2 * f, h), (e_count, h, f)):
        w = torch.randn(shape, device="cuda", generator=gen) * 0.02
        pools = []
        for c in range(cohorts):
            ids = list(range(c, e_count, cohorts))
            bits, gs, sb = encode.CANONICAL_NINT[(3, 4, 6)[c % 3]]
            pools.append((ids, f"NINT{bits}", encode.nint_blob(encode.quantize_nint(w[ids].reshape(-1, shape[2]), bits, gs, sb, device="cuda"))))
        blobs.append(encode.nintm_blob(e_count, shape[1], shape[2], pools))
    gu, dn = (moe.MoeWeight(b) for b in blobs)
    x = torch.randn(tokens, h, device="cuda", generator=gen).to(torch.bfloat16)
    ids, wts = moe.moe_topk(torch.randn(tokens, e_count, device="cuda", generator=gen), k)
    gw, dw = (torch.stack([w.dequantize_expert(e) for e in range(e_count)]).double() for w in (gu, dn))
    every = torch.einsum("th,eoh->teo", x.double(), gw)
    act = every[..., f:] * every[..., :f] / (1 + torch.exp(-every[..., :f]))
    out = torch.gather(torch.einsum("tef,ehf->teh", act, dw), 1, ids.long()[:, :, None].expand(-1, -1, h))
    want = (out * wts.double()[:, :, None]).sum(1)
    names = _kernels(lambda: moe.moe_ffn(gu, dn, x, ids, wts))
    assert sum("tile_tc_kernel" in name for name in names) == 2, names
    assert ((moe.moe_ffn(gu, dn, x, ids, wts).double() - want).norm() / want.norm()).item() <= REL_L2
    gu.free()
    dn.free()


def _ffn_reference(gu, dn, x, ids, wts):
    e_count, f = gu.info.n_experts, dn.info.k
    gw, dw = (torch.stack([w.dequantize_expert(e) for e in range(e_count)]).double() for w in (gu, dn))
    every = torch.einsum("th,eoh->teo", x.double(), gw)
    act = every[..., f:] * every[..., :f] / (1 + torch.exp(-every[..., :f]))
    out = torch.gather(torch.einsum("tef,ehf->teh", act, dw), 1, ids.long()[:, :, None].expand(-1, -1, dn.info.out_per_expert))
    return (out * wts.double()[:, :, None]).sum(1)


@pytest.mark.parametrize("tokens", [40, 300, 700])
@pytest.mark.parametrize("bits", [[4, 6], [5, 3]])
def test_hot_experts_take_several_token_tiles(tokens, bits):
    """One expert draws half of all routes: more pairs than a tile holds, so its later tiles start inside its rows."""
    e_count, h, f, k = 16, 200, 72, 2
    gu_blob, dn_blob = _moe_case(e_count, h, f, bits * 8, seed=61)
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    gen = torch.Generator("cuda").manual_seed(tokens)
    x = torch.randn(tokens, h, device="cuda", generator=gen).to(torch.bfloat16)
    z = torch.randn(tokens, e_count, device="cuda", generator=gen)
    z[:, 5] += 20.0
    ids, wts = moe.moe_topk(z, k)
    want = _ffn_reference(gu, dn, x, ids, wts)
    got = moe.moe_ffn(gu, dn, x, ids, wts).double()
    assert ((got - want).norm() / want.norm()).item() <= REL_L2
    assert ((got[-8:] - want[-8:]).norm() / want[-8:].norm()).item() <= REL_L2
    gu.free()
    dn.free()


def test_integer_tiles_of_four_pairs():
    """Between one and a half and two pairs per expert."""
    e_count, h, f, k, tokens = 16, 200, 72, 4, 7
    gu_blob, dn_blob = _moe_case(e_count, h, f, [3, 4, 6, 8] * 4, seed=71)
    gu, dn = moe.MoeWeight(gu_blob), moe.MoeWeight(dn_blob)
    gen = torch.Generator("cuda").manual_seed(72)
    x = torch.randn(tokens, h, device="cuda", generator=gen).to(torch.bfloat16)
    ids, wts = moe.moe_topk(torch.randn(tokens, e_count, device="cuda", generator=gen), k)
    want = _ffn_reference(gu, dn, x, ids, wts)
    names = _kernels(lambda: moe.moe_ffn(gu, dn, x, ids, wts))
    assert any("moe_hetero_tiles_kernel" in name for name in names) and not any("tile_tc_kernel" in name for name in names), names
    assert ((moe.moe_ffn(gu, dn, x, ids, wts).double() - want).norm() / want.norm()).item() <= 2e-4   # 16-bit float32 activations
    gu.free()
    dn.free()
