"""The kernels of the chain (projections, attention, residual + norm) at the sizes where their cuts change, against the oracle
within the reference harness's band.  Every test needs a B200."""
import ctypes
import re

import pytest
import torch

from oracle import pi05_oracle as O
from pi05_megakernel_b200 import fixture as FX

pytestmark = pytest.mark.gpu


# (prefix, batch, mask, steps and layers).  128-key chunks: up to 64 valid keys in the last one and more, one key; the keys of a
# tile over 1, 4 and 8 CTAs; projections on tiles of up to 64 and up to 128 tokens, on two, three, six and eight of them,
# on single CTAs and on pairs, persistent or not; attention on tiles of 2, 4 and 6 tokens.
CUTS = [
    (1, 1, "full", "b200-s2-l2"), (63, 1, "scatter", "b200-s2-l2"), (128, 2, "pad", "b200-s2-l2"), (129, 3, "scatter", "b200-s2-l2"),
    (192, 5, "pad", "b200-s1-l2"), (193, 6, "scatter", "b200-s1-l2"), (301, 1, "scatter", "b200-s2-l2"), (968, 1, "pad", "b200-s2-l2"),
    (1100, 2, "scatter", "b200-s1-l2"), (130, 7, "full", "b200-s1-l2"), (65, 11, "pad", "b200-s1-l2"), (257, 16, "scatter", "b200-s1-l2")]
# (prefix, batch, tokens per page).  What is left of the attention's cuts on a B200: tiles of 2, 4, 6, 8 and 14 tokens over one to eight
# CTAs, the widest with a second segment of probabilities and a ring of four units, also over eight CTAs; dense caches and pages of 64 and 128 tokens
ATTENTION_CUTS = [(512, 1, 64), (600, 5, 0), (700, 6, 128), (700, 3, 64), (896, 9, 0), (896, 5, 64), (1700, 12, 0), (1300, 9, 64),
                  (440, 1, 64), (456, 1, 64), (900, 6, 0), (768, 4, 0), (840, 4, 128), (2176, 11, 0), (2177, 11, 64), (2816, 5, 0),
                  (834, 1, 64), (250, 4, 128), (968, 2, 128), (960, 3, 64), (968, 4, 0), (700, 5, 0), (800, 7, 64), (250, 12, 64), (1160, 9, 0), (2950, 5, 0), (3457, 3, 64),
                  (2945, 3, 64)]
# (The suffix joins the last chunk of the prefix with 1, 4, 6 and 8 cached keys there (2177 and 2945, 900, 2950, 1160), 36, 56 and 60 (1700, 440, 700) and
# with as many as there is room for: 64 on pages of 64 (960), 72 on pages of 128 and dense (968).  72 keys on pages of 64 stay apart (456), and where that is
# no chunk more (840).)
# Attention with the O projection (up to 128 cached tokens, up to two observations): 1, 8 and 9 keys, 64 and 65 (Wo in a place of its own and in that of the keys),
# 72 and 73 (suffix within the first 128 rows and across them), 120 and 128 (an odd and an even number of eights), one page and two
ATTENTION_O = [(1, 1, 0), (1, 2, 64), (8, 1, 0), (9, 2, 64), (64, 1, 64), (65, 1, 64), (65, 2, 0), (72, 1, 128), (73, 2, 64), (120, 1, 0), (127, 2, 64), (128, 1, 64), (128, 2, 128)]


@pytest.mark.parametrize("prefix,batch,mask,variant", CUTS)
def test_chunk_cuts(prefix, batch, mask, variant):
    from pi05_megakernel_b200.arm import Pi05Arm
    geo, ogeo = FX.Geometry(prefix=prefix), O.Geo(prefix=prefix)
    stacked, per = FX.make_batch(geo, FX.SEEDS[1], batch, "cpu", [mask] * batch)
    arm = Pi05Arm(geo, variant, "cuda", batch=batch)
    arm.bind({k: v.cuda() for k, v in (stacked if batch > 1 else per[0]).items()})
    arm.launch()
    arm.status()
    first = arm.outputs()["actions"].cpu()
    arm.launch()
    arm.status()
    assert torch.equal(first, arm.outputs()["actions"].cpu())          # no order of arrival enters the sums
    for b in {0, batch // 2, batch - 1}:
        want, exact = (O.chunk(per[b], ogeo, widen, arm.steps, arm.layers) for widen in (False, True))
        d = O.band(want, first.reshape(batch, 50, 32)[b], exact)
        assert d["pass"], (b, d)
    arm.close()


@pytest.mark.parametrize("prefix,batch,page", ATTENTION_CUTS)
def test_attention_cuts(prefix, batch, page):
    from pi05_megakernel_b200.arm import PagedPrefix, Pi05Arm
    geo, ogeo = FX.Geometry(prefix=prefix), O.Geo(prefix=prefix)
    masks = ["scatter" if b % 2 else "pad" for b in range(batch)]
    stacked, per = FX.make_batch(geo, FX.SEEDS[1], batch, "cpu", masks)
    dev = {k: v.cuda() for k, v in (stacked if batch > 1 else per[0]).items()}
    pages = None
    if page:
        n = -(-prefix // page)
        order = torch.randperm(batch * n, generator=torch.Generator().manual_seed(3))
        pools = []
        for name in ("prefix_k", "prefix_v"):
            t = dev[name].view(batch, geo.layers, prefix, 1, 256)
            t = torch.nn.functional.pad(t, (0, 0, 0, 0, 0, n * page - prefix), value=float("nan"))     # no token behind the prefix is read
            pool = torch.empty((batch * n, geo.layers, page, 1, 256), dtype=t.dtype, device="cuda")
            pool[order.cuda()] = t.view(batch, geo.layers, n, page, 1, 256).transpose(1, 2).reshape(pool.shape)
            pools.append(pool)
        pages = PagedPrefix(*pools, order.view(batch, n))
    arm = Pi05Arm(geo, "b200-s1-l2", "cuda", batch=batch)
    arm.bind(dev, kv_pages=pages)
    arm.launch()
    arm.status()
    got = arm.outputs()["actions"].cpu().reshape(batch, 50, 32)
    for b in {0, batch - 1}:
        want, exact = (O.chunk(per[b], ogeo, widen, 1, 2) for widen in (False, True))
        d = O.band(want, got[b], exact)
        assert d["pass"], (b, d)
    arm.close()


@pytest.mark.parametrize("prefix,batch,page", ATTENTION_O)
def test_attention_with_o_projection(prefix, batch, page):
    test_attention_cuts(prefix, batch, page)


def test_rotary_tables_of_the_chain():
    """What a launch of the chain leaves in its two rotary tables: cos | sin of dim j of token t, [token][128] as the workspace's "rope"
    has been, and in groups of four dims, tokens of all observations next to each other, as the QKV projection reads them."""
    from pi05_megakernel_b200.arm import Pi05Arm
    geo, batch = FX.Geometry(prefix=77), 3
    stacked, per = FX.make_batch(geo, FX.SEEDS[0], batch, "cpu", ["pad", "scatter", "full"])
    arm = Pi05Arm(geo, "b200-s1-l1", "cuda", batch=batch)
    arm.bind({k: v.cuda() for k, v in stacked.items()})
    arm.launch()
    arm.status()
    rows = arm.region("rope", torch.bfloat16, (batch * 50, 128, 2)).cpu()
    grouped = arm.region("rope2", torch.bfloat16, (32, batch * 50, 4, 2)).cpu()
    assert torch.equal(grouped.permute(1, 0, 2, 3).reshape(batch * 50, 128, 2), rows)
    inv = 1.0 / (O.ROPE_THETA ** (torch.arange(0, 256, 2, dtype=torch.int64).float() / 256))
    phase = torch.cat([O.suffix_layout(v["prefix_mask"], 50)[0] for v in per]).float()[:, None] * inv[None]
    # (values up to 1: a rounding to BF16 apart where the FP32 phase differs in its last bit)
    assert float((rows.float() - torch.stack((phase.cos(), phase.sin()), -1).to(torch.bfloat16).float()).abs().max()) <= 2 ** -7
    arm.close()


def test_smaller_binding_stays_in_the_workspace():
    """Four observations of 968 tokens on an engine made for 1100: an attention cut with more partial sums than the longest prefix's.
    What lies behind the workspace stays as it was, and the actions are those of an engine of the binding's own size."""
    from pi05_megakernel_b200 import _lib
    from pi05_megakernel_b200.arm import Pi05Arm
    geo, batch, longest = FX.Geometry(prefix=968), 4, 1100
    lib, sms = _lib.load(), torch.cuda.get_device_properties(0).multi_processor_count
    info, held, needed = (ctypes.c_int * 4)(), ctypes.c_size_t(), [ctypes.c_size_t() for _ in range(2)]
    for p, n in zip((geo.prefix, longest), needed):
        assert lib.pi05_chunk_plan(sms, batch, longest, batch, p, info, ctypes.byref(held), ctypes.byref(n)) == _lib.OK
    assert needed[0].value > needed[1].value            # else room for the longest prefix's sums would do
    stacked, _ = FX.make_batch(geo, FX.SEEDS[0], batch, "cpu", ["pad"] * batch)
    dev = {k: v.cuda() for k, v in stacked.items()}
    arm = Pi05Arm(geo, "b200-s1-l2", "cuda", batch=batch)
    arm.bind(dev)
    arm.launch()
    arm.status()
    want = arm.outputs()["actions"].clone()
    arm.close()
    h, n = ctypes.c_void_p(), ctypes.c_size_t()
    assert lib.pi05_create(0, longest, batch, 0, 1, ctypes.byref(h)) == _lib.OK
    assert lib.pi05_workspace_bytes(h, ctypes.byref(n)) == _lib.OK
    ws = torch.full((n.value + (4 << 20),), 0xA5, dtype=torch.uint8, device="cuda")
    got = torch.zeros_like(want)
    ptrs = (ctypes.c_void_p * _lib.NUM_INPUTS)(*[dev[k].data_ptr() for k in FX.ORDER])
    assert lib.pi05_bind(h, ptrs, geo.prefix, batch, got.data_ptr(), ws.data_ptr(), n.value) == _lib.OK
    assert lib.pi05_launch(h, 1, 2, torch.cuda.current_stream().cuda_stream, None) == _lib.OK
    code, where = ctypes.c_int(), ctypes.c_int()
    assert lib.pi05_status(h, ctypes.byref(code), ctypes.byref(where)) == _lib.OK
    assert bool((ws[n.value:] == 0xA5).all())
    assert torch.equal(got, want)
    assert lib.pi05_destroy(h) == _lib.OK


@pytest.mark.parametrize("batch,variant", [(1, "b200"), (3, "b200-s2-l2")])
def test_launch_into_a_capture(batch, variant):
    """A launch may be recorded into a CUDA graph by its caller; a replay is what a launch is, on the inputs of the moment."""
    from pi05_megakernel_b200.arm import Pi05Arm
    geo = FX.Geometry(prefix=200)
    stacked, _ = FX.make_batch(geo, FX.SEEDS[0], batch, "cpu", ["pad"] * batch)
    dev = {k: (v if batch > 1 or k not in FX.OBSERVATION else v[0]).cuda() for k, v in stacked.items()}
    arm = Pi05Arm(geo, variant, "cuda", batch=batch)
    arm.bind(dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        arm.launch()
    for scale in (1.0, -0.5):
        dev["noise"].mul_(scale)
        arm.outputs()["actions"].zero_()
        graph.replay()
        torch.cuda.synchronize()
        replayed = arm.outputs()["actions"].clone()
        arm.launch()
        arm.status()
        assert bool(replayed.abs().max() > 0) and torch.equal(replayed, arm.outputs()["actions"])
    del graph
    arm.close()


def test_steps_and_layers_may_change_from_launch_to_launch():
    """Other numbers of steps and layers than at the last call: each the result of an arm of that variant, no device memory taken."""
    from pi05_megakernel_b200 import _lib
    from pi05_megakernel_b200.arm import Pi05Arm
    geo = FX.Geometry(prefix=130)
    dev = {k: v.cuda() for k, v in FX.make_inputs(geo, FX.SEEDS[1], "cpu", "scatter").items()}
    sizes = [(10, 18), (3, 18), (2, 2), (10, 18), (9, 5), (1, 18)]
    want = {}
    for steps, layers in set(sizes):
        one = Pi05Arm(geo, f"b200-s{steps}-l{layers}", "cuda")
        one.bind(dev)
        one.launch()
        one.status()
        want[steps, layers] = one.outputs()["actions"].clone()
        assert one.config["launches_per_chunk"] == 5 + 7 * steps * layers
        one.close()
    arm = Pi05Arm(geo, "b200", "cuda")
    arm.bind(dev)
    got = [torch.empty_like(arm.outputs()["actions"]) for _ in sizes]
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for out, (steps, layers) in zip(got, sizes):
        assert arm.lib.pi05_launch(arm.handle, steps, layers, stream, None) == _lib.OK
        out.copy_(arm.outputs()["actions"])
    arm.status()
    assert torch.cuda.mem_get_info()[0] == free
    for out, size in zip(got, sizes):
        assert torch.equal(out, want[size]), size
    arm.close()


@pytest.mark.parametrize("prefix,batch", [(128, 1), (968, 1), (130, 3), (65, 16)])
def test_wait_of_the_chain_that_runs_out(prefix, batch):
    """A projection waits for data that never comes: its waits give up after 10 ms, the kernels behind it return early, the
    status says so, the actions are NaN, and the next launch, on its graphs again, is what it was.  Projections on single CTAs and on
    pairs, attention on one CTA per tile and on a cluster."""
    from pi05_megakernel_b200 import _lib
    from pi05_megakernel_b200.arm import Pi05Arm
    geo = FX.Geometry(prefix=prefix)
    stacked, _ = FX.make_batch(geo, FX.SEEDS[0], batch, "cpu", ["pad"] * batch)
    arm = Pi05Arm(geo, "b200-s1", "cuda", batch=batch)
    arm.bind({k: (v if batch > 1 or k not in FX.OBSERVATION else v[0]).cuda() for k, v in stacked.items()})
    arm.launch()
    arm.status()
    good = arm.outputs()["actions"].clone()
    for layer in (0, 16):
        arm.debug(-1, 20_000_000, -1)
        arm.debug_withhold(layer)
        arm.launch()
        with pytest.raises(_lib.EngineError) as info:
            arm.status()
        assert info.value.code == _lib.ERR_DEVICE_TIMEOUT
        # the MMAs and the epilogue wait for what never comes (and the producers for slots): the header's codes of a projection
        assert int(re.search(r"wait kind (\d+)", str(info.value))[1]) in (1, 2, 3, 6), str(info.value)
        assert bool(torch.isnan(arm.outputs()["actions"]).all())
        arm.debug_withhold(-1)
        arm.debug(-1, 4_000_000_000, -1)
        arm.launch()
        assert arm.status() == (0, 0)
        assert torch.equal(arm.outputs()["actions"], good)
    arm.close()


# Two to nine chunks per CTA: the suffix joined and apart, one CTA per tile and a cluster, the widest tile, whose lanes hold two rows.
@pytest.mark.parametrize("prefix,batch", [(200, 1), (256, 4), (600, 5), (900, 6), (700, 6), (2177, 11)])
def test_attention_reference_moves(prefix, batch):
    """Scores that grow from one chunk of keys to the next, by more than the exponents' reference stands: every CTA has to move it, some
    of them twice.  (The keys of chunk c are scaled by 1 + 3 (c mod 6).)"""
    from pi05_megakernel_b200 import _lib
    from pi05_megakernel_b200.arm import Pi05Arm
    info = (ctypes.c_int * 5)()
    assert _lib.load().pi05_chunk_attention(torch.cuda.get_device_properties(0).multi_processor_count, batch, prefix, prefix, info) == _lib.OK
    assert info[3] >= 2 and not info[4]                 # a CTA with one chunk never moves
    geo, ogeo = FX.Geometry(prefix=prefix), O.Geo(prefix=prefix)
    stacked, per = FX.make_batch(geo, FX.SEEDS[2], batch, "cpu", ["full"] * batch)
    grow = 1.0 + 3.0 * (torch.arange(prefix) // 128 % 6)
    for case in (stacked, *per):
        case["prefix_k"] = (case["prefix_k"].float() * grow.view(prefix, 1, 1)).to(torch.bfloat16)
    arm = Pi05Arm(geo, "b200-s1-l3", "cuda", batch=batch)
    arm.bind({k: v.cuda() for k, v in (stacked if batch > 1 else per[0]).items()})
    arm.launch()
    arm.status()
    got = arm.outputs()["actions"].cpu().reshape(batch, 50, 32)
    for b in {0, batch - 1}:
        want, exact = (O.chunk(per[b], ogeo, widen, arm.steps, arm.layers) for widen in (False, True))
        d = O.band(want, got[b], exact)
        assert d["pass"], (b, d)
    arm.close()


# (800: QKV on single CTAs of 128 features; 2400: QKV and O on persistent pairs)
@pytest.mark.parametrize("tokens", [1, 65, 128, 129, 297, 600, 800, 900, 1200, 2400])
def test_prefill_cuts(tokens):
    from pi05_megakernel_b200.prefill import Pi05Prefill
    geo = FX.PrefillGeometry(tokens=tokens)
    inputs = FX.make_prefill_inputs(geo, 7, "full")
    dev = {k: v.cuda() for k, v in inputs.items()}
    pre = Pi05Prefill(geo, "cuda")
    pre.bind(dev)
    k, v = pre.run(dev["embeddings"], dev["valid"], 2)
    pre.status()
    args = (inputs, inputs["embeddings"], inputs["valid"], geo.q_heads, geo.kv_heads, geo.head_dim)
    wk, wv = O.prefill(*args, widen=False, layers=2)
    ek, ev = O.prefill(*args, widen=True, layers=2)
    for got, want, exact in ((k.cpu()[:2], wk, ek), (v.cpu()[:2], wv, ev)):
        d = O.band(want.float(), got.float(), exact.float())
        assert d["pass"], d
    pre.close()
