"""Host-side logic that needs no GPU: fixtures, variants, the C ABI's exports and argument checks."""
import ctypes
import os
import re

import pytest
import torch

from pi05_megakernel_b200 import _lib, build
from pi05_megakernel_b200 import fixture as FX
from pi05_megakernel_b200.arm import parse_variant

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.load()


def test_header_and_library_agree(lib):
    """Every function include/pi05_b200.h declares is exported, and nothing else is bound."""
    text = open(os.path.join(ROOT, "include", "pi05_b200.h")).read()
    declared = set(re.findall(r"\b(pi05_[a-z_]+)\s*\(", text))
    assert declared == set(_lib.SIGNATURES)
    for name in declared:
        assert hasattr(lib, name)


def test_error_strings(lib):
    assert lib.pi05_error_string(_lib.OK) == b"ok"
    for code in range(1, 7):
        assert lib.pi05_error_string(code) not in (b"ok", b"unknown error")
    assert lib.pi05_error_string(99) == b"unknown error"


def test_argument_errors_never_touch_a_gpu(lib):
    h = ctypes.c_void_p()
    assert lib.pi05_create(0, 128, 1, 0, 1, None) == _lib.ERR_ARGUMENT
    assert lib.pi05_create(-1, 128, 1, 0, 1, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    assert lib.pi05_create(0, 0, 1, 0, 1, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    assert lib.pi05_create(0, 128, 1, 2, 2, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    assert lib.pi05_create(0, 128, 17, 0, 1, ctypes.byref(h)) == _lib.ERR_UNSUPPORTED
    assert lib.pi05_create(0, 128, 1, 0, 3, ctypes.byref(h)) == _lib.ERR_UNSUPPORTED     # 2, 4 or 8 ranks
    assert lib.pi05_create(0, 128, 2, 0, 2, ctypes.byref(h)) == _lib.ERR_UNSUPPORTED     # one observation per launch
    n = ctypes.c_size_t()
    assert lib.pi05_workspace_bytes(None, ctypes.byref(n)) == _lib.ERR_ARGUMENT
    assert lib.pi05_launch(None, 10, 18, None, None) == _lib.ERR_ARGUMENT
    assert lib.pi05_destroy(None) == _lib.ERR_ARGUMENT
    if not torch.cuda.is_available():
        assert lib.pi05_create(0, 128, 1, 0, 1, ctypes.byref(h)) == _lib.ERR_NO_DEVICE
        assert not h.value


def test_prefill_argument_errors_never_touch_a_gpu(lib):
    """The prefill entry points check their arguments before they look for a device, and the Python wrapper has no CPU path."""
    h = ctypes.c_void_p()
    assert lib.pi05_prefill_create(0, 968, None) == _lib.ERR_ARGUMENT
    assert lib.pi05_prefill_create(-1, 968, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    assert lib.pi05_prefill_create(0, 0, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    assert lib.pi05_prefill_create(0, 4097, ctypes.byref(h)) == _lib.ERR_ARGUMENT
    n = ctypes.c_size_t()
    assert lib.pi05_prefill_workspace_bytes(None, ctypes.byref(n)) == _lib.ERR_ARGUMENT
    assert lib.pi05_prefill_run(None, None, None, 1, None, None, 18, None) == _lib.ERR_ARGUMENT
    assert lib.pi05_prefill_destroy(None) == _lib.ERR_ARGUMENT
    if not torch.cuda.is_available():
        assert lib.pi05_prefill_create(0, 968, ctypes.byref(h)) == _lib.ERR_NO_DEVICE
        assert not h.value
        from pi05_megakernel_b200.prefill import Pi05Prefill
        with pytest.raises(RuntimeError):
            Pi05Prefill(FX.PrefillGeometry(tokens=64), "cuda")


@pytest.mark.parametrize("sms", [148, 132])
@pytest.mark.parametrize("tokens", [1, 64, 129, 200, 256, 300, 512, 513, 968, 4096])
def test_prefill_plan(lib, sms, tokens):
    """The launch decisions of the prefill, and for a stream-K down projection the partition of (tile, k block) units over
    the CTAs: every unit exactly once, contiguous ranges of equal size (+-1), and for every tile cut over several CTAs one
    owner (the CTA that has its k block 0) followed by contributors that are the next CTAs' FIRST segments - the order
    that lets an owner wait for CTAs of higher index only while contributors wait for nobody."""
    info, count = (ctypes.c_int * 6)(), ctypes.c_int()
    assert lib.pi05_prefill_plan(sms, tokens, 0, info, None, 0, ctypes.byref(count)) == _lib.OK
    m_tiles, pairs, sk, tiles, kblocks, ctas = list(info)
    assert m_tiles == (tokens + 127) // 128 and pairs == (m_tiles >= 2) and sk == (m_tiles * 16 * 2 <= sms)
    if not sk:
        assert (tiles, kblocks, ctas, count.value) == (0, 0, 0, 0)
        return
    assert (tiles, kblocks, ctas) == (m_tiles * 8, 256, min(sms, m_tiles * 8 * 256))
    assert lib.pi05_prefill_plan(sms, tokens, ctas, info, None, 0, ctypes.byref(count)) == _lib.ERR_ARGUMENT
    per_cta = []
    for cta in range(ctas):
        buf = (ctypes.c_int * (3 * 8))()
        assert lib.pi05_prefill_plan(sms, tokens, cta, info, buf, 8, ctypes.byref(count)) == _lib.OK
        assert 1 <= count.value <= 8
        per_cta.append([tuple(buf[3 * i: 3 * i + 3]) for i in range(count.value)])
    units = [(t, kb) for segs in per_cta for (t, a, b) in segs for kb in range(a, b)]
    assert units == [(t, kb) for t in range(tiles) for kb in range(kblocks)]          # every unit once, in order
    sizes = [sum(b - a for (_t, a, b) in segs) for segs in per_cta]
    assert max(sizes) - min(sizes) <= 1
    for cta, segs in enumerate(per_cta):
        for i, (t, a, b) in enumerate(segs):
            assert i == 0 or a == 0                      # only a CTA's first segment can start inside a tile
            if a == 0 and b < kblocks:                   # owner of a tile that goes on in the following CTAs
                assert i == len(segs) - 1
                end, peer = b, cta + 1
                while end < kblocks:
                    pt, pa, pb = per_cta[peer][0]
                    assert (pt, pa) == (t, end) and pa > 0
                    end, peer = pb, peer + 1


@pytest.mark.parametrize("sms", [132, 148, 152])
def test_prefill_partials_fit_the_workspace(lib, sms):
    """A handle for up to max_tokens tokens holds the partial sums of every shorter prompt, whatever cut that one takes."""
    held, needed = ctypes.c_size_t(), ctypes.c_size_t()
    need = [0]
    for tokens in range(1, 4097):
        assert lib.pi05_prefill_partials(sms, tokens, tokens, ctypes.byref(held), ctypes.byref(needed)) == _lib.OK
        need.append(max(need[-1], needed.value))
        assert held.value >= need[tokens], tokens
    for args in ((1, 64, 64), (sms, 64, 65), (sms, 4097, 1), (sms, 64, 0)):
        assert lib.pi05_prefill_partials(*args, ctypes.byref(held), ctypes.byref(needed)) == _lib.ERR_ARGUMENT


@pytest.mark.parametrize("tokens", [1200, 1500, 2340, 2700, 3000, 4096])
def test_prefill_splits_no_k_where_tiles_fill_the_gpu(lib, tokens):
    """Long prompts leave one slice of partial sums per projection: their whole-K tiles occupy every SM."""
    held, needed = ctypes.c_size_t(), ctypes.c_size_t()
    assert lib.pi05_prefill_partials(148, tokens, tokens, ctypes.byref(held), ctypes.byref(needed)) == _lib.OK
    assert needed.value == tokens * 2048


@pytest.mark.parametrize("sms", [132, 148, 152])
def test_chunk_partials_fit_the_workspace(lib, sms):
    """An engine for (max_batch, max_prefix) holds the partial sums of every smaller batch and shorter prefix."""
    info, held, needed = (ctypes.c_int * 4)(), ctypes.c_size_t(), ctypes.c_size_t()

    def plan(mb, mp, b, p):
        assert lib.pi05_chunk_plan(sms, mb, mp, b, p, info, ctypes.byref(held), ctypes.byref(needed)) == _lib.OK
        return held.value, needed.value

    prefixes = sorted({p for c in range(32) for p in (c * 128 + 1, c * 128 + 77, c * 128 + 128)})
    need = {(b, p): plan(b, p, b, p)[1] for b in range(1, 17) for p in prefixes}
    for mb in range(1, 17):
        for mp in prefixes:
            most = max(n for (b, p), n in need.items() if b <= mb and p <= mp)
            assert plan(mb, mp, 1, 1)[0] >= most, (mb, mp)
    for args in ((1, 1, 64, 1, 64), (sms, 17, 64, 1, 64), (sms, 2, 64, 3, 64), (sms, 2, 64, 1, 65), (sms, 1, 4097, 1, 1)):
        assert lib.pi05_chunk_plan(*args, info, ctypes.byref(held), ctypes.byref(needed)) == _lib.ERR_ARGUMENT


def test_every_attention_cut_has_a_gpu_test(lib):
    """The sizes of the GPU tests reach every (query tokens, CTAs per tile, suffix in the last chunk of the prefix, with the O projection)
    that a B200 chooses for any batch, any prefix and a dense cache or pages of 64 or 128 tokens."""
    from tests.test_gpu_chain import ATTENTION_CUTS, ATTENTION_O, CUTS
    info = (ctypes.c_int * 5)()

    def cut(batch, prefix, page):
        assert lib.pi05_chunk_attention(148, batch, prefix, page or prefix, info) == _lib.OK
        return info[0], info[1], info[2], info[4]

    chosen = {cut(b, p, page) for b in range(1, 17) for p in range(1, 4097) for page in (0, 64, 128)}
    assert chosen == {cut(b, p, 0) for p, b, _mask, _variant in CUTS} | {cut(b, p, page) for p, b, page in ATTENTION_CUTS + ATTENTION_O}
    for args in ((1, 1, 64, 64), (148, 0, 64, 64), (148, 17, 64, 64), (148, 1, 0, 64), (148, 1, 4097, 4097), (148, 1, 64, 0), (148, 1, 200, 100)):
        assert lib.pi05_chunk_attention(*args, info) == _lib.ERR_ARGUMENT


# ms of an action chunk on a B200 by attention cut (query tokens, CTAs per tile, suffix joined), several cuts in turn in one process; (batch, prefix, page)
TIMED_CUTS = {
    (3, 552, 64): {(6, 4, 0): 6.72, (6, 4, 1): 6.79, (8, 4, 1): 6.87, (2, 1, 1): 7.29},
    (9, 960, 64): {(8, 2, 1): 10.50, (8, 2, 0): 10.62, (4, 1, 0): 11.05, (4, 1, 1): 11.08},
    (5, 574, 64): {(4, 1, 1): 7.53, (4, 2, 0): 7.55, (4, 2, 1): 7.68, (2, 1, 1): 7.86},
    (6, 768, 64): {(6, 2, 0): 8.91, (14, 4, 0): 9.17, (4, 1, 0): 9.26},
    (7, 703, 64): {(6, 2, 1): 8.90, (6, 2, 0): 9.02, (8, 2, 1): 9.17, (4, 1, 1): 9.31},
    (3, 576, 128): {(6, 4, 0): 6.72, (4, 2, 0): 6.78, (8, 4, 0): 6.89, (2, 1, 1): 6.98},
    (16, 959, 128): {(6, 1, 0): 12.62, (8, 1, 0): 12.75, (6, 1, 1): 12.76},
    (11, 958, 128): {(4, 1, 0): 11.11, (4, 1, 1): 11.22, (6, 1, 0): 11.37},
    (2, 259, 64): {(2, 1, 1): 5.30, (4, 1, 1): 5.32, (2, 1, 0): 5.45},
    (1, 191, 64): {(2, 1, 1): 4.54, (2, 1, 0): 4.63, (4, 1, 1): 4.65},
    (14, 190, 64): {(6, 1, 1): 10.02, (8, 1, 1): 10.15, (6, 1, 0): 10.20},
    (4, 808, 0): {(4, 2, 0): 7.04, (8, 4, 0): 7.06, (8, 4, 1): 7.15},
    (2, 680, 0): {(4, 4, 1): 5.65, (4, 4, 0): 5.67, (2, 2, 0): 5.86},
}


@pytest.mark.parametrize("batch,prefix,page", TIMED_CUTS)
def test_attention_cut_is_one_of_the_fastest_timed(lib, batch, prefix, page):
    """The cost model picks a cut within 0.8 % of the fastest one (runs of one cut differ by up to 0.4 %)."""
    info = (ctypes.c_int * 5)()
    assert lib.pi05_chunk_attention(148, batch, prefix, page or prefix, info) == _lib.OK
    timed = TIMED_CUTS[batch, prefix, page]
    assert timed.get(tuple(info)[:3], 1e9) <= 1.008 * min(timed.values())


@pytest.mark.parametrize("sms", [132, 148, 152])
def test_partials_of_paged_caches_fit_the_workspace(lib, sms):
    """The parts of a split attention over several pages, whose cuts are not those of a dense cache."""
    info, held, needed = (ctypes.c_int * 5)(), ctypes.c_size_t(), ctypes.c_size_t()
    plan = (ctypes.c_int * 4)()
    for batch in range(1, 17):
        most = 0
        for prefix in sorted({p for c in range(32) for p in (c * 128 + 1, c * 128 + 64, c * 128 + 72, c * 128 + 128)}):
            for page in (64, 128):
                assert lib.pi05_chunk_attention(sms, batch, prefix, page, info) == _lib.OK
                tokens, splits = info[0], info[1]
                if splits > 1:                              # a part: 8 rows per token, 256 dims, reference and sum
                    most = max(most, batch * -(-50 // tokens) * splits * tokens * 8 * 258)
            assert lib.pi05_chunk_plan(sms, batch, prefix, batch, prefix, plan, ctypes.byref(held), ctypes.byref(needed)) == _lib.OK
            assert held.value >= most, (batch, prefix)


def test_prefill_fixture_is_deterministic():
    geo = FX.PrefillGeometry(tokens=96, layers=1)
    shapes = FX.prefill_shapes(geo)
    assert set(FX.PREFILL_WEIGHTS) <= set(shapes) and shapes["ld"][0] == (1, 2048, 16384)
    a, b = FX.make_prefill_inputs(geo, 5, "pad"), FX.make_prefill_inputs(geo, 5, "pad")
    assert all(torch.equal(a[k], b[k]) for k in a)
    assert a["valid"].dtype == torch.bool and 48 <= int(a["valid"].sum()) <= 96
    assert bool(a["valid"][: int(a["valid"].sum())].all())          # right-padded: the valid tokens come first


def test_no_cpu_fallback():
    if torch.cuda.is_available():
        pytest.skip("GPU present")
    from pi05_megakernel_b200.arm import Pi05Arm
    with pytest.raises(RuntimeError):
        Pi05Arm(FX.Geometry(), "b200", "cuda")


def test_variants():
    assert parse_variant("b200") == {"steps": None, "layers": None}
    assert parse_variant("b200-s2-l3") == {"steps": 2, "layers": 3}
    for bad in ("k64", "b200-x", "b200-s2-s3", "b200-l"):
        with pytest.raises(ValueError):
            parse_variant(bad)


def test_fixture_shapes_and_determinism():
    geo = FX.Geometry(prefix=24, layers=2, hidden=64, intermediate=128, q_heads=2, head_dim=16)
    a, b = FX.make_inputs(geo, 5), FX.make_inputs(geo, 5)
    assert list(a) == list(FX.ORDER)
    for name, (shape, dtype) in FX.shapes(geo).items():
        assert tuple(a[name].shape) == tuple(shape) and a[name].dtype == dtype
        assert torch.equal(a[name], b[name])
    assert float(a["wq"].float().std()) == pytest.approx(0.02, rel=0.1)
    pad = FX.make_observation(geo, 5, "pad")["prefix_mask"]
    n = int(pad.sum())
    assert geo.prefix // 2 <= n <= geo.prefix and bool(pad[:n].all()) and not bool(pad[n:].any())
    sc = FX.make_observation(geo, 5, "scatter")["prefix_mask"]
    assert geo.prefix // 2 <= int(sc.sum()) <= geo.prefix


def test_bind_view_argument_errors(lib):
    view = _lib.KvView()
    ptrs = (ctypes.c_void_p * _lib.NUM_INPUTS)()
    assert lib.pi05_bind_view(None, ptrs, ctypes.byref(view), 128, 1, None, None, 0) == _lib.ERR_ARGUMENT
    assert lib.pi05_bind(None, ptrs, 128, 1, None, None, 0) == _lib.ERR_ARGUMENT


STAGES = {0: 8, 1: 16, 2: 8, 3: 32}          # 128-k stages of the full K of QKV, O, gate/up, down
TILES = {0: 20, 1: 8, 2: 64, 3: 8}           # 128-row weight tiles (QKV: 16 q + 2 k + 2 v)


@pytest.mark.parametrize("batch,prefix", [(1, 128), (1, 968), (2, 128), (3, 128), (4, 128), (5, 128), (7, 128),
                                          (8, 128), (12, 128), (16, 128)])
def test_schedule_plan_invariants(lib, batch, prefix, monkeypatch):
    """The work schedule of the GEMM CTAs on a 148-SM part, computed on the host.  Whatever the batch: every
    (GEMM, group of observations, tile) is covered over its whole K exactly once; the units per observation that
    the stage counters wait for are the same for every group; no row CTA appears; and with named groups every
    CTA's list follows one global order (cycle position, then group), which is what rules out circular waits."""
    for name in ("PI05_OBS_PER_MMA", "PI05_LATENCY_SCHEDULE", "PI05_ONE_STREAM", "PI05_ROW_GROUPS", "PI05_KEY_GROUPS"):
        monkeypatch.delenv(name, raising=False)
    entries, plan = _lib.schedule_plan(148, batch, prefix)
    ngroups = plan["groups"]
    assert ngroups == (batch + plan["obs_per_mma"] - 1) // plan["obs_per_mma"]
    assert plan["gemm_ctas"] == 148 - 25 * max(plan["row_groups"], plan["key_groups"])
    cover: dict = {}
    per_cta: dict = {}
    for cta, gemm, lag, group, tile, k0, nk in entries:
        assert 0 <= cta < plan["gemm_ctas"] and nk >= 1 and 0 <= tile < TILES[gemm]
        groups = range(ngroups) if group < 0 else [group]
        for g in groups:
            cover.setdefault((gemm, g, tile), []).append((k0, nk))
        per_cta.setdefault(cta, []).append((gemm, lag, group))
    for gemm in range(4):
        for g in range(ngroups):
            units = 0
            for tile in range(TILES[gemm]):
                runs = sorted(cover[(gemm, g, tile)])
                units += len(runs)
                pos = 0
                for k0, nk in runs:                       # contiguous, no overlap, whole K
                    assert k0 == pos
                    pos += nk
                assert pos == STAGES[gemm]
            assert units == list(plan["units"].values())[gemm]
    assert max(len(v) for v in per_cta.values()) <= 32
    if batch >= 5:
        assert plan["stream_split"] == (ngroups + 1) // 2
    named = [e for e in entries if e[3] >= 0]
    assert bool(named) == (batch >= 3)
    if named:
        split = plan["stream_split"]

        def position(gemm, lag, group):
            if not split:
                return (gemm, group)
            b = group >= split
            assert lag == (1 if b and gemm >= 2 else 0)
            # q(A) gate/up(B) O(A) down(B) gate/up(A) q(B) down(A) O(B)
            order = {(0, False): 0, (2, True): 1, (1, False): 2, (3, True): 3, (2, False): 4, (0, True): 5,
                     (3, False): 6, (1, True): 7}
            return (order[(gemm, b)], group)
        for cta, lst in per_cta.items():
            keys = [position(*e) for e in lst]
            assert keys == sorted(keys), (cta, lst)


def test_schedule_plan_argument_errors(lib):
    count, info = ctypes.c_int(), (ctypes.c_int * _lib.PLAN_INFO)()
    assert lib.pi05_schedule_plan(148, 0, 128, None, None, 0, ctypes.byref(count), info) == _lib.ERR_ARGUMENT
    assert lib.pi05_schedule_plan(148, 17, 128, None, None, 0, ctypes.byref(count), info) == _lib.ERR_ARGUMENT
    assert lib.pi05_schedule_plan(148, 1, 128, None, None, 4, ctypes.byref(count), info) == _lib.ERR_ARGUMENT
    assert lib.pi05_schedule_plan(148, 1, 128, None, None, 0, None, info) == _lib.ERR_ARGUMENT
    assert lib.pi05_schedule_plan(60, 1, 128, None, None, 0, ctypes.byref(count), info) == _lib.ERR_UNSUPPORTED


@pytest.mark.parametrize("sms", list(range(132, 161, 2)))
@pytest.mark.parametrize("batch,prefix", [(1, 128), (1, 968), (5, 128), (16, 128)])
def test_schedule_plan_on_other_sm_counts(lib, sms, batch, prefix):
    """Parts with a few SMs more or fewer than 148: the plan sheds groups of row CTAs until the GEMM side keeps the
    fewest CTAs a schedule needs, instead of refusing."""
    count, info = ctypes.c_int(), (ctypes.c_int * _lib.PLAN_INFO)()
    assert lib.pi05_schedule_plan(sms, batch, prefix, None, None, 0, ctypes.byref(count), info) == _lib.OK
    assert info[0] >= 72 and info[0] == sms - 25 * max(info[1], info[2])


def test_tuning_defaults_and_clamping(lib):
    t = _lib.Tuning()
    assert lib.pi05_tuning_defaults(ctypes.byref(t)) == _lib.OK
    assert (t.poll_ns, t.two_streams, t.grouped_from, t.streams_from, t.clusters) == (20, 1, 3, 5, 1)
    assert lib.pi05_tuning_defaults(None) == _lib.ERR_ARGUMENT
    assert lib.pi05_tune(None, ctypes.byref(t)) == _lib.ERR_ARGUMENT
    # the plan follows the struct, not the environment
    count, info = ctypes.c_int(), (ctypes.c_int * _lib.PLAN_INFO)()
    t.two_streams = 0
    assert lib.pi05_schedule_plan(148, 8, 128, ctypes.byref(t), None, 0, ctypes.byref(count), info) == _lib.OK
    assert info[5] == 0
    t.two_streams, t.row_groups = 1, 99          # out of range: clamped to 3
    assert lib.pi05_schedule_plan(148, 8, 128, ctypes.byref(t), None, 0, ctypes.byref(count), info) == _lib.OK
    assert info[5] == 4 and info[1] == 3


@pytest.mark.parametrize("size", [2, 4, 8])
def test_tensor_parallel_plans_partition_the_work(lib, size):
    """The ranks' schedules together cover exactly the one-GPU schedule's work: the q tiles, the K range of the O
    projection, the gate/up tiles and the K range of the down projection are cut into `size` disjoint shares, rank r
    taking share r (heads 8 r / size .., MLP columns 4096 r / size ..); the k / v tiles run on every rank."""
    cover: dict = {}
    for rank in range(size):
        entries, plan = _lib.schedule_plan(148, 1, 128, rank, size)
        assert plan["gemm_ctas"] == 123
        mine: dict = {}
        for cta, gemm, lag, group, tile, k0, nk in entries:
            assert lag == 0 and group == -1
            for k in range(k0, k0 + nk):
                mine.setdefault((gemm, tile), []).append(k)
        for (gemm, tile), ks in mine.items():
            assert len(ks) == len(set(ks))
            if gemm == 0 and tile >= 16:
                assert sorted(ks) == list(range(STAGES[0]))               # k / v: the whole K on every rank
                continue
            if gemm == 0:
                assert tile // (16 // size) == rank and sorted(ks) == list(range(STAGES[0]))
            elif gemm == 2:
                assert tile // (64 // size) == rank and sorted(ks) == list(range(STAGES[2]))
            else:
                share = STAGES[gemm] // size
                assert sorted(ks) == list(range(rank * share, (rank + 1) * share))
            for k in ks:
                assert (gemm, tile, k) not in cover
                cover[(gemm, tile, k)] = rank
        assert plan["units"]["qkv"] == 4 + (16 // size) * 4
    for gemm in range(4):
        tiles = 16 if gemm == 0 else TILES[gemm]
        assert sum(1 for key in cover if key[0] == gemm) == tiles * STAGES[gemm]
    count, info = ctypes.c_int(), (ctypes.c_int * _lib.PLAN_INFO)()
    assert lib.pi05_schedule_plan_tp(148, 1, 128, 2, 2, None, None, 0, ctypes.byref(count), info) == _lib.ERR_ARGUMENT
    assert lib.pi05_schedule_plan_tp(148, 2, 128, 0, 2, None, None, 0, ctypes.byref(count), info) == _lib.ERR_UNSUPPORTED
    assert lib.pi05_schedule_plan_tp(148, 1, 128, 0, 3, None, None, 0, ctypes.byref(count), info) == _lib.ERR_UNSUPPORTED


def test_reference_arm_prints_the_contract_line():
    """`bench.py --impl reference` runs on the host cores alone: the reference's own eager path where it is installed
    beside the benchmark, else the oracle port; its one JSON line carries the keys the driver of the benchmark reads."""
    import json
    import subprocess
    import sys
    proc = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "3"],
                          capture_output=True, text=True, timeout=900, cwd=ROOT)
    assert proc.returncode == 0, proc.stderr[-2000:]
    lines = [l for l in proc.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["unit"] == "chunks/s" and d["higher_is_better"] is True and d["n_gpus"] == 1
    assert d["steps"] == 1 and d["warmup"] >= 3 and d["value"] > 0 and abs(d["value"] * d["ms_per_step"] - 1e3) < 1e-6 * 1e3
    assert d["cpu_baseline"]["kind"] in ("reference", "port") and d["cpu_baseline"]["cores"] >= 1
    assert d["cpu_baseline"]["value"] == d["value"]
    assert d["e2e"] == {"value": d["value"], "unit": "chunks/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
    assert "workload" in d["config"]
