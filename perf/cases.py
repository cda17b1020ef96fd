"""The work that a user of this package has it do, as cases that can be timed and compared.

Three kinds of call, through the package's public entry points:

* ``chunk``    one action chunk for ``batch`` observations (``Pi05Arm``: bind once, ``launch()`` per chunk), 10 Euler
               steps x 18 expert layers over a prefix cache of ``prefix`` tokens; the cache is dense or a paged pool
               (``page`` tokens per page, 0 = dense) with a validity mask that is full, right-padded or scattered;
* ``prefill``  the Gemma-2B prefix prefill of ``prefix`` tokens (``Pi05Prefill.run``), which fills that cache;
* ``policy``   both in turn, as a controller calls them for a new observation: embeddings and mask in, actions out.

Inputs follow the package's fixture: weights and biases N(0, 0.02) for the action expert, N(0, 1 / fan_in) for the
prefill, unit-variance keys, values, embeddings and noise, and masks whose valid count is uniform in [prefix / 2, prefix].
They are drawn on the GPU from the seed.
"""
import math

import torch

from pi05_megakernel_b200 import fixture as FX
from pi05_megakernel_b200.arm import PagedPrefix, Pi05Arm
from pi05_megakernel_b200.prefill import Pi05Prefill

DEV = "cuda"
MIN_PREFIX, MAX_PREFIX = 16, 968      # 968 = 3 cameras x 256 image tokens + 200 prompt tokens
MAX_BATCH = 16
MASKS = ("full", "pad", "scatter")
PAGES = (0, 0, 64, 128)


def _chunk(name, prefix, batch=1, mask="full", page=0):
    return {"name": name, "kind": "chunk", "prefix": prefix, "batch": batch, "mask": mask, "page": page}


def _prefill(name, prefix, mask="pad"):
    return {"name": name, "kind": "prefill", "prefix": prefix, "batch": 1, "mask": mask, "page": 0}


def listed():
    return [
        # one robot, the headline latency: a short cached prefix
        _chunk("chunk-p128", 128),
        # one robot, three cameras and a full prompt, right-padded as the prompt builder pads it
        _chunk("chunk-p968-pad", 968, mask="pad"),
        # one robot, cache kept by a paged allocator, ragged last page, tokens dropped here and there
        _chunk("chunk-p301-paged", 301, mask="scatter", page=64),
        # the smallest prefix in use: a low-resolution single view
        _chunk("chunk-p40", 40, mask="scatter"),
        # two robots (or two candidate plans) on one GPU, full context
        _chunk("chunk-b2-p968", 968, batch=2, mask="pad"),
        # one camera, a handful of robots
        _chunk("chunk-b4-p256", 256, batch=4, mask="pad"),
        # simulation fleet, ragged prefix, paged cache
        _chunk("chunk-b7-p419-paged", 419, batch=7, mask="pad", page=128),
        # simulation fleet, short prefix: throughput
        _chunk("chunk-b16-p128", 128, batch=16),
        # the largest launch there is: sixteen observations with full context
        _chunk("chunk-b16-p968", 968, batch=16, mask="pad"),
        # a text-only or single low-resolution prefix
        _prefill("prefill-61", 61),
        # one camera without a prompt, every token valid
        _prefill("prefill-256", 256, mask="full"),
        # a new observation with full context: prefill, then the chunk on the cache it leaves
        {"name": "policy-p968", "kind": "policy", "prefix": 968, "batch": 1, "mask": "pad", "page": 0},
    ]


def draw(rng):
    kind = rng.choice(("chunk", "chunk", "fleet", "fleet", "prefill", "policy"))
    prefix = int(round(math.exp(rng.uniform(math.log(MIN_PREFIX), math.log(MAX_PREFIX)))))
    case = {"kind": kind, "prefix": min(max(prefix, MIN_PREFIX), MAX_PREFIX), "batch": 1, "mask": rng.choice(MASKS), "page": 0}
    if kind == "fleet":
        case["kind"], case["batch"] = "chunk", int(round(math.exp(rng.uniform(math.log(2), math.log(MAX_BATCH)))))
    if case["kind"] == "chunk":
        case["page"] = rng.choice(PAGES)
    elif case["mask"] == "scatter":
        case["mask"] = "pad"            # a prompt is padded on the right
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _mask(kind, n, g):
    """A validity mask of ``n`` tokens on the GPU."""
    if kind == "full":
        return torch.ones(n, dtype=torch.bool, device=DEV)
    valid = torch.randint(n // 2, n + 1, (1,), generator=g, device=DEV)
    order = torch.arange(n, device=DEV) if kind == "pad" else torch.randperm(n, generator=g, device=DEV)
    return order < valid


def _expert_weights(geo, g):
    out = {}
    for name, (shape, dtype) in FX.shapes(geo).items():
        if name not in FX.OBSERVATION:
            out[name] = torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, FX.WEIGHT_STD, generator=g)
    return out


def _prefill_weights(geo, g):
    out = {}
    for name in FX.PREFILL_WEIGHTS:
        shape, dtype = FX.prefill_shapes(geo)[name]
        std = 0.1 if name in ("ln1", "ln2") else shape[-1] ** -0.5
        out[name] = torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=g)
    return out


def _paged(dense, page, order):
    """A dense cache [batch, layers, tokens, 1, 256] as a pool of shuffled pages [pages, layers, page, 1, 256]."""
    batch, layers, tokens = dense.shape[:3]
    per = -(-tokens // page)
    padded = torch.zeros((batch, layers, per * page, 1, 256), dtype=dense.dtype, device=DEV)
    padded[:, :, :tokens] = dense
    pages = padded.view(batch, layers, per, page, 1, 256).transpose(1, 2).reshape(batch * per, layers, page, 1, 256)
    pool = torch.zeros((len(order), layers, page, 1, 256), dtype=dense.dtype, device=DEV)
    pool[torch.tensor(order[:batch * per], device=DEV)] = pages
    return pool


def _prepare_chunk(case, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    geo, batch = FX.Geometry(prefix=case["prefix"]), case["batch"]
    inputs = _expert_weights(geo, g)
    kv = (batch, geo.layers, geo.prefix, 1, 256)
    noise = torch.randn((batch, geo.horizon, geo.action_dim), generator=g, device=DEV)
    k = torch.empty(kv, dtype=torch.bfloat16, device=DEV).normal_(generator=g)
    v = torch.empty(kv, dtype=torch.bfloat16, device=DEV).normal_(generator=g)
    mask = torch.stack([_mask(case["mask"], geo.prefix, g) for _ in range(batch)])
    inputs["noise"], inputs["prefix_mask"] = (noise, mask) if batch > 1 else (noise[0], mask[0])
    arm = Pi05Arm(geo, "b200", DEV, batch=batch)
    pages = None
    if case["page"]:
        per = -(-geo.prefix // case["page"])
        order = torch.randperm(batch * per + 3, generator=torch.Generator().manual_seed(seed)).tolist()
        table = [order[b * per:(b + 1) * per] for b in range(batch)]
        pages = PagedPrefix(_paged(k, case["page"], order), _paged(v, case["page"], order), table)
    else:
        inputs["prefix_k"], inputs["prefix_v"] = (k, v) if batch > 1 else (k[0], v[0])
    arm.bind(inputs, kv_pages=pages)
    return {"kind": "chunk", "arm": arm}


def _prepare_prefill(case, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    geo = FX.PrefillGeometry(tokens=case["prefix"])
    prefill = Pi05Prefill(geo, DEV)
    prefill.bind(_prefill_weights(geo, g))
    embeddings = torch.empty((geo.tokens, geo.hidden), dtype=torch.bfloat16, device=DEV).normal_(generator=g)
    return {"kind": "prefill", "prefill": prefill, "embeddings": embeddings, "valid": _mask(case["mask"], geo.tokens, g)}


def _prepare_policy(case, seed):
    state = _prepare_prefill(case, seed)
    g = torch.Generator(DEV).manual_seed(seed ^ 0x5EED)
    geo = FX.Geometry(prefix=case["prefix"])
    inputs = _expert_weights(geo, g)
    cache = (geo.layers, geo.prefix, 1, 256)
    inputs["noise"] = torch.randn((geo.horizon, geo.action_dim), generator=g, device=DEV)
    inputs["prefix_k"] = torch.zeros(cache, dtype=torch.bfloat16, device=DEV)
    inputs["prefix_v"] = torch.zeros(cache, dtype=torch.bfloat16, device=DEV)
    inputs["prefix_mask"] = state["valid"]
    arm = Pi05Arm(geo, "b200", DEV)
    arm.bind(inputs)
    state.update(kind="policy", arm=arm, cache=(inputs["prefix_k"], inputs["prefix_v"]))
    return state


def prepare(case, seed):
    return {"chunk": _prepare_chunk, "prefill": _prepare_prefill, "policy": _prepare_policy}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    if state["kind"] == "chunk":
        state["arm"].launch()
        return state["arm"].outputs()["actions"]
    if state["kind"] == "prefill":
        return state["prefill"].run(state["embeddings"], state["valid"])
    keys, values = state["prefill"].run(state["embeddings"], state["valid"], out=state["cache"])
    state["arm"].launch()
    return {"keys": keys, "values": values, "actions": state["arm"].outputs()["actions"]}


# ------------------------------------------------------------------------------------------------ what a pass needs
def _work_chunk(case):
    """Every Euler step reads the expert's weights and the caches once (they exceed the L2), the FP32 layers once."""
    s = FX.sol(FX.Geometry(prefix=case["prefix"]), case["batch"])
    return s["bytes_restream"], s["flops"]


def _work_prefill(case):
    geo, tokens = FX.PrefillGeometry(tokens=case["prefix"]), case["prefix"]
    h, layers, inter = geo.hidden, geo.layers, geo.intermediate
    qd, kvd = geo.q_heads * geo.head_dim, geo.kv_heads * geo.head_dim
    attention, mlp = h * (qd + 2 * kvd) + qd * h, 3 * h * inter
    weights = layers * attention + (layers - 1) * mlp           # the last layer's MLP reaches no key or value
    flops = 2 * tokens * weights + layers * 4 * tokens * tokens * qd
    return 2 * weights + 2 * tokens * h + 4 * layers * tokens * kvd, flops


def work(case):
    total = [0, 0]
    if case["kind"] in ("chunk", "policy"):
        total = [a + b for a, b in zip(total, _work_chunk(case))]
    if case["kind"] in ("prefill", "policy"):
        total = [a + b for a, b in zip(total, _work_prefill(case))]
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    """BF16 activations through 18 layers.  The actions of a BF16 evaluation lie 2e-3 from the FP32 result, so two of
    them may be 5e-3 apart; the deepest keys and values of the prefill lie 1.3e-2 from it, two of them up to 2e-2."""
    if case["kind"] == "chunk":
        return {"rel": 5e-3, "max": 0.1}
    return {"rel": 2e-2, "max": 0.5}
