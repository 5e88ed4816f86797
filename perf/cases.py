"""What the performance of this framework is measured on: the calls that a serving engine and an
accuracy study make, each through its public entry point, from one request to a full batch.

A case is a dict of plain values with a ``kind``:

* ``decode``   one decode step of a stack of layers, one slot-indexed call per layer;
* ``verify``   T speculative tokens per request through the multi-token call, a stack of layers;
* ``handoff``  a prefill chunk: the slots' state out of the pool in floating point, the final state back in;
* ``events``   cache events of a scheduler: preempt, prefix fork, checkpoint, roll back, resume;
* ``step``     one fused step through the statequant op (fresh outputs);
* ``chain``    T chained steps from a floating-point state through the statequant decode;
* ``fp32``     the unquantised step, the yardstick of every accuracy run.

``prepare`` makes the inputs and the state on the GPU from the seed, ``run`` is one pass, ``work`` the bytes
and operations that it cannot do without, ``tolerance`` how far another correct implementation may be off.
"""

import math

import torch

from carrykernel_b200.cuda import binding
from carrykernel_b200.statequant import kernel as sq
from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
from carrykernel_b200.vllm_integration import state_pool
from carrykernel_b200.vllm_integration.state_cache import SlotCache

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
RES = {"fp32": sq.RES_FP32, "fp16": sq.RES_FP16, "fp8": sq.RES_FP8, "int8": sq.RES_INT8, "int4": sq.RES_INT4,
       "none": sq.RES_NONE}
SLOT_RES = {"int8": qpd.RESID_INT8, "int4": qpd.RESID_INT4}
RES_BYTES = {"fp32": 4.0, "fp16": 2.0, "fp8": 1.0, "int8": 1.0, "int4": 0.5, "none": 0.0}
STATE_STEP = 2e-3        # a typical state scale: values of about 0.1 at 8 bits


def _slot(name, kind, layers, requests, heads=32, key_heads=32, dim=128, resid="int4", rscale="head",
          act="bf16", slots=0, pad=0, **more):
    return dict(name=name, kind=kind, layers=layers, requests=requests, heads=heads, key_heads=key_heads, dim=dim,
                resid=resid, rscale=rscale, act=act, slots=slots or requests + 1, pad=pad, **more)


def _dense(name, kind, requests, heads=32, dim=128, resid="int8", rscale="v", sscale="v", bits=8, act="bf16", **more):
    return dict(name=name, kind=kind, requests=requests, heads=heads, dim=dim, resid=resid, rscale=rscale,
                sscale=sscale, bits=bits, act=act, **more)


def listed():
    return [
        # one interactive user: every layer of the model waits for a call on a single request
        _slot("decode_1", "decode", 24, 1, slots=33),
        # the serving step: 64 requests scattered over a pool of 256 slots, 24 layers
        _slot("decode_64", "decode", 24, 64, slots=257),
        # the largest batch of the sweep, a few layers of it
        _slot("decode_512", "decode", 4, 512, slots=513),
        # a batch that the engine padded to its graph size, two value heads per key head, and the call's
        # defaults (int8 residual, one scale per V row)
        _slot("decode_ragged_int8", "decode", 12, 40, key_heads=16, resid="int8", rscale="v", slots=101, pad=3),
        # a model with narrow heads, fp16 activations
        _slot("decode_narrow", "decode", 12, 48, heads=16, key_heads=8, dim=64, resid="int8", rscale="v", act="fp16",
              slots=65),
        # checking four speculated tokens of every request in one call
        _slot("verify_4", "verify", 8, 32, key_heads=16, tokens=4, slots=65),
        # a chunk of a chunked prefill: 16 requests' state out in fp32 and the new state back in, error kept
        _slot("handoff_16", "handoff", 8, 16, slots=65, state="fp32", keep_error=True),
        # the scheduler under memory pressure: preemption, prefix fork, rejected speculation
        _slot("events_4", "events", 12, 4, slots=33),
        # a single layer of a 4B hybrid model: 8 slots, int8 residual with one scale per head
        _dense("step_8_int8", "step", 8, rscale="head"),
        # the bit-width study's plain arm: uniform 4-bit grid, one scale per head, no error feedback
        _dense("step_256_plain", "step", 256, resid="none", sscale="head", bits=4, act="fp32"),
        # its other arm: T chained steps with per-V scales and the op's default fp32 residual
        _dense("chain_64", "chain", 64, resid="fp32", act="fp32", tokens=8),
        # the unquantised recurrence that both are compared with
        _dense("fp32_96", "fp32", 96, resid="none", act="fp32"),
    ]


# No drawn case moves more than the largest listed one.
MOST_BYTES = 512 * 4 * 32 * 51216


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_once(rng):
    kind = rng.choice(["decode", "decode", "decode", "verify", "handoff", "events", "step", "step", "chain", "fp32"])
    dim = rng.choice([128, 128, 128, 64])
    heads = rng.choice([8, 12, 16, 24, 32, 48])
    if kind in ("decode", "verify", "handoff", "events"):
        requests = _log_int(rng, 1, {"decode": 512, "verify": 96, "handoff": 64, "events": 8}[kind])
        layers = _log_int(rng, 1, 12 if kind == "events" else 24)
        c = _slot("", kind, layers, requests, heads=heads, key_heads=heads // rng.choice([1, 1, 2, 4]), dim=dim,
                  resid=rng.choice(["int4", "int8"]), rscale=rng.choice(["head", "v"]),
                  act=rng.choice(["bf16", "bf16", "fp16", "fp32"]), slots=requests + 1 + rng.randrange(2, 40))
        if kind == "decode":
            c["pad"] = rng.randrange(0, 1 + requests // 8)
        elif kind == "verify":
            c["tokens"] = rng.randrange(2, 7)
            c["dim"] = 128
        elif kind == "handoff":
            c["state"], c["keep_error"] = rng.choice(["fp32", "bf16", "fp16"]), rng.random() < 0.5
        else:
            c["slots"] = 3 * requests + 8
    elif kind == "chain":
        c = _dense("", kind, _log_int(rng, 1, 64), heads=heads, resid=rng.choice(["fp32", "fp32", "fp16", "fp8"]),
                   bits=rng.choice([3, 4, 5, 6, 8]), act=rng.choice(["fp32", "bf16"]), tokens=rng.randrange(2, 9))
    elif kind == "step":
        resid = rng.choice(["int8", "int4", "none"])
        c = _dense("", kind, _log_int(rng, 1, 256), heads=heads, dim=dim, resid=resid, rscale=rng.choice(["v", "head"]),
                   sscale=rng.choice(["v", "head"]) if resid == "none" else "v", bits=rng.choice([4, 6, 8, 8]),
                   act=rng.choice(["bf16", "fp16", "fp32"]))
    else:
        c = _dense("", kind, _log_int(rng, 1, 128), heads=heads, dim=dim, resid="none", act=rng.choice(["fp32", "bf16"]))
    del c["name"]
    return c


def draw(rng):
    while True:
        c = _draw_once(rng)
        if work(c)["bytes"] <= MOST_BYTES:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gauss_codes(shape, sigma, qmax, g):
    """int8 codes of a state whose rows fill the grid: normal, rounded, clamped."""
    out = torch.empty(shape, dtype=torch.int8, device=DEV)
    for part in out:                                    # leading index by index: bounds the fp32 scratch
        part.copy_(torch.empty(part.shape, device=DEV).normal_(0.0, sigma, generator=g).round_().clamp_(-qmax, qmax))
    return out


def _nibbles(shape, g):
    """Packed int4 residual codes, uniform in -7..7 (a rounding error is uniform within its step)."""
    out = torch.empty(shape, dtype=torch.int8, device=DEV)
    for part in out:
        lo = torch.randint(-7, 8, part.shape, dtype=torch.int8, device=DEV, generator=g)
        hi = torch.randint(-7, 8, part.shape, dtype=torch.int8, device=DEV, generator=g)
        part.copy_((lo & 15) | (hi << 4))
    return out


def _uniform(shape, g, lo=0.5, hi=1.5):
    return torch.empty(shape, device=DEV).uniform_(lo, hi, generator=g)


def _pools(c, g):
    """The pools of all layers, one tensor per kind with the layer in front."""
    L, S, HV, D = c["layers"], c["slots"], c["heads"], c["dim"]
    codes = _gauss_codes((L, S, HV, D, D), 42.0, 127, g)
    sscale = _uniform((L, S, HV, D), g).mul_(STATE_STEP)
    if c["resid"] == "int4":
        resid, levels = _nibbles((L, S, HV, D, D // 2), g), 14.0
    else:
        resid, levels = torch.empty((L, S, HV, D, D), dtype=torch.int8, device=DEV), 254.0
        for part in resid:
            part.copy_(torch.randint(-127, 128, part.shape, dtype=torch.int8, device=DEV, generator=g))
    rscale = sscale / levels if c["rscale"] == "v" else _uniform((L, S, HV), g, 1.2, 1.5).mul_(STATE_STEP / levels)
    return codes, sscale, resid, rscale


def _slots(c, g):
    """Slot ids in random order; the last ``pad`` entries are padding."""
    idx = (torch.randperm(c["slots"] - 1, device=DEV, generator=g)[:c["requests"]] + 1).to(torch.int32)
    if c["pad"]:
        idx[-c["pad"]:] = 0
    return idx


def _activations(c, g, tokens):
    L, B, H, HV, D = c["layers"], c["requests"], c["key_heads"], c["heads"], c["dim"]
    dt = DTYPES[c["act"]]
    lead = (L, B) if tokens is None else (L, B, tokens)
    mixed = torch.empty((*lead, 2 * H * D + HV * D), device=DEV).normal_(generator=g).to(dt)
    a = torch.empty((*lead, HV), device=DEV).normal_(generator=g).to(dt)
    b = torch.empty((*lead, HV), device=DEV).normal_(generator=g).to(dt)
    out = torch.zeros((L, B, tokens or 1, HV, D), dtype=dt, device=DEV)
    return mixed, a, b, out


def _dense_inputs(c, g, lead):
    """q, k (unit length), v, decay exp(-0.1 softplus(N(0,1))), write strength sigmoid(N(0,1))."""
    HV, D, dt = c["heads"], c["dim"], DTYPES[c["act"]]
    normal = lambda *shape: torch.empty(shape, device=DEV).normal_(generator=g)  # noqa: E731
    q, k = (torch.nn.functional.normalize(normal(*lead, HV, D), dim=-1).to(dt) for _ in range(2))
    v = normal(*lead, HV, D).to(dt)
    alpha = torch.exp(-0.1 * torch.nn.functional.softplus(normal(*lead, HV)))
    return q, k, v, alpha, torch.sigmoid(normal(*lead, HV))


def prepare(case, seed):
    c = dict(case)
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    st = {"case": c}
    B, HV, D = c["requests"], c["heads"], c["dim"]
    if c["kind"] in ("decode", "verify"):
        st["pools"] = _pools(c, g)
        st["layer_pools"] = list(zip(*st["pools"]))
        st["idx"] = _slots(c, g)
        mixed, a, b, st["out"] = _activations(c, g, c.get("tokens"))
        st["layers"] = list(zip(mixed, a, b, st["out"], st["layer_pools"]))
        st["A_log"] = torch.full((HV,), math.log(0.1), device=DEV)
        st["dt_bias"] = torch.zeros(HV, device=DEV)
    elif c["kind"] == "handoff":
        st["pools"] = _pools(c, g)
        st["layer_pools"] = list(zip(*st["pools"]))
        st["idx"] = _slots(c, g)
        dt = DTYPES[c["state"]]
        st["initial"] = torch.zeros((c["layers"], B, HV, D, D), dtype=dt, device=DEV)
        st["final"] = torch.empty((c["layers"], B, HV, D, D), dtype=dt, device=DEV)
        for part in st["final"]:
            part.copy_(torch.empty(part.shape, device=DEV).normal_(0.0, 0.1, generator=g))
    elif c["kind"] == "events":
        cache = SlotCache(c["layers"], c["slots"], HV, D, D, DEV, resid_fmt=SLOT_RES[c["resid"]],
                          resid_scale=c["rscale"], spill_slots=2 * B + 2)
        for pool, made in zip(cache.pools, zip(*_pools(c, g))):
            for to, of in zip(pool, made):
                to.copy_(of)
        for n in range(2 * B):
            cache.allocate(n)
        st["cache"] = cache
    elif c["kind"] == "step":
        qmax = 2 ** (c["bits"] - 1) - 1
        codes = _gauss_codes((B, HV, D, D), qmax / 3.0, qmax, g)
        scale = _uniform((B, HV, D) if c["sscale"] == "v" else (B, HV), g).mul_(0.254 / qmax)
        e = e_scale = None
        if c["resid"] == "int4":
            e, levels = _nibbles((B, HV, D, D // 2), g), 14.0
        elif c["resid"] == "int8":
            e, levels = torch.randint(-127, 128, (B, HV, D, D), dtype=torch.int8, device=DEV, generator=g), 254.0
        if e is not None:
            e_scale = scale / levels if c["rscale"] == "v" else scale.amax(-1) / levels
        st["args"] = (codes, scale, e, e_scale, *_dense_inputs(c, g, (B,)))
    elif c["kind"] == "chain":
        st["h0"] = torch.empty((B, HV, D, D), device=DEV).normal_(0.0, 0.1, generator=g)
        st["args"] = _dense_inputs(c, g, (c["tokens"], B))
    else:
        st["h"] = torch.empty((B, HV, D, D), device=DEV).normal_(0.0, 0.1, generator=g)
        st["args"] = _dense_inputs(c, g, (B,))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    c = state["case"]
    if c["kind"] in ("decode", "verify"):
        call = (qpd.quantized_gated_delta_rule_packed_decode if c["kind"] == "decode"
                else qpd.quantized_gated_delta_rule_packed_decode_multi)
        A_log, dt_bias, idx = state["A_log"], state["dt_bias"], state["idx"]
        fmt, qscale = SLOT_RES[c["resid"]], c["dim"] ** -0.5
        for mixed, a, b, out, pool in state["layers"]:
            call(mixed, a, b, A_log, dt_bias, qscale, *pool, out, idx, use_qk_l2norm_in_kernel=True, resid_fmt=fmt)
        return {"out": state["out"], "pools": state["pools"]}
    if c["kind"] == "handoff":
        fmt, idx = SLOT_RES[c["resid"]], state["idx"]
        for pool, h_in, h_out in zip(state["layer_pools"], state["initial"], state["final"]):
            state_pool.load_state(pool, idx, out=h_in, resid_fmt=fmt)
            state_pool.store_state(h_out, pool, idx, resid_fmt=fmt, keep_error=c["keep_error"])
        return {"initial": state["initial"], "pools": state["pools"]}
    if c["kind"] == "events":
        cache, n = state["cache"], c["requests"]
        for r in range(n):                               # room for newcomers
            cache.preempt(r)
        for r in range(n):                               # that share a prefix with a running request
            cache.fork(n + r, ("new", r))
        marks = [cache.checkpoint(("new", r)) for r in range(n)]
        for r in range(n):
            cache.resume(r)
        for mark in marks:                               # whose speculation is rejected
            cache.rollback(mark)
        idx = cache.indices(range(2 * n), pad_to=2 * n + 1)
        for r in range(n):
            cache.free(("new", r))
        return {"pools": cache.pools, "indices": idx}
    if c["kind"] == "step":
        return binding.gdn_quant_step_cuda(*state["args"], bits=c["bits"], res_fmt=RES[c["resid"]],
                                           resid_scale=c["rscale"], state_scale=c["sscale"])
    if c["kind"] == "chain":
        return binding.gdn_quant_decode_cuda(state["h0"], *state["args"], c["tokens"], bits=c["bits"],
                                             res_fmt=RES[c["resid"]])
    return binding.gdn_fp32_step_cuda(state["h"], *state["args"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far results may be off
# ---------------------------------------------------------------------------

def work(case):
    c = case
    B, HV, D = c["requests"], c["heads"], c["dim"]
    el = D * D
    per_v = lambda what: D * 4 if c.get(what, "v") == "v" else 4  # noqa: E731
    tile = el + el * RES_BYTES[c["resid"]]               # codes and residual of one (request, head), one way
    scales = per_v("sscale") + (per_v("rscale") if c["resid"] in ("int8", "int4") else 0)
    kind, act = c["kind"], SIZE[c["act"]]
    step_flops = 12.0 * el                               # two dot products, rank-1 write, decay, feedback, two roundings
    if kind in ("decode", "verify"):
        T, live = c.get("tokens", 1), B - c["pad"]
        vecs = T * (3 * D * act + 2 * act + D * act)     # q, k, v, the two gates, the output row
        return {"bytes": c["layers"] * (live * HV * (2 * (tile + scales) + vecs) + 4 * B),
                "flops": c["layers"] * live * HV * T * step_flops}
    if kind == "handoff":
        # out: slot read, state written; in: state read, slot written
        return {"bytes": c["layers"] * B * HV * 2.0 * (tile + scales + el * SIZE[c["state"]]),
                "flops": c["layers"] * B * HV * 8.0 * el}
    if kind == "events":
        return {"bytes": c["layers"] * 5.0 * B * HV * 2 * (tile + scales), "flops": 0.0}
    vecs = 3 * D * act + 8 + D * 4
    if kind == "step":
        return {"bytes": B * HV * (2.0 * (tile + scales) + vecs), "flops": B * HV * step_flops}
    if kind == "chain":
        T = c["tokens"]                                  # every step hands its state to the next call
        return {"bytes": B * HV * (el * 4.0 + tile + scales + T * (2.0 * (tile + scales) + vecs)),
                "flops": B * HV * T * step_flops}
    return {"bytes": B * HV * (8.0 * el + vecs), "flops": B * HV * 8.0 * el}


def tolerance(case):
    """Codes are rounded quotients of fp32 sums, so another order of summation flips the ones at a tie:
    about 2e-6 of the state codes, 3e-5 of the int4 and 4e-4 of the int8 residual codes per step, and a flip
    is carried on by the steps after it.  A bf16 output is off by one unit in the last place at most."""
    kind = case["kind"]
    if kind == "events":
        return "exact"                                   # copies
    if kind == "handoff":
        return {"rel": 1e-6, "differ": 1e-5}             # every rounding is defined
    if kind == "chain":
        return {"rel": 1e-4, "differ": 1e-4}
    if kind == "fp32":
        return {"rel": 1e-5}
    differ = 2e-3 if case["resid"] == "int8" else 1e-3
    if kind == "verify":
        differ *= 3
    if kind in ("decode", "verify") and case["act"] != "fp32":
        return {"rel": 2e-3, "max": 2e-2, "differ": differ}
    return {"rel": 1e-4, "max": 1e-2, "differ": differ}
