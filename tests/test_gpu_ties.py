"""State codes at and beside rounding ties on 128- and 64-wide heads: not one may differ from round_half_even(target / scale).

The kernels round by a reciprocal of the scale and decide again where a remainder lies within a guard of half a step.
Scales here are odd multiples of a power of two, 17 bits long, so that their reciprocals are not exact, and targets are
``code * scale + (scale -+ ulp) / 2``, up to half a unit in the last place of the quotient beside a tie.  Every product and sum up to
the target is exact in fp32 (whole numbers below 2^24, times a power of two), so the order in which a kernel takes them
does not matter and the oracle's codes are the only right ones; rounding by the best fp32 reciprocal gets one in six wrong,
as each test makes sure of first."""

from __future__ import annotations

import pytest
import torch

from oracle import gdn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
UNIT = 2.0 ** -30


def _halves(lead, g, lo=32769, hi=43000):
    """A residual step per head; the scales beside twice of it: S = 2 E - 1, 2 E, 2 E + 1 make ties and their neighbours."""
    return torch.randint(lo, hi, lead, generator=g)


def _codes_and_signs(shape, qmax, g):
    """Codes 0..qmax-1 along the last axis, a residual of one step up or down; one element holds the largest code."""
    n = shape[-1]
    c = (torch.arange(n) % qmax).expand(shape).clone()
    r = torch.randint(0, 2, shape, generator=g) * 2 - 1
    at = torch.randint(0, n, (*shape[:-1], 1), generator=g)
    c.scatter_(-1, at, qmax)
    r.scatter_(-1, at, 0)
    sign = torch.randint(0, 2, shape, generator=g) * 2 - 1
    return c * sign, r * sign


def _rows(lead, edge, qmax, seed, exact=False, lo=32769, hi=43000):
    """``(codes, residual codes, S, E)`` of rows ``[*lead, edge (row), edge (along the scale's axis)]``."""
    g = torch.Generator().manual_seed(seed)
    E = _halves(lead, g, lo, hi)
    S = 2 * E[..., None] + (0 if exact else 1) * torch.randint(-1, 2, (*lead, edge), generator=g)
    c, r = _codes_and_signs((*lead, edge, edge), qmax, g)
    return c, r, S, E


def _reciprocal_misses(target, scale, want):
    """The inputs can tell: the best fp32 reciprocal, without a second look, gets some of the codes wrong."""
    plain = torch.round(target.double() * (1.0 / scale).double())
    assert int((plain != want.double()).sum()) > want.numel() // 20


@pytest.mark.parametrize("edge,T", [(128, None), (128, 1), (64, None)])       # streaming, multi-token, 64-wide kernel
@pytest.mark.parametrize("resid_fmt", [orc.RESID_INT8, orc.RESID_INT4])
@pytest.mark.parametrize("rscale", ["v", "head"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_slot_layout(edge, T, resid_fmt, rscale, dtype):
    from carrykernel_b200 import _lib
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    B, H, HV = 5, 4, 8
    c, r, S, E = _rows((B + 1, HV), edge, 127, seed=edge)
    es = (E * UNIT).float()
    pool = [c.to(torch.int8), (S * UNIT).float(), (orc.pack_int4(r) if resid_fmt == orc.RESID_INT4 else r.to(torch.int8)),
            es if rscale == "head" else es[..., None].expand(B + 1, HV, edge).contiguous()]
    lead = (B,) if T is None else (B, T)
    mixed = torch.zeros(*lead, (2 * H + HV) * edge, dtype=dtype)         # k = v = 0: nothing is written
    a = b = torch.full((*lead, HV), -60.0, dtype=dtype)                  # a decay of exactly 1
    zeros, idx = torch.zeros(HV), torch.tensor([4, 1, 5, 2, 3], dtype=torch.int32)
    want = [x.clone() for x in pool]
    orc.packed_decode_step(mixed.reshape(B, -1), a.reshape(B, HV), b.reshape(B, HV), zeros, zeros, 1.0, *want,
                           torch.empty(B, 1, HV, edge, dtype=dtype), idx, resid_fmt=resid_fmt)
    assert torch.equal(want[1][1:], pool[1][1:])                         # the largest code pins the scale
    _reciprocal_misses(((c * S[..., None] + r * E[..., None, None]) * UNIT).float()[1:], pool[1][1:, ..., None], want[0][1:])
    got = [x.to(DEV) for x in pool]
    out = torch.empty(B, T or 1, HV, edge, dtype=dtype, device=DEV)
    call = qpd.quantized_gated_delta_rule_packed_decode if T is None else qpd.quantized_gated_delta_rule_packed_decode_multi
    call(*(x.to(DEV) for x in (mixed, a, b, zeros, zeros)), 1.0, *got, out, idx.to(DEV), resid_fmt=resid_fmt)
    assert _lib.load_library().carry_gdn_last_kernel() == (6 if edge == 64 else 2 if T is None else 3)
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1])


def _columns(edge, qmax, seed, res_fmt, B=3, HV=8):
    """The same in the statequant layout: codes, scale, residual of one of its formats and residual step."""
    few = {orc.RES_FP16: (1025, 2047), orc.RES_FP8: (5, 7)}.get(res_fmt)       # residuals that the format holds: ties alone
    c, r, S, E = _rows((B, HV), edge, qmax, seed, exact=few is not None, **(dict(lo=few[0], hi=few[1] + 1) if few else {}))
    unit = UNIT if few is None else 2.0 ** -12
    c, r = c.transpose(-1, -2).contiguous(), r.transpose(-1, -2).contiguous()
    target = ((c * S[..., None, :] + r * E[..., None, None]) * unit).float()
    return c, r, (S * unit).float(), (E * unit).float(), target


@pytest.mark.parametrize("edge", [128, 64])
@pytest.mark.parametrize("res_fmt,rscale", [(0, "v"), (1, "v"), (2, "v"), (3, "v"), (3, "head"), (4, "v"), (4, "head")])
@pytest.mark.parametrize("bits", [8, 4])
def test_statequant_layout(edge, res_fmt, rscale, bits):
    """Streaming kernel (fp32, fp16 and fp8 residuals), 16 warps per tile (int8, int4), 64-wide kernel, generic kernel."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    qmax = orc.qmax_for_bits(bits)
    c, r, scale, es, target = _columns(edge, int(qmax), 10 * edge + res_fmt, res_fmt)
    B, HV = es.shape
    if res_fmt < 3:
        e, e_scale = (r * es[..., None, None]).to(orc.residual_dtype(res_fmt)), None
        assert torch.equal(e.double(), r * es[..., None, None].double())
    else:
        e = orc.pack_int4(r) if res_fmt == 4 else r.to(torch.int8)
        e_scale = es if rscale == "head" else es[..., None].expand(B, HV, edge).contiguous()
    z, ones = torch.zeros(B, HV, edge), torch.ones(B, HV)
    kw = dict(bits=bits, res_fmt=res_fmt, resid_scale=rscale)
    want = orc.quant_step(c.to(torch.int8), scale, e, e_scale, z, z, z, ones, ones, **kw)
    assert torch.equal(want[2], scale)
    _reciprocal_misses(target, scale[..., None, :], want[1])
    dev = [x if x is None else x.to(DEV) for x in (c.to(torch.int8), scale, e, e_scale, z, z, z, ones, ones)]
    got = sq.gdn_quant_step_fused(*dev, **kw)
    kernel = _lib.load_library().carry_gdn_last_kernel()
    assert kernel == (2 if edge == 128 else 8 if res_fmt > 2 else 1)
    assert torch.equal(got[1].cpu(), want[1]) and torch.equal(got[2].cpu(), scale)


@pytest.mark.parametrize("edge", [128, 64])
@pytest.mark.parametrize("sscale", ["v", "head"])
@pytest.mark.parametrize("bits", [8, 4])
def test_statequant_layout_without_a_residual(edge, sscale, bits):
    """The targets come in as k (x) v over a state of zeros: the columns of a head are alike up to their signs."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    qmax = orc.qmax_for_bits(bits)
    _, _, scale, _, target = _columns(edge, int(qmax), edge, orc.RES_NONE)
    B, HV = scale.shape[:2]
    k, scale = target[..., 0].contiguous(), scale[..., 0].contiguous()
    v = torch.ones(B, HV, edge)
    v[..., 1::2] = -1.0
    codes = torch.zeros(B, HV, edge, edge, dtype=torch.int8)
    s_in = torch.ones(B, HV, edge) if sscale == "v" else torch.ones(B, HV)
    ones, kw = torch.ones(B, HV), dict(bits=bits, res_fmt=sq.RES_NONE, state_scale=sscale)
    args = (codes, s_in, None, None, torch.zeros_like(k), k, v, ones, ones)
    want = orc.quant_step(*args, **kw)
    assert torch.equal(want[2].reshape(B, HV, -1), scale[..., None].expand(B, HV, edge if sscale == "v" else 1))
    _reciprocal_misses(k[..., None] * v[..., None, :], scale[..., None, None], want[1])
    got = sq.gdn_quant_step_fused(*(x if x is None else x.to(DEV) for x in args), **kw)
    assert _lib.load_library().carry_gdn_last_kernel() == (5 if edge == 128 else 8)
    assert torch.equal(got[1].cpu(), want[1]) and torch.equal(got[2].cpu(), want[2])


@pytest.mark.parametrize("res_fmt", [orc.RES_FP32, orc.RES_FP16, orc.RES_FP8])
def test_chain(res_fmt):
    """The targets come in as k (x) v over a state of zeros; two tokens later code and residual still add up to them."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    T, edge = 3, 128
    _, _, scale, _, target = _columns(edge, 127, 5 + res_fmt, res_fmt)
    B, HV = scale.shape[:2]
    scale = scale[..., 0].contiguous()
    k = torch.zeros(T, B, HV, edge)
    k[0] = target[..., 0]
    v = torch.ones(T, B, HV, edge)
    v[..., 1::2] = -1.0
    ones, h0, q = torch.ones(T, B, HV), torch.zeros(B, HV, edge, edge), torch.zeros(T, B, HV, edge)
    want = orc.quant_decode(h0, q, k, v, ones, ones, res_fmt=res_fmt)
    assert torch.equal(want[2], scale[..., None].expand(B, HV, edge))
    _reciprocal_misses(k[0][..., None] * v[0][..., None, :], scale[..., None, None], want[1])
    got = sq.gdn_quant_decode_fused(*(x.to(DEV) for x in (h0, q, k, v, ones, ones)), T, res_fmt=res_fmt)
    assert _lib.load_library().carry_gdn_last_kernel() == 7
    for x, y in zip(got[1:4], want[1:4]):
        assert torch.equal(x.cpu().float(), y.float())
