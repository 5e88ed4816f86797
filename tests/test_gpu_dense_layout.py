"""The statequant-layout kernels for 128- and 64-wide heads against the generic kernel, which takes the same call when the
codes do not start on a vector boundary: one tile, head counts that are no multiple of anything, one tile more than there
are CTAs (2 x 148), and enough of them to go round a CTA's ring of stages.  The two sum in different orders, so codes at a
rounding tie may differ; tolerances are those of the comparison with the oracle."""

from __future__ import annotations

import pytest
import torch

from oracle import gdn_oracle as orc
from parity import assert_close, assert_codes, check_quant_step, seeded_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _off_grid(x):
    """A contiguous copy that starts one element behind a 16-byte boundary."""
    wide = torch.empty(x.numel() + 16, dtype=x.dtype, device=x.device)
    view = wide[1:1 + x.numel()].view(x.shape)
    view.copy_(x)
    return view


@pytest.mark.parametrize("edge", [128, 64])
@pytest.mark.parametrize("B,HV", [(1, 1), (2, 3), (27, 11), (47, 32)])
@pytest.mark.parametrize("res_fmt,rscale,sscale", [(3, "v", "v"), (3, "head", "v"), (4, "v", "v"), (4, "head", "v"),
                                                   (5, "v", "v"), (5, "v", "head")])
@pytest.mark.parametrize("dtype,bits", [(torch.float32, 8), (torch.bfloat16, 4), (torch.float16, 3)])
def test_step_against_the_generic_kernel(edge, B, HV, res_fmt, rscale, sscale, dtype, bits):
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    assert (res_fmt, sq.RES_INT8, sq.RES_INT4) == (res_fmt, 3, 4) and sq.RES_NONE == orc.RES_NONE == 5
    h0, q, k, v, alpha, beta = seeded_inputs(B, HV, edge, edge, seed=B, dtype=dtype, alpha_mode="gated")
    h0[0, 0, :, 2] = 0.0
    state = orc.init_quant_state(h0[:2], bits, res_fmt, rscale, sscale)
    reps = -(-B // state[0].shape[0])
    state = [None if x is None else x.repeat(reps, *([1] * (x.dim() - 1)))[:B].to(DEV) for x in state]
    g = torch.Generator(device=DEV).manual_seed(1)
    if res_fmt == 3:
        state[2] = torch.randint(-127, 128, state[2].shape, generator=g, dtype=torch.int8, device=DEV)
    elif res_fmt == 4:                                    # two codes of -7..7 per byte
        lo, hi = (torch.randint(-7, 8, state[2].shape, generator=g, dtype=torch.int8, device=DEV) for _ in range(2))
        state[2] = (lo & 15) | (hi << 4)
    if state[3] is not None:
        state[3] = torch.rand(state[3].shape, generator=g, device=DEV) * 1e-6 + 1e-7
    acts = [x.to(DEV) for x in (q, k, v, alpha, beta)]
    kw = dict(bits=bits, res_fmt=res_fmt, resid_scale=rscale, state_scale=sscale)
    got = sq.gdn_quant_step_fused(*state, *acts, **kw)
    kernel = _lib.load_library().carry_gdn_last_kernel()
    assert kernel == (8 if edge == 64 else 5 if res_fmt == 5 else 2)
    want = sq.gdn_quant_step_fused(_off_grid(state[0]), *state[1:], *acts, **kw)
    assert _lib.load_library().carry_gdn_last_kernel() == 1
    # at most 6e-4 of the int8 residual codes differ at 8 bits, fewer at fewer bits (a residual step is then larger against
    # the unit in the last place of its target); the smallest case has 4096 codes, 2.3 of them expected: allow 8 more
    check_quant_step(got, [None if x is None else x.cpu() for x in want], res_fmt, unpack_int4=orc.unpack_int4,
                     what=f"{edge} {res_fmt} {rscale} {sscale}", max_frac=1e-3 + 8 / got[1].numel())


@pytest.mark.parametrize("edge", [128, 64])
@pytest.mark.parametrize("rscale", ["v", "head"])
def test_int4_residual_scale_of_a_larger_column(edge, rscale):
    """Columns of very different magnitudes under residual scales that belong to the largest one: a residual code of 0 adds
    exactly 0, so that a column a million times smaller is rounded as well as the largest, and a zero column stays zero.

    A target is three roundings of its own size and a sum of `edge` products: within 2e-5 of the column's step of the oracle's,
    which flips 4e-5 of the codes."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    B, HV = 3, 8
    h0, q, k, v, alpha, beta = seeded_inputs(B, HV, edge, edge, seed=edge, alpha_mode="gated")
    mags = torch.tensor([1.0, 1e-2, 1e-4, 1e-6, 0.0])
    kind = torch.arange(edge) % len(mags)
    h0, v = h0 * mags[kind], v * mags[kind]
    h, scale, _, _ = orc.init_quant_state(h0, 8, orc.RES_INT4, rscale)
    codes = torch.randint(-7, 8, h.shape, generator=torch.Generator().manual_seed(2)) * (kind == 0)
    top = scale.amax(-1) / 14.0                            # half a step of the largest column is 7 codes
    es = top if rscale == "head" else top[..., None].expand(B, HV, edge).contiguous()
    state = (h, scale, orc.pack_int4(codes.to(torch.int8)), es)
    want = orc.quant_step(*state, q, k, v, alpha, beta, res_fmt=orc.RES_INT4, resid_scale=rscale)
    got = sq.gdn_quant_step_fused(*[x.to(DEV) for x in (*state, q, k, v, alpha, beta)], res_fmt=sq.RES_INT4, resid_scale=rscale)
    assert _lib.load_library().carry_gdn_last_kernel() == (8 if edge == 64 else 2)
    for j, mag in enumerate(mags.tolist()):
        of_kind = kind == j
        a, b = got[1].cpu()[..., of_kind], want[1][..., of_kind]
        assert int((a.int() - b.int()).abs().max()) <= 1, mag
        assert float((a != b).float().mean()) <= 2e-4, mag
        assert_close(got[2].cpu()[..., of_kind], want[2][..., of_kind], f"scales of columns x {mag}", rtol=1e-5, atol=0.0)
    assert not got[1].cpu()[..., kind == 4].any()


@pytest.mark.parametrize("case", ["2 bits", "129 heads", "activations", "scales"])
@pytest.mark.parametrize("sscale", ["v", "head"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_step_without_residual_at_any_width_and_alignment(case, sscale, dtype):
    """128-wide heads without a residual need nothing but codes on a 16-byte boundary: the smallest grid (one level on either
    side of zero), more heads than the streaming kernel's tables hold, and vectors that start anywhere."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    B, HV, bits = (3, 129, 4) if case == "129 heads" else (20, 16, 2 if case == "2 bits" else 8)
    h0, q, k, v, alpha, beta = seeded_inputs(B, HV, 128, 128, seed=B, dtype=dtype, alpha_mode="gated")
    h, scale, _, _ = [None if x is None else x.to(DEV) for x in orc.init_quant_state(h0, bits, orc.RES_NONE, "v", sscale)]
    acts = [x.to(DEV) for x in (q, k, v, alpha, beta)]
    if case == "activations":
        acts = [_off_grid(x) for x in acts]
    elif case == "scales":
        scale = _off_grid(scale)
    kw = dict(bits=bits, res_fmt=sq.RES_NONE, state_scale=sscale)
    got = sq.gdn_quant_step_fused(h, scale, None, None, *acts, **kw)
    assert _lib.load_library().carry_gdn_last_kernel() == 5
    want = sq.gdn_quant_step_fused(_off_grid(h), scale, None, None, *acts, **kw)
    assert _lib.load_library().carry_gdn_last_kernel() == 1
    check_quant_step(got, [None if x is None else x.cpu() for x in want], orc.RES_NONE, unpack_int4=orc.unpack_int4,
                     what=f"{case} {sscale}", max_frac=1e-3)


def _spoil(what, state, acts):
    """Copies with one value of head (1, 1) replaced; column 5 where the tensor has columns."""
    state, acts = [None if x is None else x.clone() for x in state], [x.clone() for x in acts]
    name, value = what.rsplit(" ", 1)
    t = {"v": acts[2], "k": acts[1], "alpha": acts[3], "scale": state[1], "resid scale": state[3]}[name]
    t.view(t.shape[0], t.shape[1], -1)[1, 1, min(5, t.numel() // (t.shape[0] * t.shape[1]) - 1)] = float(value)
    return state, acts


def _spoiled_case(edge, res_fmt, rscale, sscale, what):
    h0, q, k, v, alpha, beta = seeded_inputs(2, 3, edge, edge, seed=1, alpha_mode="gated")
    state = [None if x is None else x.to(DEV) for x in orc.init_quant_state(h0, 8, res_fmt, rscale, sscale)]
    if state[3] is not None:
        g = torch.Generator().manual_seed(1)
        codes = torch.randint(-7, 8, h0.shape, generator=g).to(torch.int8)
        state[2] = (orc.pack_int4(codes) if res_fmt == 4 else codes).to(DEV)
        state[3] += 1e-5
    acts = [x.to(DEV) for x in (q, k, v, alpha, beta)]
    return (state, acts), _spoil(what, state, acts), dict(bits=8, res_fmt=res_fmt, resid_scale=rscale, state_scale=sscale)


@pytest.mark.parametrize("res_fmt,rscale,sscale", [(3, "v", "v"), (3, "head", "v"), (4, "v", "v"), (4, "head", "v"),
                                                   (5, "v", "v"), (5, "v", "head")])
@pytest.mark.parametrize("what", ["v nan", "v inf", "k nan", "k inf", "alpha inf", "scale nan", "scale inf",
                                  "resid scale nan", "resid scale inf"])
def test_narrow_heads_with_a_value_that_is_not_finite(res_fmt, rscale, sscale, what):
    """A NaN or an infinity leaves what the generic kernel leaves: maxima that pass a NaN over, clamped codes.  (The
    kernels sum in different orders: codes elsewhere may differ at a tie, as in the comparison above.)"""
    from carrykernel_b200 import _lib
    from carrykernel_b200.statequant import kernel as sq
    if res_fmt == 5 and what.startswith("resid"):
        pytest.skip("no residual")
    _, (state, acts), kw = _spoiled_case(64, res_fmt, rscale, sscale, what)
    got = [None if x is None else x.cpu() for x in sq.gdn_quant_step_fused(*state, *acts, **kw)]
    assert _lib.load_library().carry_gdn_last_kernel() == 8
    want = [None if x is None else x.cpu() for x in sq.gdn_quant_step_fused(_off_grid(state[0]), *state[1:], *acts, **kw)]
    assert _lib.load_library().carry_gdn_last_kernel() == 1
    limit = 2e-3 + 8 / got[1].numel()
    flips, _ = assert_codes(got[1], want[1], "state codes", max_frac=limit)
    if res_fmt < 5:
        a, b = (orc.unpack_int4(x) if res_fmt == 4 else x for x in (got[3], want[3]))
        assert_codes(a, b, "residual codes", max_frac=limit, exclude=flips)
    assert torch.equal(torch.isfinite(got[0]), torch.isfinite(want[0]))
    for i in (0, 2, 4):
        if got[i] is not None:
            a, b = got[i], want[i]
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b)), i
            ok = torch.isfinite(b)
            assert_close(a[ok], b[ok], f"output {i}", rtol=1e-3, atol=1e-5 if i == 0 else 1e-9)


@pytest.mark.parametrize("edge", [128, 64])
@pytest.mark.parametrize("res_fmt", [3, 4, 5])
@pytest.mark.parametrize("what", ["v nan", "v inf", "scale nan", "scale inf"])
def test_columns_beside_one_that_is_not_finite(edge, res_fmt, what):
    """With scales per column a NaN or an infinity in one stays in it: every other column is left bit for bit as it would be
    without it, residual codes that share a byte with the lost column's among them."""
    from carrykernel_b200.statequant import kernel as sq
    clean, spoiled, kw = _spoiled_case(edge, res_fmt, "v", "v", what)
    want, got = (sq.gdn_quant_step_fused(*state, *acts, **kw) for state, acts in (clean, spoiled))
    keep = torch.ones(2, 3, edge, dtype=torch.bool, device=DEV)
    keep[1, 1, 5] = False
    assert not torch.isfinite(got[0][1, 1, 5]) and (what != "v inf" or res_fmt != 5 or torch.isinf(got[2][1, 1, 5]))
    for a, b in zip(got, want):
        if a is not None:
            if res_fmt == 4 and a.dim() == 4 and a.shape[-1] == edge // 2:
                a, b = (orc.unpack_int4(x.cpu()).to(DEV) for x in (a, b))
            where = keep[:, :, None].expand(a.shape) if a.dim() == 4 else keep
            assert torch.equal(a[where], b[where])


@pytest.mark.parametrize("B,HV", [(1, 1), (2, 3), (40, 31)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_fp32_step_of_narrow_heads(B, HV, dtype):
    """Sums of 64 products of magnitude 0.1: 1e-6 apart in another order."""
    from carrykernel_b200.statequant import kernel as sq
    h0, q, k, v, alpha, beta = [x.to(DEV) for x in seeded_inputs(B, HV, 64, 64, seed=B, dtype=dtype, alpha_mode="gated")]
    h, o = sq.gdn_step_fused_fp32(h0, q, k, v, alpha, beta)
    hr, orf = orc.gdn_step(h0.cpu(), q.float().cpu(), k.float().cpu(), v.float().cpu(), alpha.cpu(), beta.cpu())
    assert_close(h.cpu(), hr, "state", rtol=1e-5, atol=2e-6)
    assert_close(o.cpu(), orf, "output", rtol=1e-5, atol=4e-6)


@pytest.mark.parametrize("resid_fmt", [orc.RESID_INT8, orc.RESID_INT4])
@pytest.mark.parametrize("rscale", ["v", "head"])
@pytest.mark.parametrize("keep_error", [False, True])
@pytest.mark.parametrize("edge", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_square_tiles_in_and_out_of_the_pool(resid_fmt, rscale, keep_error, edge, dtype):
    """Bit for bit the oracle's, with a padding request and a pool whose slots are further apart than they need be."""
    from carrykernel_b200.vllm_integration import state_pool as sp
    B, HV, slots = 4, 3, 7
    g = torch.Generator().manual_seed(edge)
    h = torch.randn(B, HV, edge, edge, generator=g) * 0.1
    h[0, 0, 0] = 0.0
    h[0, 0, 1] *= 1e-20
    h[0, 0, 2] = (torch.arange(edge) % 253 - 126).float() + 0.5      # ties
    h[0, 0, 2, 0] = 127.0
    h = h.to(dtype)
    idx = torch.tensor([5, 0, 2, 6], dtype=torch.int32)
    want = list(orc.init_quantized_pool(slots, HV, edge, edge, resid_fmt=resid_fmt, resid_scale=rscale))
    got = []
    for t in want:
        wide = torch.zeros(slots, t[0].numel() + 16, dtype=t.dtype, device=DEV)
        got.append(wide.as_strided(t.shape, (wide.stride(0), *t.stride()[1:])))
        got[-1].copy_(t)
    orc.pool_store(h, *want, idx, resid_fmt=resid_fmt, keep_error=keep_error)
    sp.store_state(h.to(DEV), got, idx.to(DEV), resid_fmt=resid_fmt, keep_error=keep_error)
    for x, y in zip(got, want):
        assert torch.equal(x.cpu(), y)
    out = torch.full((B, HV, edge, edge), 9.0, dtype=dtype, device=DEV)
    sp.load_state(got, idx.to(DEV), resid_fmt=resid_fmt, out=out)
    ref = orc.pool_load(*want, idx, resid_fmt=resid_fmt)
    assert torch.equal(out.cpu(), ref.to(dtype))
