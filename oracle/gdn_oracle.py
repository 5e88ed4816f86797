"""CPU oracle for the fused Gated-DeltaNet decode step on a quantized state.

TEST INFRASTRUCTURE ONLY.  This module is the oracle the CUDA kernels are
compared against; the shipped package never imports it.  It restates, with
plain torch CPU ops, the arithmetic that tomalmog/carrykernel defines for the
path (paths below are relative to that project):

  * the exact recurrence            statequant/reference.py:20-53
  * the quantizers + error feedback statequant/quant.py:23-42,65-80
  * the fused one-step reference    statequant/kernel.py:99-202
  * the per-head residual quantizer modal_residual.py:42-56
  * the slot-indexed [V, K] step    vllm_integration/quantized_packed_decode.py:101-239,330-369
    (that file only has a Triton kernel; the step here follows its statements
    one by one and is cross-checked against the reference's own partial
    oracle in vllm_integration/test_quantized_packed_decode.py:54-105)

Parity of this restatement is pinned two ways: bit-for-bit against the golden
vectors in tests/golden/ (generated by importing the reference; script beside
them), and, where the reference checkout is present, bit-for-bit against the
imported reference functions themselves.

Conventions
-----------
statequant layout: state ``[B, HV, K, V]`` (V contiguous), one scale per
V-column (amax over K, ``dim=-2``).  Slot layout: pool ``[slots, HV, V, K]``
(K contiguous), one scale per V-row (amax over K, ``dim=-1``).  Both are "one
scale per V channel"; only the memory order differs.

Operation order matters for code-level parity and is kept exactly:
``(code * scale) * alpha``; ``h + (k * dv)`` with the product rounded first;
true division before ``torch.round`` (round half to even).
"""

from __future__ import annotations

import torch

EPS = 1e-12
QMAX_INT8 = 127.0
QMAX_INT4 = 7.0
SOFTPLUS_THRESHOLD = 20.0
NULL_BLOCK_ID = 0

# residual formats of the statequant signature (statequant/kernel.py:59-63);
# RES_INT4 and RES_NONE are additive ids that do not exist upstream.
RES_FP32, RES_FP16, RES_FP8, RES_INT8, RES_INT4, RES_NONE = 0, 1, 2, 3, 4, 5
# residual formats of the slot path (quantized_packed_decode.py:82-83)
RESID_INT8, RESID_INT4 = 0, 1

# how the scale floor is applied
EPS_ON_AMAX = 0    # max(amax, EPS) / qmax      statequant/kernel.py:110,143,173
EPS_ON_SCALE = 1   # max(amax / qmax, EPS)      quantized_packed_decode.py:206,213


def qmax_for_bits(bits: int) -> float:
    """Largest code magnitude of a symmetric signed grid (statequant/quant.py:18-20)."""
    return float(2 ** (bits - 1) - 1)


def _scale_from_amax(amax: torch.Tensor, qmax: float, eps_mode: int) -> torch.Tensor:
    if eps_mode == EPS_ON_AMAX:
        return amax.clamp(min=EPS) / qmax
    return torch.clamp(amax / qmax, min=EPS)


# ---------------------------------------------------------------------------
# recurrence (statequant/reference.py:20-53, statequant/kernel.py:116-123)
# ---------------------------------------------------------------------------

def gdn_step(h, q, k, v, alpha, beta):
    """One exact GDN step.  ``h [..., K, V]``; ``q,k [..., K]``; ``v [..., V]``;
    ``alpha,beta [...]``.  Leading dims are ``[HV]`` or ``[B, HV]``.
    Returns ``(h_new, o)``.  The einsum subscripts are the reference's, so the
    CPU reduction order is the reference's too."""
    if h.dim() == 3:
        h = alpha[:, None, None] * h
        read = torch.einsum("hkv,hk->hv", h, k)
        dv = beta[:, None] * (v - read)
        h = h + torch.einsum("hk,hv->hkv", k, dv)
        o = torch.einsum("hkv,hk->hv", h, q)
        return h, o
    h = alpha[..., None, None] * h
    read = torch.einsum("bhkv,bhk->bhv", h, k)
    dv = beta[..., None] * (v - read)
    h = h + torch.einsum("bhk,bhv->bhkv", k, dv)
    o = torch.einsum("bhkv,bhk->bhv", h, q)
    return h, o


def gdn_decode(h0, q, k, v, alpha, beta):
    """T chained exact steps (statequant/reference.py:37-53).  Inputs carry a
    leading T axis.  Returns ``(o [T, ...], h_final)``."""
    h = h0.clone()
    outs = []
    for t in range(q.shape[0]):
        h, o = gdn_step(h, q[t], k[t], v[t], alpha[t], beta[t])
        outs.append(o)
    return torch.stack(outs), h


# ---------------------------------------------------------------------------
# quantizers (statequant/quant.py:23-42, statequant/kernel.py:99-113)
# ---------------------------------------------------------------------------

def quantize_per_column(x, bits: int = 8, eps_mode: int = EPS_ON_AMAX):
    """One scale per V-column of ``x [..., K, V]`` (amax over K).
    Returns ``(codes int8, scale [..., V], dequantized)``."""
    qmax = qmax_for_bits(bits)
    scale = _scale_from_amax(x.abs().amax(dim=-2, keepdim=True), qmax, eps_mode)
    code = torch.round(x / scale).clamp(-qmax, qmax)
    return code.to(torch.int8), scale.squeeze(-2), code * scale


def quantize_per_head(x, bits: int = 8):
    """One scale per ``[K, V]`` matrix (statequant/quant.py:23-34).
    Returns ``(codes int8, scale [...], dequantized)``."""
    qmax = qmax_for_bits(bits)
    scale = x.abs().amax(dim=(-1, -2), keepdim=True).clamp(min=EPS) / qmax
    code = torch.round(x / scale).clamp(-qmax, qmax)
    return code.to(torch.int8), scale[..., 0, 0], code * scale


def error_feedback(x, e, quant_fn):
    """``target = x + e; xq = quant(target); e' = target - xq``
    (statequant/quant.py:75-80).  ``quant_fn`` returns the dequantized tensor.
    Returns ``(xq, e')``."""
    target = x + e
    xq = quant_fn(target)
    return xq, target - xq


# ---------------------------------------------------------------------------
# int4 nibble packing (quantized_packed_decode.py:195-200, 221-237)
# ---------------------------------------------------------------------------

def pack_int4(codes: torch.Tensor) -> torch.Tensor:
    """Pack signed 4-bit codes (values in [-8, 7], any integer dtype) two per
    byte along the last axis: even index -> low nibble, odd index -> high."""
    c = codes.to(torch.int32) & 0xF
    byte = c[..., 0::2] | (c[..., 1::2] << 4)
    byte = torch.where(byte > 127, byte - 256, byte)
    return byte.to(torch.int8)


def unpack_int4(packed: torch.Tensor) -> torch.Tensor:
    """Inverse of :func:`pack_int4`; returns int32 codes in [-8, 7]."""
    b = packed.to(torch.int32) & 0xFF
    lo = b & 0xF
    hi = (b >> 4) & 0xF
    lo = torch.where(lo > 7, lo - 16, lo)
    hi = torch.where(hi > 7, hi - 16, hi)
    return torch.stack([lo, hi], dim=-1).reshape(*packed.shape[:-1], packed.shape[-1] * 2)


# ---------------------------------------------------------------------------
# residual codec, statequant layout (statequant/kernel.py:126-146;
# per-head scale: modal_residual.py:51-55)
# ---------------------------------------------------------------------------

def residual_dtype(res_fmt: int):
    return {RES_FP32: torch.float32, RES_FP16: torch.float16,
            RES_FP8: torch.float8_e5m2, RES_INT8: torch.int8,
            RES_INT4: torch.int8}[res_fmt]


def dequant_residual_kv(e, e_scale, res_fmt: int):
    """Stored residual -> fp32 ``[..., K, V]``.  ``e_scale`` is ``[..., V]``
    (per V-column) or ``[...]`` (per head)."""
    if res_fmt == RES_NONE:
        return None
    if res_fmt in (RES_INT8, RES_INT4):
        codes = unpack_int4(e).float() if res_fmt == RES_INT4 else e.float()
        if e_scale.dim() == codes.dim() - 1:            # per V-column
            return codes * e_scale[..., None, :]
        return codes * e_scale[..., None, None]          # per head
    return e.float()


def quant_residual_kv(e_fp32, res_fmt: int, resid_scale: str = "v",
                      eps_mode: int = EPS_ON_AMAX):
    """fp32 residual -> ``(stored, scale | None)`` in the statequant layout."""
    if res_fmt == RES_FP32:
        return e_fp32, None
    if res_fmt == RES_FP16:
        return e_fp32.to(torch.float16), None
    if res_fmt == RES_FP8:
        return e_fp32.to(torch.float8_e5m2), None
    if res_fmt not in (RES_INT8, RES_INT4):
        raise ValueError(f"unknown residual format {res_fmt}")
    qmax = QMAX_INT4 if res_fmt == RES_INT4 else QMAX_INT8
    if resid_scale == "v":
        scale = _scale_from_amax(e_fp32.abs().amax(dim=-2), qmax, eps_mode)      # [..., V]
        code = torch.round(e_fp32 / scale[..., None, :]).clamp(-qmax, qmax)
    elif resid_scale == "head":
        scale = _scale_from_amax(e_fp32.abs().amax(dim=(-1, -2)), qmax, eps_mode)  # [...]
        code = torch.round(e_fp32 / scale[..., None, None]).clamp(-qmax, qmax)
    else:
        raise ValueError(f"resid_scale must be 'v' or 'head', got {resid_scale!r}")
    code = code.to(torch.int8)
    if res_fmt == RES_INT4:
        code = pack_int4(code)
    return code, scale


# ---------------------------------------------------------------------------
# the fused step, statequant layout (statequant/kernel.py:149-178)
# ---------------------------------------------------------------------------

def quant_step(h_int8, scale, e, e_scale, q, k, v, alpha, beta,
               bits: int = 8, res_fmt: int = RES_FP32, resid_scale: str = "v",
               state_scale: str = "v", eps_mode: int = EPS_ON_AMAX):
    """One fused step on ``[B, HV, K, V]`` codes.

    ``state_scale='v'`` is the reference's per-V-column state scale (``scale``
    is ``[B, HV, V]``); ``'head'`` is the uniform per-head grid of
    statequant/quant.py:23-34 (``scale`` is ``[B, HV]``), used by the
    no-error-feedback arm of the bit-width sweep.  ``res_fmt=RES_NONE`` drops
    the residual (plain re-quantization each step).

    Returns ``(o, h_int8_new, scale_new, e_new, e_scale_new)``.
    """
    qmax = qmax_for_bits(bits)
    q, k, v = q.float(), k.float(), v.float()
    alpha, beta = alpha.float(), beta.float()
    if state_scale == "v":
        h = h_int8.float() * scale[..., None, :]
    else:
        h = h_int8.float() * scale[..., None, None]
    h, o = gdn_step(h, q, k, v, alpha, beta)

    e_deq = dequant_residual_kv(e, e_scale, res_fmt)
    target = h if e_deq is None else h + e_deq
    if state_scale == "v":
        scale_new = _scale_from_amax(target.abs().amax(dim=-2), qmax, eps_mode)
        s_b = scale_new[..., None, :]
    else:
        scale_new = _scale_from_amax(target.abs().amax(dim=(-1, -2)), qmax, eps_mode)
        s_b = scale_new[..., None, None]
    q_int = torch.round(target / s_b).clamp(-qmax, qmax)
    h_new = q_int.to(torch.int8)
    if res_fmt == RES_NONE:
        return o, h_new, scale_new, None, None
    deq = q_int.float() * s_b
    e_new, e_scale_new = quant_residual_kv(target - deq, res_fmt, resid_scale, eps_mode)
    return o, h_new, scale_new, e_new, e_scale_new


def init_quant_state(h0, bits: int = 8, res_fmt: int = RES_FP32,
                     resid_scale: str = "v", state_scale: str = "v"):
    """fp32 ``h0 [..., K, V]`` -> ``(codes, scale, e=0, e_scale)``
    (statequant/kernel.py:181-202).  ``e_scale`` is a zero tensor for the
    integer residual formats and ``None`` otherwise."""
    if state_scale == "v":
        codes, scale, _ = quantize_per_column(h0, bits)
    else:
        codes, scale, _ = quantize_per_head(h0, bits)
    if res_fmt == RES_NONE:
        return codes, scale, None, None
    lead = h0.shape[:-2]
    K, V = h0.shape[-2:]
    if res_fmt in (RES_INT8, RES_INT4):
        vv = V // 2 if res_fmt == RES_INT4 else V
        e = torch.zeros((*lead, K, vv), dtype=torch.int8)
        es_shape = (*lead, V) if resid_scale == "v" else lead
        return codes, scale, e, torch.zeros(es_shape, dtype=torch.float32)
    return codes, scale, torch.zeros(h0.shape, dtype=residual_dtype(res_fmt)), None


def quant_decode(h0, q, k, v, alpha, beta, bits: int = 8, res_fmt: int = RES_FP32,
                 resid_scale: str = "v", state_scale: str = "v"):
    """T chained fused steps (statequant/kernel.py:436-452); inputs carry a
    leading T axis.  Returns ``(o [T, ...], codes, scale, e, e_scale)``."""
    codes, scale, e, e_scale = init_quant_state(h0, bits, res_fmt, resid_scale, state_scale)
    outs = []
    for t in range(q.shape[0]):
        o, codes, scale, e, e_scale = quant_step(
            codes, scale, e, e_scale, q[t], k[t], v[t], alpha[t], beta[t],
            bits, res_fmt, resid_scale, state_scale)
        outs.append(o)
    return torch.stack(outs), codes, scale, e, e_scale


def dequant_state(codes, scale):
    """codes ``[..., K, V]`` with scale ``[..., V]`` (per column) or ``[...]``."""
    if scale.dim() == codes.dim() - 1:
        return codes.float() * scale[..., None, :]
    return codes.float() * scale[..., None, None]


def chained_ef_decode(h0, q, k, v, alpha, beta, bits: int = 8,
                      granularity: str = "column", use_ef: bool = True):
    """The mechanism experiment: exact recurrence + fp32 error feedback around a
    dequantizing quantizer (experiments/exp2b_granularity.py:37-46,
    experiments/test_cuda_kernel.py:47-61).  ``h0 [HV, K, V]`` is used as is
    (not pre-quantized).  Returns the final dequantized state."""
    if granularity == "column":
        qf = lambda x: quantize_per_column(x, bits)[2]
    elif granularity == "head":
        qf = lambda x: quantize_per_head(x, bits)[2]
    else:
        raise ValueError(granularity)
    h = h0.clone()
    e = torch.zeros_like(h0)
    for t in range(q.shape[0]):
        h, _ = gdn_step(h, q[t], k[t], v[t], alpha[t], beta[t])
        if use_ef:
            h, e = error_feedback(h, e, qf)
        else:
            h = qf(h)
    return h


# ---------------------------------------------------------------------------
# slot-indexed [V, K] step (quantized_packed_decode.py:101-239)
# ---------------------------------------------------------------------------

def gates(a, b, A_log, dt_bias):
    """In-kernel gate derivation (quantized_packed_decode.py:175-182).
    ``a, b [B, HV]``; ``A_log, dt_bias [HV]`` -> ``(alpha, beta) [B, HV]`` fp32."""
    x = a.float() + dt_bias.float()
    softplus_x = torch.where(x <= SOFTPLUS_THRESHOLD, torch.log(1.0 + torch.exp(x)), x)
    g = -torch.exp(A_log.float()) * softplus_x
    return torch.exp(g), torch.sigmoid(b.float())


def unpack_mixed_qkv(mixed_qkv, H: int, HV: int, K: int, V: int, scale: float, l2norm: bool):
    """Slice q|k|v out of the packed activation row, normalise, scale, and fan
    the H query/key heads out to the HV value heads
    (quantized_packed_decode.py:161-172, head map :117)."""
    B = mixed_qkv.shape[0]
    q = mixed_qkv[:, :H * K].reshape(B, H, K).float()
    k = mixed_qkv[:, H * K:2 * H * K].reshape(B, H, K).float()
    v = mixed_qkv[:, 2 * H * K:2 * H * K + HV * V].reshape(B, HV, V).float()
    if l2norm:
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6)
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q = q * scale
    rep = HV // H
    return q.repeat_interleave(rep, dim=1), k.repeat_interleave(rep, dim=1), v


def init_quantized_pool(num_slots: int, HV: int, V: int, K: int, h0=None,
                        resid_fmt: int = RESID_INT8, resid_scale: str = "v"):
    """Zeroed pool ``(state_codes, state_scale, resid_codes, resid_scale)``,
    optionally seeded from fp32 ``h0 [slots, HV, V, K]``
    (quantized_packed_decode.py:330-352)."""
    rk = K // 2 if resid_fmt == RESID_INT4 else K
    sc = torch.zeros((num_slots, HV, V, K), dtype=torch.int8)
    ss = torch.zeros((num_slots, HV, V), dtype=torch.float32)
    rc = torch.zeros((num_slots, HV, V, rk), dtype=torch.int8)
    rs = torch.zeros((num_slots, HV, V) if resid_scale == "v" else (num_slots, HV),
                     dtype=torch.float32)
    if h0 is not None:
        s = h0.abs().amax(dim=-1).clamp(min=EPS) / QMAX_INT8
        sc.copy_(torch.round(h0 / s[..., None]).clamp(-QMAX_INT8, QMAX_INT8).to(torch.int8))
        ss.copy_(s)
    return sc, ss, rc, rs


def state_bytes_per_slot(HV: int, V: int, K: int, quantized: bool,
                         base_dtype_size: int = 4, resid_fmt: int = RESID_INT8,
                         resid_scale: str = "v") -> int:
    """Bytes of recurrent state per slot (quantized_packed_decode.py:355-369);
    ``resid_scale='head'`` shrinks the residual scale to one float per head."""
    if not quantized:
        return HV * V * K * base_dtype_size
    codes = HV * V * K
    resid = HV * V * (K // 2 if resid_fmt == RESID_INT4 else K)
    scales = HV * V * 4 + (HV * V * 4 if resid_scale == "v" else HV * 4)
    return codes + resid + scales


def packed_decode_step(mixed_qkv, a, b, A_log, dt_bias, scale,
                       state_codes, state_scale, resid_codes, resid_scale,
                       out, ssm_state_indices,
                       use_qk_l2norm_in_kernel: bool = False,
                       resid_fmt: int = RESID_INT8,
                       eps_mode: int = EPS_ON_SCALE):
    """One slot-indexed step, in place on the (CPU) pool; returns ``out``.

    Request ``n`` uses slot ``ssm_state_indices[n]``; a slot id ``<= 0`` is
    padding: zeros go to ``out[n]`` and the pool is untouched
    (quantized_packed_decode.py:129-136).  The residual scale is per V-row when
    ``resid_scale`` is ``[slots, HV, V]`` and per head when ``[slots, HV]``.
    The recurrence is evaluated in the ``[K, V]`` orientation with the same
    einsums as :func:`gdn_step`, exactly as the reference's own [V, K] oracle
    does (test_quantized_packed_decode.py:78-97).
    """
    B = mixed_qkv.shape[0]
    _, HV, V, K = state_codes.shape
    qk_dim = mixed_qkv.shape[1] - HV * V
    H = (qk_dim // 2) // K
    per_head = resid_scale.dim() == 2
    rqmax = QMAX_INT4 if resid_fmt == RESID_INT4 else QMAX_INT8

    alpha, beta = gates(a, b, A_log, dt_bias)
    q, k, v = unpack_mixed_qkv(mixed_qkv, H, HV, K, V, scale, use_qk_l2norm_in_kernel)

    for n in range(B):
        slot = int(ssm_state_indices[n])
        if slot <= 0:
            out[n] = 0
            continue
        h_vk = state_codes[slot].float() * state_scale[slot][..., None]      # [HV, V, K]
        h = h_vk.transpose(-1, -2).contiguous()                              # [HV, K, V]
        h, o = gdn_step(h, q[n], k[n], v[n], alpha[n], beta[n])
        out[n, 0] = o.to(out.dtype)

        rcodes = resid_codes[slot]
        rcodes = unpack_int4(rcodes).float() if resid_fmt == RESID_INT4 else rcodes.float()
        rs = resid_scale[slot]
        e_vk = rcodes * (rs[..., None, None] if per_head else rs[..., None])
        target = h.transpose(-1, -2) + e_vk                                  # [HV, V, K]

        s_new = _scale_from_amax(target.abs().amax(dim=-1), QMAX_INT8, eps_mode)   # [HV, V]
        codes = torch.round(target / s_new[..., None]).clamp(-QMAX_INT8, QMAX_INT8)
        e_new = target - codes * s_new[..., None]
        if per_head:
            es_new = _scale_from_amax(e_new.abs().amax(dim=(-1, -2)), rqmax, eps_mode)  # [HV]
            e_codes = torch.round(e_new / es_new[..., None, None]).clamp(-rqmax, rqmax)
        else:
            es_new = _scale_from_amax(e_new.abs().amax(dim=-1), rqmax, eps_mode)        # [HV, V]
            e_codes = torch.round(e_new / es_new[..., None]).clamp(-rqmax, rqmax)
        e_codes = e_codes.to(torch.int8)

        state_codes[slot] = codes.to(torch.int8)
        state_scale[slot] = s_new
        resid_scale[slot] = es_new
        resid_codes[slot] = pack_int4(e_codes) if resid_fmt == RESID_INT4 else e_codes
    return out



def packed_decode_multi(mixed_qkv, a, b, A_log, dt_bias, scale,
                        state_codes, state_scale, resid_codes, resid_scale,
                        out, ssm_state_indices,
                        use_qk_l2norm_in_kernel: bool = False,
                        resid_fmt: int = RESID_INT8,
                        eps_mode: int = EPS_ON_SCALE):
    """T tokens per request, ``mixed_qkv [B, T, W]``, ``a``/``b [B, T, HV]``,
    ``out [B, T, HV, V]``: by definition T calls of :func:`packed_decode_step`,
    token by token, in place on the pool.  (The reference has no multi-token
    call; this pins the meaning of the B200 library's one.)"""
    T = mixed_qkv.shape[1]
    for t in range(T):
        tmp = torch.empty((out.shape[0], 1) + tuple(out.shape[2:]), dtype=out.dtype)
        packed_decode_step(mixed_qkv[:, t].contiguous(), a[:, t].contiguous(), b[:, t].contiguous(), A_log, dt_bias,
                           scale, state_codes, state_scale, resid_codes, resid_scale, tmp, ssm_state_indices,
                           use_qk_l2norm_in_kernel, resid_fmt, eps_mode)
        out[:, t:t + 1] = tmp
    return out

def dequant_pool_state(state_codes, state_scale):
    """Pool codes ``[..., V, K]`` with per-row scale ``[..., V]`` -> fp32."""
    return state_codes.float() * state_scale[..., None]


# ---------------------------------------------------------------------------
# moving state in and out of the pool (no counterpart upstream beyond
# init_quantized_state, quantized_packed_decode.py:330-352; these pin the
# meaning of the B200 library's pool calls)
# ---------------------------------------------------------------------------

def pool_store(h, state_codes, state_scale, resid_codes, resid_scale, slots,
               resid_fmt: int = RESID_INT8, keep_error: bool = False):
    """Quantise ``h [B, HV, V, K]`` into the slots ``slots [B]`` of the (CPU)
    pool, in place.  State codes and scale as ``init_quantized_state``
    (quantized_packed_decode.py:346-350).  The residual is zeroed, or with
    ``keep_error`` set to ``h - codes * scale`` encoded as one decode step
    encodes its residual (quantized_packed_decode.py:203-230)."""
    per_head = resid_scale.dim() == 2
    rqmax = QMAX_INT4 if resid_fmt == RESID_INT4 else QMAX_INT8
    for n in range(h.shape[0]):
        slot = int(slots[n])
        if slot <= 0:
            continue
        x = h[n].float()
        s = x.abs().amax(dim=-1).clamp(min=EPS) / QMAX_INT8
        codes = torch.round(x / s[..., None]).clamp(-QMAX_INT8, QMAX_INT8)
        state_codes[slot] = codes.to(torch.int8)
        state_scale[slot] = s
        if not keep_error:
            resid_codes[slot] = 0
            resid_scale[slot] = 0
            continue
        e = x - codes * s[..., None]
        if per_head:
            es = _scale_from_amax(e.abs().amax(dim=(-1, -2)), rqmax, EPS_ON_SCALE)
            ec = torch.round(e / es[..., None, None]).clamp(-rqmax, rqmax)
        else:
            es = _scale_from_amax(e.abs().amax(dim=-1), rqmax, EPS_ON_SCALE)
            ec = torch.round(e / es[..., None]).clamp(-rqmax, rqmax)
        ec = ec.to(torch.int8)
        resid_scale[slot] = es
        resid_codes[slot] = pack_int4(ec) if resid_fmt == RESID_INT4 else ec


def pool_load(state_codes, state_scale, resid_codes, resid_scale, slots,
              resid_fmt: int = RESID_INT8, with_residual: bool = True, dtype=torch.float32):
    """``[B, HV, V, K]``: ``codes * scale`` plus, with ``with_residual``,
    ``resid_codes * resid_scale`` -- the sum :func:`packed_decode_step` forms
    before it re-quantises -- for each slot; zeros for slot ids ``<= 0``."""
    _, HV, V, K = state_codes.shape
    per_head = resid_scale.dim() == 2
    out = torch.zeros((len(slots), HV, V, K), dtype=torch.float32)
    for n in range(len(slots)):
        slot = int(slots[n])
        if slot <= 0:
            continue
        x = state_codes[slot].float() * state_scale[slot][..., None]
        if with_residual:
            rc = resid_codes[slot]
            rc = unpack_int4(rc).float() if resid_fmt == RESID_INT4 else rc.float()
            rs = resid_scale[slot]
            x = x + rc * (rs[..., None, None] if per_head else rs[..., None])
        out[n] = x
    return out.to(dtype)


def pool_copy(src_pool, dst_pool, src_slots, dst_slots):
    """Slot ``src_slots[n]`` of ``src_pool`` onto slot ``dst_slots[n]`` of
    ``dst_pool``, all four tensors; pairs with an id ``<= 0`` skipped."""
    for s, d in zip(src_slots.tolist(), dst_slots.tolist()):
        if s <= 0 or d <= 0:
            continue
        for a, b in zip(src_pool, dst_pool):
            b[d] = a[s].clone()
