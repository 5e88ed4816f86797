"""The one-launch move of a slot through a stack of layers, at the edges of what one launch holds (48 layers) and with runs
that are not multiples of 16 bytes; and the slot ids of a batch, whatever its length and on whatever stream they are read."""

from __future__ import annotations

import pytest
import torch

from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("layers,HV,V,K", [(1, 32, 128, 128), (3, 1, 5, 6), (48, 2, 16, 32), (49, 3, 64, 64)])
@pytest.mark.parametrize("resid_fmt,rscale", [(qpd.RESID_INT4, "head"), (qpd.RESID_INT8, "v")])
def test_layer_stack_moves_bit_for_bit(layers, HV, V, K, resid_fmt, rscale):
    from carrykernel_b200.vllm_integration.state_cache import SlotCache
    g = torch.Generator().manual_seed(layers)
    c = SlotCache(layers, 4, HV, V, K, DEV, resid_fmt, rscale, spill_slots=2)
    c.allocate("a"), c.allocate("b")
    for pool in c.pools:
        for t in pool:
            x = torch.randint(-128, 128, t.shape, generator=g) if t.dtype == torch.int8 else torch.randn(t.shape, generator=g)
            t.copy_(x.to(t.dtype))
    before = [[t.clone() for t in pool] for pool in c.pools]
    a, b = c.slot("a"), c.slot("b")
    c.preempt("a")
    new = c.fork("b", "child")                       # takes a's old slot
    assert new == a
    back = c.resume("a")
    assert back not in (a, b)
    for pool, was in zip(c.pools, before):
        for t, w in zip(pool, was):
            assert torch.equal(t[a], w[b]) and torch.equal(t[b], w[b]) and torch.equal(t[back], w[a])
            assert torch.equal(t[0], w[0])


@pytest.mark.parametrize("n", [1, 959, 960, 961, 2000])
def test_indices_of_any_length(n):
    from carrykernel_b200.vllm_integration.state_cache import SlotCache
    c = SlotCache(1, n + 1, 1, 2, 2, DEV)
    for r in range(n):
        c.allocate(r)
    idx = c.indices(range(n), pad_to=n + 3)
    assert idx.dtype == torch.int32 and idx.is_cuda
    assert idx.tolist() == [c.slot(r) for r in range(n)] + [0, 0, 0]


def test_indices_are_in_place_for_any_stream():
    """Ids asked for on a stream that is busy are read by another one that waits for nothing."""
    from carrykernel_b200.vllm_integration.state_cache import SlotCache
    n = 1000
    c = SlotCache(1, n + 1, 1, 2, 2, DEV)
    for r in range(n):
        c.allocate(r)
    want = [c.slot(r) for r in range(n)]
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    c.indices(range(n))                              # whatever is set up on first use
    with torch.cuda.stream(busy):
        stale = torch.full((n,), -5, dtype=torch.int32, device=DEV)      # what a block of this size holds
        torch.cuda.synchronize()
        del stale
        torch.cuda._sleep(100_000_000)               # 50 ms
        idx = c.indices(range(n))
    with torch.cuda.stream(other):
        seen = idx.clone()
    other.synchronize()
    assert seen.tolist() == want
    busy.synchronize()
