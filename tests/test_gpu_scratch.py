"""A context's scratch: what earlier launches allocated is enough for later ones of no greater size, whatever their hints
and their number of rows, so a launch can be captured and stays valid while others follow."""
import numpy as np
import pytest

import oracle
from geistlib_b200 import api
from helpers import independent_states, normal_logits, per_seq, to_dev, u64_from_dev, u64_to_dev

pytestmark = pytest.mark.gpu
LANES = 4


def launches(ctx, rows, V, T, K, P, seed, **kw):
    """A prepared launch and the CPU checker's answer to it."""
    x = normal_logits(rows, V, 1.2, seed)
    st = independent_states(oracle.port, seed, rows)
    dev = to_dev(x), *per_seq(rows, T, K, P), u64_to_dev(st)
    d = ctx.sample_batch(*dev, launch=False, **kw)
    d["_inputs"] = dev  # the descriptor holds pointers into these
    return d, oracle.port.sample_batch(x, T, K, P, st)


def right(d, o):
    assert (d["status"].cpu().numpy() & api.ROW_INVALID == 0).all()
    assert np.array_equal(d["tokens"].cpu().numpy(), o["tokens"])
    assert np.array_equal(u64_from_dev(d["rng_state"]), o["rng_state"])


@pytest.mark.parametrize("first,then", [
    # a launch that was hinted as top-k, then the same size with every kind of row
    (dict(rows=40, V=20000, T=0.8, K=40, P=1.0, finish_hint=api.FINISH_GREEDY_TOPK), dict(rows=40, V=20000)),
    # few long rows, then many short ones
    (dict(rows=2, V=400000, T=0.9, K=0, P=0.9), dict(rows=150, V=600)),
])
def test_a_later_launch_is_captured_without_allocating(first, then):
    import torch
    ctx = api.Context(0)
    d0, o0 = launches(ctx, seed=1, **first)
    T = np.where(np.arange(then["rows"]) % 3 == 0, 0.0, 0.9).astype(np.float32)
    d1, o1 = launches(ctx, T=T, K=0, P=0.9, seed=2, **then)
    s = torch.cuda.Stream()
    for _ in range(LANES):
        ctx.relaunch(d0, s.cuda_stream)
    s.synchronize()
    right(d0, o0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.relaunch(d1, s.cuda_stream)
    # more rows of every kind in between: the captured launch keeps what it was captured with
    d2, o2 = launches(ctx, rows=then["rows"] + 40, V=300, T=0.9, K=0, P=0.9, seed=3)
    for _ in range(LANES):
        ctx.relaunch(d2, s.cuda_stream)
    s.synchronize()
    right(d2, o2)
    for _ in range(2):
        d1["tokens"].fill_(-7)
        with torch.cuda.stream(s):
            g.replay()
        s.synchronize()
        right(d1, o1)
    del g
    ctx.close()


def test_accept_behind_launches_on_two_streams_is_captured(ctx):
    """The accept rule's kernel behind sampling launches that two streams made, in one graph."""
    import torch
    n, k, V = 6, 3, 5000
    d0, o0 = launches(ctx, rows=n * k // 2, V=V, T=0.0, K=0, P=1.0, seed=4)
    d1, o1 = launches(ctx, rows=n * k // 2, V=V, T=0.0, K=0, P=1.0, seed=5)
    want = np.concatenate([o0["tokens"], o1["tokens"]]).reshape(n, k)
    fed = np.full((n, k), 3, np.int32)
    for i in range(n):  # sequence i accepts its first i % k proposals
        fed[i, 1:1 + i % k] = want[i, :i % k]
        fed[i, 1 + i % k:] = (want[i, i % k:k - 1] + 1) % V
    out = torch.full((n * k,), -7, dtype=torch.int32, device="cuda")
    for d, at in ((d0, 0), (d1, n * k // 2)):
        d["_desc"].tokens = out[at:].data_ptr()
    dfed = to_dev(fed)
    acc, nem, em = (torch.full(s, -7, dtype=torch.int32, device="cuda") for s in ((n,), (n,), (n, k + 1)))
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(LANES):
        ctx.relaunch(d0, s.cuda_stream)
    s.synchronize()
    out.fill_(-7)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        t.wait_stream(s)
        ctx.relaunch(d0, s.cuda_stream)
        ctx.relaunch(d1, t.cuda_stream)
        s.wait_stream(t)
        api._check(api.lib.geist_b200_accept_batch(ctx.handle, n, k, dfed.data_ptr(), out.data_ptr(), acc.data_ptr(), nem.data_ptr(), em.data_ptr(), s.cuda_stream))
    for _ in range(3):
        out.fill_(-7)
        acc.fill_(-7)
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            g.replay()
        s.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(n, k), want)
        assert np.array_equal(acc.cpu().numpy(), np.arange(n) % k)
        assert np.array_equal(em.cpu().numpy()[:, 0], fed[:, 0])
    del g
