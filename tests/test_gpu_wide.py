"""Top-p rows with wide nuclei (sampler_wide.cuh) against the CPU checker: rows around the pieces they are dealt out in,
off the 16-byte grid, more rows than row copies, every way a row can be changed, ties, and long lists."""
import numpy as np
import pytest

import oracle
from geistlib_b200 import api
from helpers import histories, independent_states, normal_logits, per_seq, to_dev, u64_to_dev
from test_gpu_parity import check_tokens, run_gpu

pytestmark = pytest.mark.gpu
RANKED = 512  # lists up to here are walked by ranking (kWideRank)


def same(g, o):
    check_tokens(g, o)
    assert np.array_equal(g["kept_n"], o["detail_n"])


@pytest.mark.parametrize("V,rows", [(33, 5), (511, 7), (512, 7), (513, 9), (1025, 3), (1537, 700), (4096, 24), (4099, 40), (8193, 300), (100003, 24), (128256, 3)])
@pytest.mark.parametrize("kind", ["plain", "rep", "freq", "mask"])
def test_pieces_and_changes(ctx, V, rows, kind):
    x = normal_logits(rows, V, 1.0, V + rows)
    st = independent_states(oracle.port, 3, rows)
    P = np.linspace(0.5, 0.98, rows).astype(np.float32)
    kw, okw, xo = {}, {}, x
    if kind in ("rep", "freq"):
        h = histories(rows, 70 if kind == "rep" else 1100, V, 4)
        kw = {"history": h, "rep": 1.3, "freq": 0.1 if kind == "freq" else 0.0, "pres": 0.2}
        okw = {"hist": h, "rep": 1.3, "freq": kw["freq"], "pres": 0.2}
    if kind == "mask":
        allowed = np.random.default_rng(5).random((rows, V)) < 0.7
        allowed[:, :2] = True
        words = np.zeros((rows, (V + 31) // 32 * 32), bool)
        words[:, :V] = allowed
        kw = {"logit_mask": to_dev(np.packbits(words, axis=1, bitorder="little").view(np.int32))}
        xo = np.where(allowed, x, np.float32(-np.inf)).astype(np.float32)
    g = run_gpu(ctx, x, 1.1, 0, P, st, kept_cap=4, **kw)
    same(g, oracle.port.sample_batch(xo, 1.1, 0, P, st, detail_cap=4, **okw))
    opened, by_lists, longest = ctx.wide_counts()[:3]
    if V > 1000:  # normal rows: wide, and all of them decided where they are shared out
        assert opened > rows // 2 and by_lists == opened and 0 < longest <= RANKED, (opened, by_lists, longest)
        assert ((g["status"] & api.ROW_SLOW_PATH) != 0).sum() == opened


@pytest.mark.parametrize("V,step", [(6000, 0.25), (50000, 0.0625), (50000, 0.5), (9001, 100.0)])
def test_rows_of_few_values(ctx, V, step):
    """Ties by the hundred or the thousand, as logits that were 16 bits wide have them: long lists, and where they outrun
    their room the multi-pass path."""
    rows = 12
    x = (np.round(normal_logits(rows, V, 1.5, 6) / step) * step).astype(np.float32)
    st = independent_states(oracle.port, 7, rows)
    P = np.linspace(0.3, 0.97, rows).astype(np.float32)
    same(run_gpu(ctx, x, 0.9, 0, P, st, kept_cap=4), oracle.port.sample_batch(x, 0.9, 0, P, st, detail_cap=4))
    opened, by_lists, longest = ctx.wide_counts()[:3]
    if step == 100.0:  # one value: the candidates outrun their room already, the row is not shared out
        assert opened == 0
    else:
        assert by_lists > 0
    if V == 50000:
        assert longest > RANKED, (opened, by_lists, longest)


def test_rows_that_their_lists_do_not_decide(ctx):
    """A few hundred large values and then 40000 equal ones, in which the crossing falls: more than a list holds."""
    rows, V = 8, 40400
    rng = np.random.default_rng(12)
    x = np.zeros((rows, V), np.float32)
    for r in range(rows):
        x[r, rng.choice(V, 400, replace=False)] = rng.uniform(3.0, 4.5, 400)
    st = independent_states(oracle.port, 13, rows)
    P = np.linspace(0.6, 0.97, rows).astype(np.float32)
    same(run_gpu(ctx, x, 0.9, 0, P, st, kept_cap=4), oracle.port.sample_batch(x, 0.9, 0, P, st, detail_cap=4))
    assert ctx.wide_counts()[:2] == (rows, 0)


def test_rows_written_out_and_mixed_with_others(ctx):
    """Wide rows between greedy, top-k and temperature ones, launched several times over, their logits written out."""
    rows, V, H = 64, 30000, 40
    x = normal_logits(rows, V, 1.2, 8)
    h = histories(rows, H, V, 9)
    T = np.where(np.arange(rows) % 4 == 0, 0.0, 0.9).astype(np.float32)
    K = np.where(np.arange(rows) % 4 == 1, 30, 0).astype(np.int32)
    P = np.where(np.arange(rows) % 4 == 2, 1.0, 0.9).astype(np.float32)
    for seed in range(6):
        st = independent_states(oracle.port, 100 * seed, rows)
        g = run_gpu(ctx, x, T, K, P, st, history=h, rep=1.2, want_logits=seed % 2 == 1)
        check_tokens(g, oracle.port.sample_batch(x, T, K, P, st, hist=h, rep=1.2))


@pytest.mark.parametrize("rows,V", [(24, 60000), (330, 9000)])
def test_a_wait_that_runs_out(rows, V):
    """Thread blocks that wait no time for the others' pieces go on without them: the rows come out the same, and what the
    launch leaves behind serves the next ones as before."""
    ctx = api.Context(0)
    x = normal_logits(rows, V, 1.0, 21)
    st = independent_states(oracle.port, 22, rows)
    o = oracle.port.sample_batch(x, 1.1, 0, 0.95, st, detail_cap=4)
    gave_up = 0
    for wait in (10 ** 12, 0, 10 ** 12):
        api._check(api.lib.geist_b200_set_wide_wait(ctx.handle, wait))
        for _ in range(4):  # every set of scratch
            same(run_gpu(ctx, x, 1.1, 0, 0.95, st, kept_cap=4), o)
            counts = ctx.wide_counts()
            assert counts[0] == rows
            if wait:
                assert counts[1] == rows and counts[3] == 0
            gave_up += counts[3]
    assert gave_up > 0 or V < 60000
    ctx.close()


def test_nobody_waits_in_launches_without_top_p_rows():
    """Thread blocks without a row of their own wait for wide rows only where a launch has top-p rows; a captured launch whose
    rows become top-p rows and temperature rows again between its replays finds out each time."""
    import torch
    ctx = api.Context(0)
    rows, V = 5, 40000
    x = normal_logits(rows, V, 1.0, 31)
    st = independent_states(oracle.port, 32, rows)
    narrow, wide = np.ones(rows, np.float32), np.array([1.0, 0.9, 0.95, 1.0, 0.8], np.float32)
    dev = [to_dev(x), *per_seq(rows, 1.1, 0, narrow), u64_to_dev(st)]
    d = ctx.sample_batch(*dev, launch=False)
    s = torch.cuda.Stream()
    for _ in range(4):
        ctx.relaunch(d, s.cuda_stream)
    s.synchronize()
    assert ctx.wide_counts()[0] == 0 and ctx.wide_counts()[4] == 0
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.relaunch(d, s.cuda_stream)
    for P in (narrow, wide, wide, narrow, wide):
        dev[3].copy_(to_dev(P))
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            g.replay()
        s.synchronize()
        o = oracle.port.sample_batch(x, 1.1, 0, P, st)
        assert np.array_equal(d["tokens"].cpu().numpy(), o["tokens"])
        counts = ctx.wide_counts()
        assert counts[:2] == ((3, 3) if P is wide else (0, 0))
        assert counts[4] == 1 if P is wide else True
    del g
    for P, waits in ((narrow, False), (wide, True), (narrow, False)):  # launched anew, each is told apart
        dev[3].copy_(to_dev(P))
        for _ in range(4):
            ctx.relaunch(d, s.cuda_stream)
            s.synchronize()
            assert (ctx.wide_counts()[4] == 1) == waits
    ctx.close()


@pytest.mark.parametrize("V,seqs,k", [(5000, 3, 4), (40001, 8, 6), (9000, 80, 5)])
def test_wide_verify_rows(ctx, V, seqs, k):
    """Rows of one sequence share a generator word, and each counts the tokens fed before it; also more rows than row copies."""
    rows = seqs * k
    x = normal_logits(rows, V, 1.0, 41)
    st = independent_states(oracle.port, 42, seqs)
    h, fed = histories(seqs, 50, V, 43), histories(seqs, k, V, 44)
    P = np.linspace(0.6, 0.97, seqs).astype(np.float32)
    g = run_gpu(ctx, x, 1.1, 0, P, st, rows_per_seq=k, history=h, fed=fed, rep=1.3, freq=0.05, kept_cap=4)
    same(g, oracle.port.sample_batch(x, 1.1, 0, P, st, rows_per_seq=k, hist=h, extra=fed, rep=1.3, freq=0.05, detail_cap=4))
    assert ctx.wide_counts()[:2] == (rows, rows)


@pytest.mark.parametrize("cap", [0.0, 3.0])
def test_wide_rows_with_all_changes(ctx, cap):
    """Cap, then mask, then the penalties of a long history, on rows on and off the 16-byte grid."""
    for V, rows in ((20000, 9), (20003, 9)):
        x = normal_logits(rows, V, 1.0, 51)
        st = independent_states(oracle.port, 52, rows)
        h = histories(rows, 700, V, 53)
        allowed = np.random.default_rng(54).random((rows, V)) < 0.8
        words = np.zeros((rows, (V + 31) // 32 * 32), bool)
        words[:, :V] = allowed
        kw = {"logit_mask": to_dev(np.packbits(words, axis=1, bitorder="little").view(np.int32))}
        xo = np.where(allowed, x, np.float32(-np.inf)).astype(np.float32)
        if cap > 0.0:
            # the capped row as the device writes it out for a temperature draw: tanhf is not the subject here
            kw["softcap"] = to_dev(np.full(rows, cap, np.float32))
            xo = run_gpu(ctx, x, 1.1, 0, 1.0, st, want_logits=True, **kw)["logits"]
        g = run_gpu(ctx, x, 1.1, 0, 0.95, st, history=h, rep=1.2, freq=0.1, pres=0.1, kept_cap=4, **kw)
        same(g, oracle.port.sample_batch(xo, 1.1, 0, 0.95, st, hist=h, rep=1.2, freq=0.1, pres=0.1, detail_cap=4))
        assert ctx.wide_counts()[:2] == (rows, rows)


def test_wide_rows_on_two_streams_at_once():
    """Launches with wide rows, each with scratch of its own, that overlap on the GPU."""
    import torch
    ctx = api.Context(0)
    jobs = []
    for i, (rows, V) in enumerate([(12, 60000), (40, 30001)]):
        x, st = normal_logits(rows, V, 1.0, 61 + i), independent_states(oracle.port, 63 + i, rows)
        dev = to_dev(x), *per_seq(rows, 1.1, 0, 0.93), u64_to_dev(st)
        outs = [ctx.sample_batch(*dev, launch=False) for _ in range(2)]
        jobs.append((torch.cuda.Stream(), outs, dev, oracle.port.sample_batch(x, 1.1, 0, 0.93, st)["tokens"]))
    torch.cuda.synchronize()
    for _ in range(10):
        for n in range(2):  # four launches at most in flight: one set of scratch each
            for stream, outs, _, _ in jobs:
                ctx.relaunch(outs[n], stream.cuda_stream)
        torch.cuda.synchronize()
        for _, outs, _, want in jobs:
            for out in outs:
                assert np.array_equal(out["tokens"].cpu().numpy(), want)
                out["tokens"].fill_(-7)
        torch.cuda.synchronize()
    ctx.close()


def test_steps_followed_by_launches_on_other_streams():
    """A step returns when its tokens are there. What comes right behind it must not meet what is left of it: its logits are
    overwritten from another stream, and four launches with wide rows go to four more."""
    import torch
    ctx = api.Context(0)
    n, V, steps = 12, 30001, 12
    bt = api.Batcher(ctx, V, n)
    sess = [bt.open(temperature=1.1, top_p=0.93, seed=70 + i) for i in range(n)]
    state = independent_states(oracle.port, 70, n)
    jobs, keep = [], []  # a descriptor holds pointers only
    for i, rows in enumerate([3, 40, 12, 7]):
        x, st = normal_logits(rows, V, 1.0, 71 + i), independent_states(oracle.port, 90 + i, rows)
        keep.append((to_dev(x), *per_seq(rows, 1.1, 0, 0.93), u64_to_dev(st)))
        jobs.append((torch.cuda.Stream(), ctx.sample_batch(*keep[i], launch=False), oracle.port.sample_batch(x, 1.1, 0, 0.93, st)["tokens"]))
    xs = [normal_logits(n, V, 1.0, 200 + i) for i in range(3)]
    ready = [to_dev(x) for x in xs]
    cur, side = torch.empty_like(ready[0]), torch.cuda.Stream()
    for it in range(steps):
        with torch.cuda.stream(side):
            cur.copy_(ready[it % 3])
        side.synchronize()
        got = bt.step(sess, cur)
        with torch.cuda.stream(side):
            cur.fill_(float("nan"))
        for stream, out, _ in jobs:
            ctx.relaunch(out, stream.cuda_stream)
        o = oracle.port.sample_batch(xs[it % 3], 1.1, 0, 0.93, state)
        assert np.array_equal(got, o["tokens"]), it
        state = o["rng_state"]
        torch.cuda.synchronize()
        for _, out, want in jobs:
            assert np.array_equal(out["tokens"].cpu().numpy(), want), it
            out["tokens"].fill_(-7)
        torch.cuda.synchronize()
    bt.close()
    ctx.close()
