"""GPU parity of what happens to a row before it is sampled — the final-logit soft cap
(head.c:145-159, :279-288), the mask of allowed columns — of the finishing hints, and one
penalty-free case per sampler mode straight against the reference's own sampler.c."""
import numpy as np
import pytest

import oracle
from geistlib_b200 import api
from helpers import gumbel_logits, histories, independent_states, normal_logits, per_seq, rel_err, seq_states, to_dev, u64_to_dev
from test_gpu_parity import check_tokens, run_gpu

pytestmark = pytest.mark.gpu
CAP_RTOL = 1e-5  # device tanhf against the host's: both within a few ulp of the true value

needs_ref = pytest.mark.skipif(oracle.ref is None, reason="oracle/_ref not built")


def cap_dev(n_seq, c):
    return to_dev(np.broadcast_to(np.asarray(c, np.float32), (n_seq,)))


def mask_words(allowed):
    """bool [rows, V] -> int32 words [rows, ceil(V / 32)], bit i of a row = column i allowed."""
    rows, V = allowed.shape
    W = (V + 31) // 32
    pad = np.zeros((rows, W * 32), bool)
    pad[:, :V] = allowed
    w = np.packbits(pad.reshape(rows, W, 32), axis=2, bitorder="little").view(np.uint32).reshape(rows, W)
    return np.ascontiguousarray(w.view(np.int32))


@needs_ref
@pytest.mark.parametrize("shape", ["c1", "c3"])
def test_softcap_logits_and_tokens(ctx, shape):
    """c = 30 on rows shaped like the single-row case (temperature 0.8, top-k 40) and like the
    nucleus case (Gumbel rows, top-p): capped logits within 1e-5 of the host's tanhf, tokens equal."""
    c = 30.0
    if shape == "c1":
        rows, V = 24, 128256
        x = normal_logits(rows, V, 12.0, 41)  # wide enough for the cap to bend the top of the row
        T, K, P = 0.8, 40, 0.95
        st = independent_states(oracle.port, 41, rows)
    else:
        rows, V = 24, 262144
        x = gumbel_logits(rows, V, 4.0, 43)
        T, K, P = 0.9, 0, 0.9
        st = seq_states(oracle.port, 43, rows)
    capped = oracle.ref.softcap(x, c)
    g = run_gpu(ctx, x, T, K, P, st, softcap=cap_dev(rows, c), want_logits=True)
    assert rel_err(g["logits"], capped) <= CAP_RTOL
    assert np.abs(g["logits"]).max() <= c
    o = oracle.ref.sample(capped, T, K, P, st)
    check_tokens(g, o)


def test_softcap_skipped_for_greedy_and_zero(ctx):
    """T == 0 rows skip the cap (head.c:145-149) and c == 0 means none: both bit-identical to no cap at all."""
    rows, V = 8, 50257
    x = normal_logits(rows, V, 20.0, 3)
    st = independent_states(oracle.port, 3, rows)
    T = np.array([0.0, 0.7] * 4, np.float32)
    caps = np.array([30.0, 0.0] * 4, np.float32)
    g = run_gpu(ctx, x, T, 40, 1.0, st, softcap=to_dev(caps), want_logits=True)
    assert np.array_equal(g["logits"].view(np.uint32), x.view(np.uint32))
    check_tokens(g, oracle.port.sample_batch(x, T, 40, 1.0, st))


def test_softcap_then_penalties_temperature_and_verify_rows(ctx):
    """The cap comes before the penalties; temperature rows re-read a segment of the row in the finisher,
    and the rows of one sequence share its cap."""
    S, R, V, H = 6, 3, 32000, 48
    x = normal_logits(S * R, V, 9.0, 77)
    h = histories(S, H, V, 78)
    st = independent_states(oracle.port, 77, S)
    c = 25.0
    g = run_gpu(ctx, x, 1.0, 0, 1.0, st, rows_per_seq=R, softcap=cap_dev(S, c), rep=1.2, history=h, want_logits=True)
    capped = oracle.port.softcap(x, c)
    o = oracle.port.sample_batch(capped, 1.0, 0, 1.0, st, rows_per_seq=R, rep=1.2, hist=h, want_logits=True)
    assert rel_err(g["logits"], o["logits"]) <= CAP_RTOL
    check_tokens(g, o)


def test_softcap_wide_nucleus_path(ctx):
    """Rows whose nucleus is too wide for one pass take the multi-pass path, which caps its own copy of the row."""
    rows, V = 4, 40000
    x = normal_logits(rows, V, 2.0, 9)
    st = independent_states(oracle.port, 9, rows)
    g = run_gpu(ctx, x, 1.0, 0, 0.95, st, softcap=cap_dev(rows, 30.0))
    assert (g["status"] & api.ROW_SLOW_PATH).any(), "expected the multi-pass path"
    o = oracle.port.sample_batch(oracle.port.softcap(x, 30.0), 1.0, 0, 0.95, st)
    check_tokens(g, o)


@pytest.mark.parametrize("mode", ["greedy", "topk", "topp", "temp"])
def test_logit_mask(ctx, mode):
    """Masked columns read as -inf: the sampled ids are those of the CPU sampler on rows with -inf written in."""
    rows, V = 12, 50257
    x = normal_logits(rows, V, 2.5, 500)
    rng = np.random.default_rng(501)
    allowed = rng.random((rows, V)) < 0.3
    allowed[0, :] = False
    allowed[0, 4097] = True          # a single allowed column
    allowed[1, :] = True             # nothing masked
    allowed[2, x[2].argmax()] = False  # the winner is masked
    T, K, P = {"greedy": (0.0, 0, 1.0), "topk": (0.8, 40, 1.0), "topp": (0.8, 0, 0.6), "temp": (1.0, 0, 1.0)}[mode]
    st = independent_states(oracle.port, 500, rows)
    g = run_gpu(ctx, x, T, K, P, st, logit_mask=to_dev(mask_words(allowed)), want_logits=True)
    xm = np.where(allowed, x, -np.inf).astype(np.float32)
    assert np.array_equal(g["logits"].view(np.uint32), xm.view(np.uint32))
    check_tokens(g, oracle.port.sample_batch(xm, T, K, P, st))
    assert allowed[np.arange(rows), g["tokens"]].all()
    assert g["tokens"][0] == 4097


def test_logit_mask_with_softcap_and_penalties(ctx):
    rows, V, H = 8, 128256, 64
    x = normal_logits(rows, V, 10.0, 600)
    h = histories(rows, H, V, 601)
    allowed = np.random.default_rng(602).random((rows, V)) < 0.5
    st = independent_states(oracle.port, 600, rows)
    g = run_gpu(ctx, x, 0.8, 40, 1.0, st, softcap=cap_dev(rows, 30.0), logit_mask=to_dev(mask_words(allowed)), rep=1.1, history=h)
    xm = np.where(allowed, oracle.port.softcap(x, 30.0), -np.inf).astype(np.float32)
    check_tokens(g, oracle.port.sample_batch(xm, 0.8, 40, 1.0, st, rep=1.1, hist=h))


def test_logit_mask_stride_too_short(ctx):
    rows, V = 2, 1000
    x = to_dev(normal_logits(rows, V, 1.0, 1))
    import torch
    m = torch.zeros(rows, 8, dtype=torch.int32, device="cuda")  # 256 bits < V
    dT, dK, dP = to_dev(np.zeros(rows, np.float32)), to_dev(np.zeros(rows, np.int32)), to_dev(np.ones(rows, np.float32))
    with pytest.raises(api.GeistError, match="GEIST_E_INVALID_ARG"):
        ctx.sample_batch(x, dT, dK, dP, to_dev(np.ones(rows, np.int64)), logit_mask=m)


# ------------------------------------------------------------- finishing hints --

def test_finish_hint_same_tokens(ctx):
    """A correct hint changes which kernels run, never a token."""
    rows, V = 64, 128256
    x = normal_logits(rows, V, 2.5, 900)
    st = independent_states(oracle.port, 900, rows)
    T = np.where(np.arange(rows) % 2 == 0, 0.0, 0.8).astype(np.float32)
    auto = run_gpu(ctx, x, T, 40, 1.0, st)
    fast = run_gpu(ctx, x, T, 40, 1.0, st, finish_hint=api.FINISH_GREEDY_TOPK)
    gen = run_gpu(ctx, x, T, 40, 1.0, st, finish_hint=api.FINISH_GENERAL)
    check_tokens(fast, auto)
    check_tokens(gen, auto)
    check_tokens(auto, oracle.port.sample_batch(x, T, 40, 1.0, st))
    # rows of the other modes through the general kernel alone
    Tm = np.full(rows, 0.9, np.float32)
    Pm = np.where(np.arange(rows) % 2 == 0, 1.0, 0.5).astype(np.float32)
    check_tokens(run_gpu(ctx, x, Tm, 0, Pm, st, finish_hint=api.FINISH_GENERAL), oracle.port.sample_batch(x, Tm, 0, Pm, st))


@pytest.mark.parametrize("rows,V,R", [(256, 5000, 1), (200, 40000, 1), (64, 128256, 1), (300, 9000, 1), (240, 3000, 3)])
def test_finish_hint_greedy(ctx, rows, V, R):
    """All rows greedy and the caller says so: whole-row launches write the tokens from the stream kernel alone
    (no finishing kernel), split-row launches merge as usual; ids, status and generator words as without the hint."""
    x = normal_logits(rows, V, 3.0, 77 + rows)
    x[3, :] = 1.5           # all equal: lowest index
    x[5, V // 3:] = x[5].max() + 2.0
    S = rows // R
    st = independent_states(oracle.port, 5, S)
    h = histories(S, 40, V, 6)
    g = run_gpu(ctx, x, 0.0, 0, 1.0, st, rows_per_seq=R, finish_hint=api.FINISH_GREEDY, freq=0.4, history=h)
    o = oracle.port.sample_batch(x, 0.0, 0, 1.0, st, rows_per_seq=R, freq=0.4, hist=h)
    check_tokens(g, o)
    assert np.array_equal(g["rng_state"], st), "greedy rows draw nothing"


def test_finish_hint_greedy_wrong_is_loud(ctx):
    from helpers import u64_to_dev
    rows, V = 256, 4000
    x = normal_logits(rows, V, 3.0, 9)
    T = np.zeros(rows, np.float32)
    T[17] = 0.7
    dT, dK, dP = to_dev(T), to_dev(np.zeros(rows, np.int32)), to_dev(np.ones(rows, np.float32))
    out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(independent_states(oracle.port, 1, rows)), finish_hint=api.FINISH_GREEDY)
    status, tok = out["status"].cpu().numpy(), out["tokens"].cpu().numpy()
    assert status[17] & api.ROW_INTERNAL and tok[17] == -1
    ok = np.arange(rows) != 17
    assert (status[ok] & api.ROW_INVALID == 0).all() and np.array_equal(tok[ok], x[ok].argmax(axis=1))


def test_finish_hint_wrong_is_loud(ctx):
    """GREEDY_TOPK with a temperature row in the batch: that row reports ROW_INTERNAL and token -1, the others are sampled."""
    import torch
    rows, V = 8, 32000
    x = normal_logits(rows, V, 2.5, 901)
    st = independent_states(oracle.port, 901, rows)
    T = np.full(rows, 0.8, np.float32)
    K = np.full(rows, 40, np.int32)
    K[3] = 0  # plain temperature sampling
    dT, dK, dP = to_dev(T), to_dev(K), to_dev(np.ones(rows, np.float32))
    from helpers import u64_to_dev
    out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), finish_hint=api.FINISH_GREEDY_TOPK)
    status, tok = out["status"].cpu().numpy(), out["tokens"].cpu().numpy()
    assert status[3] & api.ROW_INTERNAL and tok[3] == -1
    ok = np.arange(rows) != 3
    assert (status[ok] & api.ROW_INVALID == 0).all()
    o = oracle.port.sample_batch(x, T, K, 1.0, st)
    assert np.array_equal(tok[ok], o["tokens"][ok])
    with pytest.raises(api.GeistError, match="GEIST_E_INVALID_ARG"):
        ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), finish_hint=9)


# ------------------------------------- every mode against the reference's own code --

@needs_ref
@pytest.mark.parametrize("mode,T,K,P", [("argmax", 0.0, 0, 1.0), ("top_k", 0.8, 40, 0.95), ("top_k_wide", 1.0, 300, 1.0),
                                        ("top_p", 0.8, 0, 0.9), ("temperature", 1.1, 0, 1.0)])
def test_mode_against_reference_sampler(ctx, mode, T, K, P):
    """No penalties, no extension in play: the CUDA path against src/engine/sampler.c itself (oracle/_ref)."""
    rows, V = 48, 128256
    x = gumbel_logits(rows, V, 3.0, 1000) if mode == "top_p" else normal_logits(rows, V, 2.5, 1000)
    x[:, :4] += 9.0
    st = seq_states(oracle.port, 1000, rows)
    g = run_gpu(ctx, x, T, K, P, st)
    check_tokens(g, oracle.ref.sample(x, T, K, P, st))


# ------------------------------------------------------ how the items are dealt out --

@pytest.mark.parametrize("V", [700, 9000, 20000])  # 1, 2 and 3 slices per row
def test_run_maps_over_row_counts(ctx, V):
    """Row counts on both sides of every switch between the three ways of cutting the item list (whole rows,
    rows cut into equal parts, equal runs of items), with each hint's weighting: the tokens never depend on it."""
    sm2 = 2 * 148
    counts = sorted({1, 2, 3, 37, 73, 74, 75, 147, 148, 149, 150, 200, 255, 256, 257, sm2 - 1, sm2, sm2 + 1, 300, 2 * sm2 - 1, 2 * sm2, 2 * sm2 + 1, 640})
    rows_max = max(counts)
    x = normal_logits(rows_max, V, 2.5, 4000 + V)
    x[:, :3] += 6.0
    st = independent_states(oracle.port, 4000, rows_max)
    h = histories(rows_max, 24, V, 4001)
    for mode, (T, K, P), hints in [("greedy", (0.0, 0, 1.0), (api.FINISH_AUTO, api.FINISH_GREEDY_TOPK, api.FINISH_GREEDY)),
                                   ("topk", (0.8, 40, 1.0), (api.FINISH_AUTO, api.FINISH_GREEDY_TOPK)),
                                   ("temp", (1.0, 0, 1.0), (api.FINISH_AUTO, api.FINISH_GENERAL))]:
        o = oracle.port.sample_batch(x, T, K, P, st, rep=1.1, hist=h)
        for n in counts:
            for hint in hints:
                g = run_gpu(ctx, x[:n], T, K, P, st[:n], rep=1.1, history=h[:n], finish_hint=hint)
                bad = np.nonzero(g["tokens"] != o["tokens"][:n])[0]
                assert bad.size == 0, (mode, n, hint, bad[:5])
                assert np.array_equal(g["rng_state"], o["rng_state"][:n]), (mode, n, hint)


def test_small_finisher_hands_back_rows_whose_candidates_overflow(ctx):
    """GREEDY_TOPK promises greedy / top-k rows, not easy ones. A top-k row with thousands of equal values at the
    top (more candidates than the small kernel's lists hold) comes back unsampled with ROW_RETRY; launched again
    without the hint it is sampled. The batcher does that second launch itself."""
    from helpers import u64_to_dev
    rows, V = 6, 128256
    x = normal_logits(rows, V, 2.5, 4242)
    x[0, 1000:9000] = 30.0          # 8000 ties at the top: the k kept are the lowest ids among them
    x[1, :] = 1.0                   # a flat row
    x[2, ::3] = x[2].max() + 1.0    # every third entry tied
    st = independent_states(oracle.port, 4242, rows)
    for K in (40, 200):
        o = oracle.port.sample_batch(x, 0.9, K, 1.0, st)
        dT, dK, dP = to_dev(np.full(rows, 0.9, np.float32)), to_dev(np.full(rows, K, np.int32)), to_dev(np.ones(rows, np.float32))
        out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), finish_hint=api.FINISH_GREEDY_TOPK)
        status, tok = out["status"].cpu().numpy(), out["tokens"].cpu().numpy()
        assert (status[:3] & api.ROW_RETRY).all() and (tok[:3] == -1).all()
        assert (status[3:] & (api.ROW_RETRY | api.ROW_INVALID) == 0).all() and np.array_equal(tok[3:], o["tokens"][3:])
        check_tokens(run_gpu(ctx, x, 0.9, K, 1.0, st), o)  # the same rows without the hint
    bt = api.Batcher(ctx, V, 8)
    sess = [bt.open(temperature=0.9, top_k=40, top_p=1.0, seed=4242 + i) for i in range(rows)]  # all top-k: the batcher gives the hint
    got = bt.step(sess, to_dev(x))
    assert np.array_equal(got, oracle.port.sample_batch(x, 0.9, 40, 1.0, st)["tokens"])
    for i, s_ in enumerate(sess):
        assert bt.get_rng(s_) == oracle.port.rng_advance(int(st[i]), 1)
    bt.close()


def test_stream_kernel_finishes_whole_rows_itself(ctx):
    """GREEDY_TOPK on a launch that deals whole rows: no finishing kernel runs, the stream kernel's thread blocks
    finish greedy and top-k rows from their own lists. Same tokens and generator words as without the hint; rows
    whose candidates do not fit come back with ROW_RETRY."""
    from helpers import u64_to_dev
    rows, V = 200, 128256
    x = normal_logits(rows, V, 2.5, 777)
    x[:, :5] += 7.0
    x[3, 2000:9000] = 40.0   # thousands of ties at the top
    x[4, :] = 0.5            # flat
    st = independent_states(oracle.port, 777, rows)
    h = histories(rows, 64, V, 778)
    T = np.where(np.arange(rows) % 5 == 0, 0.0, 0.8).astype(np.float32)
    K = np.where(np.arange(rows) % 3 == 0, 200, 40).astype(np.int32)
    o = oracle.port.sample_batch(x, T, K, 1.0, st, rep=1.1, hist=h)
    assert api.grid(V, rows, 64)["thread_blocks"] == rows  # whole rows
    dT, dK, dP = to_dev(T), to_dev(K), to_dev(np.ones(rows, np.float32))
    out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), rep=to_dev(np.full(rows, 1.1, np.float32)), history=to_dev(h),
                           history_len=to_dev(np.full(rows, 64, np.int32)), finish_hint=api.FINISH_GREEDY_TOPK)
    status, tok = out["status"].cpu().numpy(), out["tokens"].cpu().numpy()
    retry = (status & api.ROW_RETRY) != 0
    assert retry[3] and retry[4] and retry.sum() == 2 and (tok[retry] == -1).all()
    assert (status[~retry] & api.ROW_INVALID == 0).all()
    assert np.array_equal(tok[~retry], o["tokens"][~retry])
    from helpers import u64_from_dev
    assert np.array_equal(u64_from_dev(out["rng_state"]), o["rng_state"])
    # verify rows (three per sequence) through the same path
    S, R = 66, 3
    xv = normal_logits(S * R, V, 2.5, 779)
    sv = independent_states(oracle.port, 779, S)
    g = run_gpu(ctx, xv, 0.9, 50, 1.0, sv, rows_per_seq=R, finish_hint=api.FINISH_GREEDY_TOPK)
    check_tokens(g, oracle.port.sample_batch(xv, 0.9, 50, 1.0, sv, rows_per_seq=R))


@pytest.mark.parametrize("c,sigma,shiftx", [(30.0, 3.0, 0.0), (30.0, 12.0, 0.0), (5.0, 2.0, 20.0), (1.0, 4.0, 0.0), (30.0, 2.0, -40.0), (1e6, 3.0, 0.0),
                                            (1e30, 3.0, 0.0), (1e-3, 3e-3, 0.0), (2.0, 1e-30, 0.0), (4.0, 2.0, -30.0)])
@pytest.mark.parametrize("hint", [0, 1])
def test_softcap_after_the_select_equals_softcap_before(ctx, c, sigma, shiftx, hint):
    """Top-k rows without ids are selected from uncapped logits and capped afterwards. Asking for the capped logits makes
    the launch cap every logit while it streams, with the same device functions: tokens and kept sets are the same ones,
    from the linear range of the cap to where it saturates and thousands of values are equal."""
    rows, V = 24, 33001
    x = normal_logits(rows, V, sigma, 61) + np.float32(shiftx)
    x[::4, ::3] = -np.inf
    x[3] = np.inf
    x[3, 500:] = 0.0
    st = independent_states(oracle.port, 61, rows)
    K = np.resize(np.array([2, 40, 64, 200], np.int32), rows)
    mask = np.random.default_rng(62).random((rows, V)) < 0.5
    for extra in ({}, {"logit_mask": to_dev(mask_words(mask))}):
        for cap in (0, 256):
            late = run_gpu(ctx, x, 0.8, K, 1.0, st, softcap=cap_dev(rows, c), kept_cap=cap, finish_hint=hint if cap == 0 else 0, **extra)
            full = run_gpu(ctx, x, 0.8, K, 1.0, st, softcap=cap_dev(rows, c), kept_cap=cap, want_logits=True, **extra)
            # every row is served, however many values the cap brings near its k-th, unless a thousand of a part's are equal:
            # row 3 (zeros) and logits that all lie four caps and more below zero
            done = (late["status"] & api.ROW_RETRY) == 0
            assert np.delete(done, 3).all() or (hint and (c, shiftx) == (4.0, -30.0))
            assert np.array_equal(late["tokens"][done], full["tokens"][done])
            if cap:
                both = ((late["status"] | full["status"]) & api.ROW_KEPT_PARTIAL) == 0
                for name in ("kept_n", "kept_idx", "kept_prob"):
                    assert np.array_equal(late[name][both], full[name][both]), name


@pytest.mark.parametrize("V", [4096, 33001, 33004, 151936])
@pytest.mark.parametrize("T,K,P", [(0.0, 0, 1.0), (0.9, 40, 1.0), (0.9, 300, 1.0), (0.8, 0, 0.9), (1.0, 0, 1.0)])
def test_logits_rewritten_where_they_lie(ctx, V, T, K, P):
    """out_logits over logits: the rows end up as they are sampled from and the tokens are those of a launch that writes
    elsewhere, on every route that reads a row again (select, segment walk, the multi-pass path)."""
    rows, H = 12, 90
    x = normal_logits(rows, V, 2.5, V)
    x[::3, :6] += 9.0
    h = histories(rows, H, V, V)
    h[:, :8] = np.argsort(-x, axis=1)[:, :8]
    st = independent_states(oracle.port, V, rows)
    mask = np.random.default_rng(V).random((rows, V)) < 0.7
    kw = dict(rep=1.3, freq=0.2, history=h, softcap=cap_dev(rows, np.resize([30.0, 0.0], rows)), logit_mask=to_dev(mask_words(mask)))
    apart = run_gpu(ctx, x, T, K, P, st, want_logits=True, **kw)
    dT, dK, dP = per_seq(rows, T, K, P)
    dx, drng = to_dev(x), u64_to_dev(st)
    like = ctx.sample_batch(dx, dT, dK, dP, drng, want_logits=True, launch=False)
    like["logits"] = dx
    dev = {"rep": to_dev(np.full(rows, 1.3, np.float32)), "freq": to_dev(np.full(rows, 0.2, np.float32)), "history": to_dev(h),
           "history_len": to_dev(np.full(rows, H, np.int32)), "softcap": kw["softcap"], "logit_mask": kw["logit_mask"]}
    over = ctx.sample_batch(dx, dT, dK, dP, drng, out=like, **dev)
    assert (over["status"].cpu().numpy() & api.ROW_INVALID == 0).all()
    assert np.array_equal(over["logits"].cpu().numpy().view(np.uint32), apart["logits"].view(np.uint32))
    assert np.array_equal(over["tokens"].cpu().numpy(), apart["tokens"])


@pytest.mark.parametrize("V", [33001, 70000, 128256])
def test_softcapped_rows_stay_on_the_short_path(ctx, V):
    """A cap far above the logits (1e6) and one that a third of them pass leave a top-k row to the select: no row is asked
    for again, none goes the long way."""
    rows = 300
    x = normal_logits(rows, V, 3.0, V)
    st = independent_states(oracle.port, V, rows)
    for c in (1e6, 2.2):  # P(|x| > 9.01 c): 0 and about 3e-11; beyond 3 c, where capped values crowd, 2 %
        for hint in (0, 1):
            g = run_gpu(ctx, x, 0.9, 40, 1.0, st, softcap=cap_dev(rows, c), finish_hint=hint)
            assert (g["status"] & (api.ROW_RETRY | api.ROW_SLOW_PATH) == 0).all()


@pytest.mark.parametrize("V,rows", [(8200, 12), (40004, 6), (100004, 300), (262144, 3)])
@pytest.mark.parametrize("c", [0.5, 30.0])
def test_masked_rows_capped_behind_the_select(ctx, V, rows, c):
    """Top-k rows under a cap and a mask: shares of a slice that begin inside a word of the mask, and rows with few allowed columns
    (the cap of a masked column is not -inf). What is kept at caps that rows come close to: the two tests below."""
    rg = np.random.default_rng(V + rows)
    x = normal_logits(rows, V, 2.5, V)
    allowed = rg.random((rows, V)) < 0.5
    allowed[0] = False
    allowed[0, rg.permutation(V)[:60]] = True
    st = np.array([oracle.port.rng_seed(5 + i) for i in range(rows)], np.uint64)
    y = (np.tanh(x / np.float32(c), dtype=np.float32) * np.float32(c)).astype(np.float32)
    y[~allowed] = -np.inf
    got = {}
    for hint in (0, 1):
        dT, dK, dP = per_seq(rows, 0.5, 40, 1.0)
        out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), softcap=to_dev(np.full(rows, c, np.float32)), logit_mask=to_dev(mask_words(allowed)),
                               kept_cap=40, finish_hint=hint)
        status, kept = out["status"].cpu().numpy(), out["kept_idx"].cpu().numpy()
        assert (status & (1 | 4 | 16)).max() == 0
        got[hint] = out["tokens"].cpu().numpy()
        for r in range(rows):
            if status[r] & (8 | 32):
                continue  # not this path
            assert allowed[r, kept[r]].all()
            if c > 1.0:  # the device's tanhf and the host's differ in the last bit: which of near-equal values is kept may too
                assert y[r, kept[r]].min() >= np.sort(y[r])[-40] - 1e-4
        if c > 1.0:
            o = oracle.port.sample_batch(y, 0.5, 40, 1.0, st)
            done = (status & 32) == 0  # row 0: more columns of value -inf at its parts' thresholds than a list holds
            assert done[1:].all() and (hint or done[0])
            assert np.mean((got[hint] == o["tokens"])[done]) >= (1.0 if rows < 100 else 0.99)


@pytest.mark.parametrize("V,rows", [(8200, 300), (40004, 24), (100004, 300), (262144, 12)])
@pytest.mark.parametrize("c", [1.5, 3.0])
def test_kept_values_close_below_the_cap(ctx, V, rows, c):
    """Caps near the rows' largest values, which crowd below them: every row is served by the select, and keeps all ids whose
    capped value is above the k-th by more than the device's and the host's tanhf can differ, and none that is below it by that."""
    k, x = 40, normal_logits(rows, V, 2.5, V) * np.float32(min(1.0, 5.0 * c / (2.5 * 5.3)))  # the largest at about 5 c, where tanh is 1 - 1e-4
    allowed = np.random.default_rng(V).random((rows, V)) < 0.5
    y = np.where(allowed, np.tanh(x.astype(np.float64) / c) * c, -np.inf)
    kth = -np.partition(-y, k - 1, axis=1)[:, k - 1]
    tol = c * 2.0 ** -20  # tanhf, the quotient and the product: 2^-21 of c, on either side of the comparison
    st = np.array([oracle.port.rng_seed(5 + i) for i in range(rows)], np.uint64)
    dT, dK, dP = per_seq(rows, 0.5, k, 1.0)
    for hint in (0, 1):
        out = ctx.sample_batch(to_dev(x), dT, dK, dP, u64_to_dev(st), softcap=cap_dev(rows, c), logit_mask=to_dev(mask_words(allowed)), kept_cap=k, finish_hint=hint)
        assert (out["status"].cpu().numpy() == 0).all()
        for r, kept in enumerate(out["kept_idx"].cpu().numpy()):
            assert len(set(kept)) == k and (y[r, kept] >= kth[r] - tol).all()
            assert set(np.nonzero(y[r] > kth[r] + tol)[0]) <= set(kept)


@pytest.mark.parametrize("V,rows", [(8200, 12), (40004, 6), (100004, 300), (262144, 3)])
def test_rows_whose_kept_ids_all_reach_the_cap(ctx, V, rows):
    """A few per cent of every row come to the cap itself: the k first of them by id are kept, with equal weights. No value lies where
    a tanhf that is good to 2 ulp may or may not come to 1: 2 e^(-2z) is 2.5 * 2^-24 at z = 8.2 and 2^-25 at 9.01. So tokens are those of
    the checker."""
    c, k = 0.5, 40
    x = normal_logits(rows, V, 2.5, V)
    x[(x > 8.1 * c) & (x < 9.5 * c)] = np.float32(10.0 * c)
    allowed = np.random.default_rng(V).random((rows, V)) < 0.5
    y = np.where(allowed, np.tanh(x.astype(np.float64) / c).astype(np.float32) * np.float32(c), np.float32(-np.inf)).astype(np.float32)
    assert ((y == c).sum(axis=1) > k).all()
    st = np.array([oracle.port.rng_seed(5 + i) for i in range(rows)], np.uint64)
    o = oracle.port.sample_batch(y, 0.5, k, 1.0, st)
    g = run_gpu(ctx, x, 0.5, k, 1.0, st, softcap=cap_dev(rows, c), logit_mask=to_dev(mask_words(allowed)))
    assert np.array_equal(g["tokens"], o["tokens"])
