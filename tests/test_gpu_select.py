"""What a part's end and its set-up decide by: the threshold among the threads' maxima, the draw over ordered weights, and a
row's ids counted by the thread block. Tokens and generator states are bit-exact against the CPU checker."""
import numpy as np
import pytest

import oracle
from helpers import independent_states, normal_logits
from test_gpu_parity import check_tokens, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 40, 128, 129, 256])
@pytest.mark.parametrize("V", [2048, 8192, 20011])
def test_threshold_of_uneven_maxima(ctx, V, k):
    """Rows whose maxima fill few of the bins at first: one value far above, rows half of which is -inf, values that span every
    exponent, values a few bits apart; whole rows, and rows cut into parts. Drawn nearly evenly, so that every place counts."""
    for rows, hint in [(256, 1), (20, 0)]:
        x = normal_logits(rows, V, 2.5, V + k)
        rg = np.random.default_rng(V + k)
        x[0::5, V // 7] = 1e30
        x[1::5, : V // 2] = -np.inf
        x[2::5] = (np.sign(x[2::5]) * np.exp2(rg.integers(-120, 120, x[2::5].shape))).astype(np.float32)
        x[3::5] = np.float32(5.0) + rg.integers(0, 4 * V, x[3::5].shape).astype(np.float32) * np.float32(2.0 ** -21)
        T = np.full(rows, 4.0, np.float32)
        T[2::5] = 1e37
        T[3::5] = 1.0
        st = independent_states(oracle.port, V + k, rows)
        g = run_gpu(ctx, x, T, k, 1.0, st, finish_hint=hint)
        assert (g["status"] & 32 == 0).all()
        check_tokens(g, oracle.port.sample_batch(x, T, k, 1.0, st))


@pytest.mark.parametrize("k", [2, 3, 63, 64, 65, 255])
@pytest.mark.parametrize("gap", [0.0, 0.05, 15.0, 16.0, 90.0])
def test_draw_over_weights_of_all_sizes(ctx, k, gap):
    """The last of the kept weights above and below 2^-22 (e^-15.2): added in parallel, and one by one; weights that are 0."""
    rows, V = 320, 4096
    x = np.full((rows, V), -500.0, np.float32)
    rg = np.random.default_rng(k)
    for r in range(rows):
        ids = rg.permutation(V)[:k]
        x[r, ids] = np.linspace(0.0, -gap, k, dtype=np.float32)
    st = independent_states(oracle.port, 11 * k, rows)
    g = run_gpu(ctx, x, 1.0, k, 1.0, st, finish_hint=1)
    assert (g["status"] & 32 == 0).all()
    check_tokens(g, oracle.port.sample_batch(x, 1.0, k, 1.0, st))


@pytest.mark.parametrize("H", [255, 256, 257, 1023, 1024, 1025])
@pytest.mark.parametrize("rows,V", [(300, 4096), (300, 40001), (152, 262144), (3, 151936)])
def test_ids_counted_by_the_thread_block(ctx, rows, V, H):
    """A row's distinct ids by a bit each (penalties that do not count, parts of up to 131072 columns) and by the table (the
    others), one, four per thread and counted ahead of the launch; ids that repeat, that lie outside the vocabulary, and rows
    with fewer of them than the launch allows for."""
    rg = np.random.default_rng(V + H)
    x = normal_logits(rows, V, 2.5, V + H)
    h = rg.integers(0, V, (rows, H)).astype(np.int32)
    likely = np.argpartition(-x, 99, axis=1)[:, :100]
    h[:, : H // 2] = np.take_along_axis(likely, rg.integers(0, 100, (rows, H // 2)), axis=1)
    h[:, -3:] = (-1, V, 2 ** 31 - 1)
    n = np.full(rows, H, np.int32)
    n[1::7] = H // 3
    n[2::7] = 0
    st = independent_states(oracle.port, V + H, rows)
    for freq in (0.0, 0.2):
        g = run_gpu(ctx, x, 0.9, 40, 1.0, st, rep=1.1, freq=freq, pres=0.1, history=h, history_len=n, finish_hint=1)
        assert (g["status"] & 32 == 0).all()
        check_tokens(g, oracle.port.sample_batch(x, 0.9, 40, 1.0, st, rep=1.1, freq=freq, pres=0.1, hist=h, hist_len=n))


@pytest.mark.parametrize("H", [200, 1000])
def test_fed_tokens_behind_a_history(ctx, H):
    """Rows of verify calls: their ids are the history's and the tokens fed before them, which begin with any thread; histories
    whose rows lie on the 16-byte grid, and ones that do not."""
    S, R, V = 20, 9, 30000
    rg = np.random.default_rng(H)
    x = normal_logits(S * R, V, 2.5, H)
    likely = np.argsort(-x, axis=1)[:, :50]
    fed = np.ascontiguousarray(likely[:, 0].reshape(S, R), np.int32)
    for stride in (H, H + 1):
        h = rg.integers(0, V, (S, stride)).astype(np.int32)
        h[:, :50] = likely[::R]
        n = rg.integers(0, stride + 1, S).astype(np.int32)
        st = independent_states(oracle.port, H, S)
        g = run_gpu(ctx, x, 0.9, 40, 1.0, st, rows_per_seq=R, rep=1.1, history=h, history_len=n, fed=fed)
        check_tokens(g, oracle.port.sample_batch(x, 0.9, 40, 1.0, st, rows_per_seq=R, rep=1.1, hist=h, hist_len=n, extra=fed))


@pytest.mark.parametrize("k", [2, 50, 100, 129, 200, 256])
@pytest.mark.parametrize("rows,V", [(1, 60001), (5, 60000), (70, 30000), (2, 262144)])
def test_candidates_of_parts_merged(ctx, rows, V, k):
    """Rows cut into parts: all candidates among the staged words and ranked (up to 128 of them, up to 220, more), more than were
    staged, and values on a grid, whose ties at the last place outrun the few; kept sets and their probabilities."""
    x = normal_logits(rows, V, 2.5, V + k)
    x[1::3] = np.round(x[1::3] * 16) / 16
    st = independent_states(oracle.port, V + k, rows)
    o = oracle.port.sample_batch(x, 3.0, k, 1.0, st, detail_cap=k)
    for hint in (0, 1):
        g = run_gpu(ctx, x, 3.0, k, 1.0, st, kept_cap=k, finish_hint=hint)
        assert (g["status"] & 32 == 0).all()
        check_tokens(g, o)
        full = (g["status"] & 8) == 0  # not by the multi-pass path
        assert np.array_equal(g["kept_idx"][full], o["detail_idx"][full])
        np.testing.assert_allclose(g["kept_prob"][full], o["detail_prob"][full], rtol=1e-5)


@pytest.mark.parametrize("rows,V", [(3, 60001), (70, 30000), (300, 5000)])
def test_narrow_nuclei_and_temperature_of_parts(ctx, rows, V):
    """Top-p rows served from the candidates, equal values at the nucleus's edge among them; temperature rows whose draw falls
    into every segment, segments of weight 0 and rows of more segments than a thread block has threads among them."""
    from helpers import gumbel_logits
    st = independent_states(oracle.port, V, rows)
    x = gumbel_logits(rows, V, 4.0, V)
    x[1::3] = np.round(x[1::3])
    check_tokens(run_gpu(ctx, x, 0.8, 0, 0.9, st), oracle.port.sample_batch(x, 0.8, 0, 0.9, st))
    y = normal_logits(rows, V, 2.0, V)
    y[1::3, : V // 2] = -np.inf
    y[2::3, V // 3:] -= 200.0
    check_tokens(run_gpu(ctx, y, 1.0, 0, 1.0, st), oracle.port.sample_batch(y, 1.0, 0, 1.0, st))
    if rows < 10:
        z = normal_logits(rows, 300000, 2.0, V)
        check_tokens(run_gpu(ctx, z, 1.0, 0, 1.0, st), oracle.port.sample_batch(z, 1.0, 0, 1.0, st))


@pytest.mark.parametrize("k", [40, 129, 200, 256])
@pytest.mark.parametrize("V", [4096, 20011, 128256])
def test_candidates_crowded_into_few_bins(ctx, V, k):
    """Many candidates that all but a few values push into one bin of values, and into few of keys: values far above the rest, of every
    size; two clusters a few bits wide; values around zero under one far above; hundreds that are equal. Whole rows, and rows whose
    parts are merged. Drawn nearly evenly, so that every place counts."""
    for rows, hint in [(300 if V < 10000 else 24, 1), (24, 0)]:
        rg = np.random.default_rng(V + k)
        x = normal_logits(rows, V, 2.5, V + k)
        T = np.full(rows, 4.0, np.float32)
        far = rg.integers(0, V, rows)
        x[np.arange(0, rows, 6), far[0::6]] = 4000.0
        x[np.arange(1, rows, 6), far[1::6]] = 1e30
        x[2::6] = np.float32(7.0) + rg.integers(0, 2 * V, x[2::6].shape).astype(np.float32) * np.float32(2.0 ** -21)
        x[np.arange(2, rows, 6), far[2::6]] = 3e38
        x[3::6] = np.where(rg.random(x[3::6].shape) < 0.5, np.float32(-2.0), np.float32(5.0)) + rg.integers(0, 64, x[3::6].shape).astype(np.float32) * np.float32(2.0 ** -20)
        x[np.arange(3, rows, 6), far[3::6]] = 100.0
        x[4::6] = np.where(rg.random(x[4::6].shape) < 400.0 / V, normal_logits(1, V, 0.01, V), np.float32(-3.0))
        x[np.arange(4, rows, 6), far[4::6]] = 50.0
        x[5::6] = np.where(rg.random(x[5::6].shape) < 600.0 / V, np.float32(1.0), x[5::6] - np.float32(20.0))
        st = independent_states(oracle.port, V + k, rows)
        g = run_gpu(ctx, x, T, k, 1.0, st, finish_hint=hint)
        done = (g["status"] & 32) == 0
        assert done.all() or (hint == 1 and done.sum() >= rows // 6)  # parts' candidates that outrun the small kernel's list ask for the other one
        o = oracle.port.sample_batch(x, T, k, 1.0, st)
        assert np.array_equal(g["tokens"][done], o["tokens"][done])
