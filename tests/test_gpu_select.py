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
