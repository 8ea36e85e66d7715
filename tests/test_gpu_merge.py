"""Rows of many parts, whose candidates the finishing kernels merge, around the number of entries that are ranked one
against all (220): the best k alone below it, at it and above it, out of more candidates than that."""
import numpy as np
import pytest

import oracle
from geistlib_b200 import api
from helpers import independent_states, normal_logits
from test_gpu_parity import check_tokens, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2, 219, 220, 221, 256])
@pytest.mark.parametrize("rows,V", [(1, 128256), (9, 50257), (2, 262144), (1, 524287)])
@pytest.mark.parametrize("hint", [api.FINISH_AUTO, api.FINISH_GREEDY_TOPK])
def test_k_around_what_is_ranked(ctx, rows, V, K, hint):
    x = normal_logits(rows, V, 2.0, V + K)
    x[0, ::1000] = 6.5  # a hundred and more equal values around the k-th
    st = independent_states(oracle.port, K, rows)
    g = run_gpu(ctx, x, 0.9, K, 1.0, st, kept_cap=256, finish_hint=hint)
    o = oracle.port.sample_batch(x, 0.9, K, 1.0, st, detail_cap=256)
    check_tokens(g, o)
    assert np.array_equal(g["kept_idx"], o["detail_idx"])
