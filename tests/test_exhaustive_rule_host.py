"""The rule by which a call is answered without the index (always_exhaustive in csrc/dci_b200.cu, asked through the
library) against the sequential restatement: wherever sizes satisfy it, the answer is the exact k nearest rows."""
import numpy as np

from dciknn_cuda_b200 import _capi
from oracle import oracle


def rule(n, parts_wanted, S, T, k, outer, max_cand):
    return bool(_capi.lib().dci_b200_always_exhaustive(n, parts_wanted, T, S, k, outer, max_cand))


def test_the_rule_lies_where_it_says():
    assert rule(2000, 100, 7, 10, 10, 5000, 100)
    assert not rule(2000, 100, 7, 10, 10, 5000, 19)                       # a quota below a partition
    assert rule(2000, 100, 7, 10, 10, 4, 20) and not rule(2000, 100, 7, 10, 10, 3, 20)      # iterations: 4 windows a simple index
    assert rule(2000, 100, 7, 10, 19, 5000, 20) and not rule(2000, 100, 7, 10, 20, 5000, 20)
    assert not rule(1, 1, 1, 1, 1, 10, 10) and rule(3, 1, 1, 2, 1, 10, 10)      # more iterations than windows: 1 against 3, 6 against 4


def test_where_the_rule_holds_the_answer_is_the_exact_one():
    rng = np.random.default_rng(3)
    held = 0
    for _ in range(400):
        n, P = int(rng.integers(1, 400)), int(rng.choice([1, 2, 3, 7, 20, 100]))
        L, S, T = int(rng.integers(1, 4)), int(rng.integers(1, 7)), int(rng.choice([1, 2, 3, 7, 10, 16, 50]))
        ppb = -(-n // P)
        k = int(rng.integers(1, min(n, 40) + 1))
        max_cand = int(rng.choice([ppb, ppb + 1, k + 1, 10 * k, 100000]))
        least = -(-(S * (-(-ppb // T) + 2)) // S)
        outer = int(rng.choice([least, least + 1, 5000]))
        if not rule(n, P, S, T, k, outer, max_cand):
            continue
        held += 1
        dim = int(rng.choice([2, 5, 16]))
        data = rng.standard_normal((n, dim)).astype(np.float32)
        query = (rng.standard_normal((4, dim)) * rng.choice([1.0, 10.0])).astype(np.float32)
        proj = rng.standard_normal((L * S, dim)).astype(np.float32)
        proj /= np.linalg.norm(proj, axis=1, keepdims=True)
        o = oracle.OracleDCI(dim, L, S, P, T, proj)
        o.add(data)
        ids, _ = o.query(query, k, outer, max_cand)
        for q in range(4):
            d = ((data.astype(np.float64) - query[q]) ** 2).sum(1)
            want = np.sort(d)[:k]
            assert (ids[q] >= 0).all() and len(set(ids[q].tolist())) == k
            # by distance, so that rows equally far within fp32 rounding may stand for one another
            np.testing.assert_allclose(np.sort(d[ids[q]]), want, rtol=(dim + 4) * 2.0 ** -22)
    assert held > 100
