"""The rule by which a call is answered without the index (always_exhaustive in csrc/dci_b200.cu), restated and checked
against the sequential restatement: wherever sizes satisfy it, the answer is the exact k nearest rows."""
import numpy as np

from oracle import oracle


def rule(n, parts_wanted, S, T, k, outer, max_cand):
    ppb = -(-n // parts_wanted)
    num_parts = -(-n // ppb)
    wcap = S * (-(-ppb // T) + 2)
    if max_cand < ppb or max_cand <= k or outer * S < wcap:
        return False
    return all(m * T >= -(-m // T) + 2 for m in (ppb, n - (num_parts - 1) * ppb))


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
