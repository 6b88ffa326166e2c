"""The bounds by which queries leave work out (csrc/distance_bounds.cuh) against 64-bit distances: never above the nearest
row of a group, whatever the mantissas that the tensor cores cut off, and not needlessly far below.  One, three and all
CTAs, so that a CTA works through many tiles; odd sizes; rows staged by ordinary loads, one and two tiles of queries."""
import numpy as np
import pytest
import torch

from tests import cases

pytestmark = pytest.mark.gpu

LOW = {"ones": 0x1FFF, "zeros": 0x0000, "alternating": 0x1555, "half": 0x1000, "below_half": 0x0FFF}     # the 13 bits cut off


def _with_low_bits(x, kind):
    if kind not in LOW:
        return x
    u = x.view(np.uint32)
    return ((u & np.uint32(0xFFFFE000)) | np.uint32(LOW[kind])).view(np.float32)


def _rows(rng, n, nq, dim, kind):
    if kind == "offset":           # nearly equal rows far from the origin
        z = np.float32(100.0) + np.float32(0.05) * rng.standard_normal((n + nq, dim)).astype(np.float32)
    elif kind == "positive":       # errors of one sign in every product
        z = rng.random((n + nq, dim), dtype=np.float32) + np.float32(0.5)
    else:
        z = cases.mixture(rng, n + nq, dim, centres=30)
    z = _with_low_bits(np.ascontiguousarray(z), kind)
    return z[:n].copy(), z[n:].copy()


def _check(n, dim, nq, kind, group_rows, max_ctas, shift=0):
    from dciknn_cuda_b200 import DCI
    rng = np.random.default_rng(n + dim + nq)
    data, query = _rows(rng, n, nq, dim, kind)
    store = torch.empty(n * dim + 4, device="cuda")
    d = store[shift:shift + n * dim].view(n, dim)
    d.copy_(torch.from_numpy(data))
    g = DCI(dim, 1, 1, 4, 10, seed=1)
    g.add(d)
    g.set_max_ctas(max_ctas)
    q = torch.from_numpy(query).cuda()
    lb = g.distance_bounds(q, group_rows)
    x64, q64 = d.double(), q.double()
    x2, q2 = (x64 * x64).sum(1), (q64 * q64).sum(1)
    d2 = q2[None, :] + x2[:, None] - 2.0 * (x64 @ q64.T)          # [n, nq]; off by about 1e-15 of the norms
    groups = -(-n // group_rows)
    pad = torch.full((groups * group_rows - n, nq), float("inf"), dtype=torch.float64, device="cuda")
    least = torch.cat([d2, pad]).view(groups, group_rows, nq).amin(1)
    norms = x2.max() + q2[None, :]
    assert lb.shape == least.shape and not torch.isnan(lb).any()
    assert (lb <= least + 1e-13 * norms).all(), float((lb - least).max())
    if group_rows % 32 == 0:
        # both operands cut off by up to 2^-10 of their norm, less the 0.32 * 2^-10 of the scale: (0.68 * 2^-10)^2 / r and
        # r = 0.2 * 2^-10 of both norms, beside the charge for the accumulation, twice each
        slack = 2.0 * ((0.68 * 0.68 / 0.2 + 0.2) * 2.0 ** -10 + dim * (2.0 ** -22 + 2.0 ** -23) + 2.0 ** -20)
        assert (lb >= least - slack * norms).all(), float(((least - lb) / norms).max())
    g.free()


@pytest.mark.parametrize("max_ctas", [0, 1, 3])
@pytest.mark.parametrize("n,dim,nq,group_rows", [
    (2500, 96, 300, 32), (2049, 8, 129, 65),                      # one tile of queries at a time
    (1537, 33, 260, 64), (1025, 130, 128, 100),                   # ordinary loads
    (1800, 512, 385, 32), (1281, 960, 700, 600)])                 # two tiles at a time, an odd number of them
def test_bounds_hold(n, dim, nq, group_rows, max_ctas):
    _check(n, dim, nq, "mixture", group_rows, max_ctas)


@pytest.mark.parametrize("kind", list(LOW) + ["offset", "positive"])
@pytest.mark.parametrize("n,dim,nq,shift", [(1300, 128, 200, 0), (1300, 128, 100, 1), (900, 4096, 100, 0), (900, 4096, 200, 0),
                                            (600, 4095, 100, 0), (1000, 4, 50, 0), (1000, 1, 50, 0)])
def test_bounds_hold_for_every_mantissa(n, dim, nq, shift, kind):
    _check(n, dim, nq, kind, 32, 2, shift)
