"""The reference raster's density sat(exp(-q/2)) = sat(2^(-q log2(e)/2)) over
all q: its error against 64 bits, and its bits against the reference's
expression with CUDA's __expf."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _q():
    rng = np.random.default_rng(11)
    bits = rng.integers(0, 1 << 32, 1 << 23, dtype=np.uint64).astype(np.uint32)  # every magnitude, NaN, infinite
    special = np.float32([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 3.4e38, -3.4e38, 174.67, 174.68, 206.0, 208.0])
    return np.concatenate([bits.view(np.float32), rng.uniform(0, 200, 1 << 22).astype(np.float32),
                           np.exp(rng.uniform(-20, 5.4, 1 << 22)).astype(np.float32), special])


def test_density(gs):
    import torch
    q = _q()
    dq = torch.from_numpy(q).cuda()
    wild, tame, expf = (torch.empty_like(dq) for _ in range(3))
    gs.probe_density(dq, wild, tame, expf)
    wild, tame, expf = (t.cpu().numpy() for t in (wild, tame, expf))
    nan = np.isnan(q)
    with np.errstate(all="ignore"):
        exact = np.minimum(np.exp(-0.5 * q.astype(np.float64)), 1.0)
    tiny = 2.0 ** -126
    for got in (wild, tame):
        d, x, qq = got[~nan].astype(np.float64), exact[~nan], np.abs(q[~nan]).astype(np.float64)
        normal = x >= tiny * (1 + 1e-4)
        # the product's rounding (2^-24) and the constant's (below 2^-26) of the exponent, ex2's 2^-22
        bound = 2.0 ** -22 + 0.5 * qq * (2.0 ** -24 + 2.0 ** -26)
        assert np.all(np.abs(d[normal] - x[normal]) <= bound[normal] * x[normal])
        assert np.all((d[~normal] >= 0) & (d[~normal] <= tiny * (1 + 1e-4)))
        big = ~nan & (expf >= tiny)
        assert np.array_equal(got[big].view(np.uint32), expf[big].view(np.uint32))
        assert np.all(got[~nan & ~big] <= tiny)
    assert np.all(wild[nan] == 0) and np.all(expf[nan] == 0)
