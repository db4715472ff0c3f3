"""Sampling through the sum tree at the sizes where its shape changes: fewer
amplitudes than lanes, one leaf of one to 32 rows, one to three stored levels
(full and partial ones), states with whole blocks and rows of zero
probability.  The sampled indices equal the oracle's for the same uniforms,
except draws within 1e-12 of a boundary of the distribution."""
import numpy as np
import pytest
import torch

from oracle import sv as osv


def _state(n, kind, rng):
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    if kind == "gaps":  # zero blocks, rows and single entries
        v[rng.random(1 << n) < 0.5] = 0
        for size in (1 << 5, 1 << 10):
            for b in range((1 << n) // size):
                if rng.random() < 0.4:
                    v[b * size:(b + 1) * size] = 0
        v[rng.integers(1 << n)] = 1.0
    return v / np.linalg.norm(v)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["full", "gaps"])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 9, 10, 11, 14, 15, 16, 20, 21])
def test_indices_match_the_oracle(n, kind):
    from quict_b200 import _native as N
    from quict_b200.simulation.engine import Engine, require_cuda
    rng = np.random.default_rng(100 + n)
    v = _state(n, kind, rng)
    eng = Engine(require_cuda(0))
    dev = torch.from_numpy(v).cuda()
    u = np.concatenate([rng.random(500), [0.0, 1.0 - 2.0 ** -53]])
    got = eng.sample_indices(dev, n, torch.from_numpy(u), N.QS_SAMPLE_CDF).cpu().numpy()
    want = osv.sample_cdf(v, u)
    sure = ~osv.near_ties(v, u)
    assert np.array_equal(got[sure], want[sure])
    assert np.all(np.abs(v[got]) > 0)
    us = rng.random((200, n))
    got = eng.sample_indices(dev, n, torch.from_numpy(us.ravel()), N.QS_SAMPLE_SEQ).cpu().numpy()
    want = osv.sample_sequential_fast(v, n, us)
    assert np.mean(got != want) <= 0.005  # one draw in 200 may sit on a boundary


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 5, 8])
def test_density_matrix_diagonal(n):
    from quict_b200 import _native as N
    from quict_b200.simulation.engine import Engine, require_cuda
    rng = np.random.default_rng(7 + n)
    p = rng.random(1 << n)
    p /= p.sum()
    rho = torch.from_numpy(np.diag(p).astype(np.complex128)).cuda()
    u = rng.random(400)
    got = Engine(require_cuda(0)).sample_indices(rho, n, torch.from_numpy(u), N.QS_SAMPLE_CDF, N.QS_SRC_DM).cpu().numpy()
    want = osv.sample_cdf(np.sqrt(p).astype(np.complex128), u)
    sure = ~osv.near_ties(np.sqrt(p).astype(np.complex128), u)
    assert np.array_equal(got[sure], want[sure])
