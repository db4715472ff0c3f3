"""Collapse and reset over pairs, and P(0), at sizes around the unrolled loops
and on every kind of bit, against the same rules in numpy (1e-15 relative: one
rounding of each kept component); a reset divides as the rule says, also
zeros and the smallest components."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("n", [1, 2, 5, 11, 18, 22])
def test_measure_kernels(n, dtype):
    from quict_b200.simulation.engine import Engine, require_cuda
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    v[rng.random(1 << n) < 0.2] = 0
    v[0] = 1e-30 + 1e-31j
    eng = Engine(require_cuda(0))
    base = torch.from_numpy(v).to("cuda", dtype)
    host = base.cpu().numpy().astype(np.complex128)
    eps = 2.0 ** -52 if dtype == torch.complex128 else 2.0 ** -23
    idx = np.arange(1 << n)
    for bit in sorted({0, 1 % n, n // 2, n - 1}):
        one = (idx >> bit) & 1 == 1
        p0 = eng.prob0(base, n, bit)
        assert abs(p0 - np.sum(np.abs(host[~one]) ** 2)) <= 1e-13
        for outcome in (0, 1):
            t = base.clone()
            eng.collapse(t, n, bit, outcome, 1.25)
            want = np.where(one == bool(outcome), host * 1.25, 0)
            assert np.all(np.abs(t.cpu().numpy() - want) <= eps * np.abs(want))
        for p in (0.37, 0.0):
            t = base.clone()
            eng.reset(t, n, bit, p)
            low, high = host[~one], host[one]
            a = np.sqrt(p)
            want = np.zeros(1 << n, dtype=np.complex128)
            want[~one] = high if p == 0.0 else low.real / a + 1j * (low.imag / a)
            got = t.cpu().numpy()
            assert np.all(np.abs(got - want) <= eps * np.abs(want))
            if dtype == torch.complex128:
                assert np.array_equal(got, want)
