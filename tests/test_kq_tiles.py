"""Dense gates on 5 to 10 qubits as tiled products: every width, with one
group, fewer groups than a tile has columns, one tile and many, targets on the
lowest, highest and mixed bits in any order, and controls below, between and
above them, against the FP64 product (1e-12 / 1e-5, as every gate)."""
import numpy as np
import pytest
import torch

from quict_b200.simulation.lowering import Op


def _want(v, n, mat, tbits, cbits):
    out = v.copy()
    idx = np.arange(1 << n)
    on = np.ones(1 << n, dtype=bool)
    for c in cbits:
        on &= ((idx >> c) & 1) == 1
    zero = on.copy()
    for t in tbits:
        zero &= ((idx >> t) & 1) == 0
    base = idx[zero]
    k = len(tbits)
    spread = np.array([sum(((r >> (k - 1 - j)) & 1) << b for j, b in enumerate(tbits)) for r in range(1 << k)])
    cols = base[None, :] + spread[:, None]
    out[cols] = mat @ v[cols]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("k", [5, 6, 7, 8, 9, 10])
def test_tiled_product(k, precision):
    from quict_b200.simulation.engine import Engine, require_cuda
    from quict_b200.workloads import haar_unitary
    rng = np.random.default_rng(k)
    eng = Engine(require_cuda(0))
    mat = haar_unitary(rng, 1 << k)
    tol = 1e-12 if precision == "double" else 1e-5
    for n, controls in ((k, 0), (k + 1, 0), (k + 2, 1), (k + 5, 2), (17 if k < 9 else 16, 0), (17, 1)):
        free = n - k
        layouts = [list(range(k)), list(range(free, n)), [int(b) for b in rng.permutation(n)[:k]]]
        for tbits in layouts:
            rest = [b for b in range(n) if b not in tbits]
            cbits = tuple(int(b) for b in rng.choice(rest, controls, replace=False)) if controls else ()
            v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
            v /= np.linalg.norm(v)
            dev = torch.from_numpy(v).to("cuda", torch.complex128 if precision == "double" else torch.complex64)
            eng.apply_single(dev, n, Op("mat", tuple(tbits), cbits, mat))
            got = dev.cpu().numpy()
            assert np.abs(got - _want(v, n, mat, tbits, cbits)).max() <= tol, (n, tbits, cbits)


@pytest.mark.gpu
def test_wide_tiles_fill_the_gpu():
    """Enough groups for the wide tiles (one CTA per SM and more)."""
    from quict_b200.simulation.engine import Engine, require_cuda
    from quict_b200.workloads import haar_unitary
    rng = np.random.default_rng(3)
    eng = Engine(require_cuda(0))
    for k, n in ((5, 21), (6, 20), (7, 20), (8, 20)):
        mat = haar_unitary(rng, 1 << k)
        tbits = [int(b) for b in rng.permutation(n)[:k]]
        v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        v /= np.linalg.norm(v)
        dev = torch.from_numpy(v).cuda()
        eng.apply_single(dev, n, Op("mat", tuple(tbits), (), mat))
        assert np.abs(dev.cpu().numpy() - _want(v, n, mat, tbits, ())).max() <= 1e-12
