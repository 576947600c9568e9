"""A density value that is not finite reaches the exchange as one: the output
entries that depend on it are not finite either, whatever digits or float
pairs the form computes in, and the others are what they are without it (the
split forms' bars: 1e-12 of max|K| for atoms, 1e-11 for molecules)."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import DiatomicOracle, FockOracle
from oracle import diatomic as dia
from gpu_util import from_dev, make_pair, to_dev, torch_cuda
from test_gpu_diatomic import bound_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nn", [7, 8, 15])
@pytest.mark.parametrize("bad", [np.nan, np.inf], ids=["nan", "inf"])
def test_diatomic_split_nonfinite(nn, bad):
    torch = torch_cuda()
    nelem, lm = 3, [4, 2]
    d = hg.Diatomic.from_grid(3, 1, 3.0, nelem, lm, Rmax=12.0, nnodes=nn)
    D = dia.build_diatomic(3, 1, 3.0, nn, nelem, lm, Rmax=12.0)
    P = bound_density(D, 1, seed=nn, blockdiag=False)
    ref = DiatomicOracle(D).exchange(P)
    n = nelem * (nn - 1)  # functions of an m = 0 shell
    first, last = slice(0, nn - 1), slice(2 * (nn - 1), n)
    for symmetric in (False, True):
        Pd = to_dev(torch, P)
        Pd[0, 0] = bad  # first element, first shell
        K = torch.zeros_like(Pd)
        d.exchange(Pd, K, symmetric=symmetric, split=True)
        k = from_dev(K)
        hit = ~np.isfinite(k)
        assert hit[:n, :n][first, first].all(), symmetric
        assert not hit[:n, :n][last, last].any(), symmetric
        assert np.allclose(k[~hit], ref[~hit], rtol=0, atol=1e-11 * np.abs(ref).max()), symmetric


# digit planes for every tile (13 nodes, 8 nodes), for the diagonal ones (17)
@pytest.mark.parametrize("nn", [8, 13, 17])
@pytest.mark.parametrize("bad", [np.nan, np.inf], ids=["nan", "inf"])
def test_atomic_split_nonfinite(nn, bad):
    torch = torch_cuda()
    A, O = make_pair(10, 1, 1, 6, nn)
    rng = np.random.default_rng(nn)
    C = rng.standard_normal((O.nbf, 5))
    P = C @ C.T
    ref = FockOracle(O).exchange(P)
    n = O.nbf // len(A.lval)

    def own(e):  # the functions inside element e
        return slice(e * (nn - 1), (e + 1) * (nn - 1) - 1)

    for a, b in ((2, 4), (3, 3)):
        r, c = own(a).start + 2, own(b).start + 1
        for symmetric in (False, True):
            Pd = to_dev(torch, P)
            Pd[c, r] = bad
            if symmetric:
                Pd[r, c] = bad
            K = torch.zeros_like(Pd)
            A.exchange(Pd, K, symmetric=symmetric, split=True)
            k = from_dev(K)
            hit = ~np.isfinite(k)
            # the s-s block of the tile, and of its transposed partner
            assert hit[:n, :n][own(a), own(b)].all(), (a, b, symmetric)
            if symmetric:
                assert hit[:n, :n][own(b), own(a)].all(), (a, b)
            rows, cols = (x % n for x in np.where(hit))
            near = {e * (nn - 1) + i - 1 for e in {a, b} for i in range(nn)}
            assert set(rows) <= near and set(cols) <= near, (a, b, symmetric)
            assert np.allclose(k[~hit], ref[~hit], rtol=0, atol=1e-12 * np.abs(ref).max()), (a, b, symmetric)
