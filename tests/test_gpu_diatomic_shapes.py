"""Diatomic exchange at the shapes where its tiles and groups can go wrong:
the shortest and longest elements (partly filled row tiles, K steps and
warps), more than 8 and more than 16 shells of one m (several groups of output
rows per k), m up to 3 with few shells each, densities that mix m (every
group active) and that do not, general and symmetric modes, against the
oracle.

Bars: the FP64 form 1e-10 of max|K| (the plain form's bar), the split form
1e-11 (its bar on the other diatomic bases)."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import DiatomicOracle
from oracle import diatomic as dia
from gpu_util import from_dev, relerr, to_dev, torch_cuda
from test_gpu_diatomic import bound_density

pytestmark = pytest.mark.gpu

CASES = [
    # nnodes, nelem, lmax per |m|
    (3, 2, [3, 2]),
    (4, 3, [9]),
    (5, 2, [17, 3]),
    (8, 2, [3, 3, 3, 3]),
    (16, 2, [2, 2]),
    (17, 2, [3]),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_e{c[1]}_l{'-'.join(map(str, c[2]))}")
def test_diatomic_exchange_shapes(case):
    torch = torch_cuda()
    nn, nelem, lm = case
    d = hg.Diatomic.from_grid(3, 1, 3.0, nelem, lm, Rmax=12.0, nnodes=nn)
    D = dia.build_diatomic(3, 1, 3.0, nn, nelem, lm, Rmax=12.0)
    F = DiatomicOracle(D)
    for blockdiag in (False, True):
        P = bound_density(D, 1, seed=nn, blockdiag=blockdiag)
        ref = F.exchange(P)
        Pd = to_dev(torch, P)
        for symmetric in (False, True):
            for split, tol in ((False, 1e-10), (True, 1e-11)):
                K = torch.full_like(Pd, np.nan)
                d.exchange(Pd, K, symmetric=symmetric, split=split)
                torch.cuda.synchronize()
                err = relerr(from_dev(K), ref)
                assert err < tol, (blockdiag, symmetric, split, err)


@pytest.mark.parametrize("nn", [7, 8, 15])
def test_diatomic_fp64_scales(nn):
    """FP64 form on either side of the line between its in-element kernels, at
    a scale far outside the float range (1e-12 of max|K|: 53-bit sums), and a
    NaN of one element's density that leaves the other elements' tiles alone."""
    torch = torch_cuda()
    nelem, lm = 3, [4, 2]
    d = hg.Diatomic.from_grid(3, 1, 3.0, nelem, lm, Rmax=12.0, nnodes=nn)
    D = dia.build_diatomic(3, 1, 3.0, nn, nelem, lm, Rmax=12.0)
    P = bound_density(D, 1, seed=nn, blockdiag=False)
    ref = DiatomicOracle(D).exchange(P)
    for scale in (1.0, 2.0**600):
        Pd = to_dev(torch, P * scale)
        for symmetric in (False, True):
            K = torch.full_like(Pd, np.nan)
            d.exchange(Pd, K, symmetric=symmetric)
            torch.cuda.synchronize()
            assert relerr(from_dev(K) / scale, ref) < 1e-12, (scale, symmetric)
    Pd = to_dev(torch, P)
    Pd[0, 0] = np.nan  # first element, first shell
    K = torch.empty_like(Pd)
    d.exchange(Pd, K)
    k = from_dev(K)
    hit = np.isnan(k)
    n = nelem * (nn - 1)  # functions of an m = 0 shell
    assert hit.any() and not hit[:n, :n][2 * (nn - 1):, 2 * (nn - 1):].any()
    assert np.allclose(k[~hit], ref[~hit], rtol=0, atol=1e-10 * np.abs(ref).max())


def test_plain_exchange_under_capture():
    """A handle's first plain exchange may be captured: what it makes on its
    first call is made outside the capture, and the replay repeats the eager
    result bit for bit (atomic form with its side stream too)."""
    torch = torch_cuda()
    lv, mv = hg.angular_basis(1, 1)
    for make in (lambda: hg.Diatomic.from_grid(3, 1, 3.0, 3, [3, 2], Rmax=12.0, nnodes=10),
                 lambda: hg.Atom(10, hg.get_grid(30.0, 6, 4, 2.0), lv, mv, nnodes=15)):
        d = make()
        rng = np.random.default_rng(3)
        C = rng.standard_normal((d.nbf, 4))
        P = to_dev(torch, C @ C.T)
        K = torch.zeros_like(P)
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            d.exchange(P, K, stream=st, symmetric=True)
        g.replay()
        torch.cuda.synchronize()
        K2 = torch.zeros_like(P)
        d.exchange(P, K2, symmetric=True)
        torch.cuda.synchronize()
        assert bool((K2 != 0).any()) and torch.equal(K, K2)
