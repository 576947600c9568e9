"""Diatomic XC at the shapes where its groups of pairs, nodes and points can go
wrong: two elements and more, 3 to 17 nodes, one shell (one pair, a mostly
idle group), enough pairs for every group size, shells of m < 0 folded into
their mirrors from densities that differ between the two, against the oracle.

Bars as on the other grids: 1e-10 of max|H|, 1e-11 of |E| and N."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import diatomic as dia
from oracle.diatomic_xc import PureMGrid
from gpu_util import relerr, torch_cuda
from test_gpu_diatomic import bound_density
from test_gpu_diatomic_xc import FUNCS

pytestmark = pytest.mark.gpu

CASES = [
    # nnodes, nelem, lmax per |m|
    (3, 2, [2]),
    (15, 2, [0]),
    (8, 3, [3, 2]),
    (17, 2, [2, 2]),
    (10, 4, [5, 4, 3]),
    (15, 6, [8]),
]


@pytest.mark.parametrize("func", ["gga", "pw"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_e{c[1]}_l{'-'.join(map(str, c[2]))}")
def test_diatomic_xc_shapes(case, func):
    torch_cuda()
    nn, nelem, lm = case
    d = hg.Diatomic.from_grid(3, 1, 3.0, nelem, lm, Rmax=12.0, nnodes=nn)
    D = dia.build_diatomic(3, 1, 3.0, nn, nelem, lm, Rmax=12.0)
    g = PureMGrid(D)
    names = FUNCS[func]
    x, c = hg.parse_xc("-".join(names))
    Pa = bound_density(D, 2, seed=nn, blockdiag=True)
    Pb = 0.5 * Pa + 0.5 * bound_density(D, 1, seed=nn, blockdiag=True)
    P = Pa + Pb
    Hr, _, Er, Nr = g.eval_Fxc(names, 0.5 * P, 0.5 * P)
    H, _, E, N = d.xc_host(x, c, P)
    assert relerr(H, Hr) < 1e-10, relerr(H, Hr)
    assert abs(E - Er) < 1e-11 * abs(Er) and abs(N - Nr) < 1e-11 * Nr
    Ha_r, Hb_r, Eu_r, _ = g.eval_Fxc(names, Pa, Pb)
    Ha, Hb, Eu, _ = d.xc_host(x, c, Pa, Pb)
    assert relerr(Ha, Ha_r) < 1e-10 and relerr(Hb, Hb_r) < 1e-10
    assert abs(Eu - Eu_r) < 1e-11 * abs(Eu_r)
