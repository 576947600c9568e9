"""Plain diatomic exchange on either side of the lines between its kernels (one
output block per item, FP64 in-element kernels, in-element digit planes), with
densities that mix m and that do not, general and symmetric modes, at a scale
outside the float range, against the oracle.

Bar: 1e-12 of max|K| (53-bit sums or more)."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import DiatomicOracle
from oracle import diatomic as dia
from gpu_util import from_dev, relerr, to_dev, torch_cuda
from test_gpu_diatomic import bound_density

pytestmark = pytest.mark.gpu

CASES = [
    # nnodes, nelem, lmax per |m|: items, then the other side
    (3, 5, [7]), (3, 5, [6]),
    (4, 5, [9]), (4, 5, [8]),
    (5, 7, [11]), (5, 7, [10]),
    (5, 2, [0]), (6, 2, [0]),
    # digit planes, then the FP64 in-element kernels
    (16, 2, [0]), (15, 2, [0]),
    (8, 2, [6]), (7, 2, [6]),
    (5, 2, [7]), (4, 2, [7]),
    (3, 2, [5, 5]), (3, 2, [4, 4]),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_e{c[1]}_l{'-'.join(map(str, c[2]))}")
def test_plain_exchange_lines(case):
    torch = torch_cuda()
    nn, nelem, lm = case
    d = hg.Diatomic.from_grid(3, 1, 3.0, nelem, lm, Rmax=12.0, nnodes=nn)
    D = dia.build_diatomic(3, 1, 3.0, nn, nelem, lm, Rmax=12.0)
    F = DiatomicOracle(D)
    for blockdiag in (False, True):
        P = bound_density(D, 1, seed=nn, blockdiag=blockdiag)
        ref = F.exchange(P)
        for scale in (1.0, 2.0**600):
            Pd = to_dev(torch, P * scale)
            for symmetric in (False, True):
                K = torch.full_like(Pd, np.nan)
                d.exchange(Pd, K, symmetric=symmetric)
                torch.cuda.synchronize()
                err = relerr(from_dev(K) / scale, ref)
                assert err < 1e-12, (blockdiag, scale, symmetric, err)
