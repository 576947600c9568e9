"""Exchange on bases that list an angular function more than once: their lists of
exchange entries are longer than those of any basis of distinct (l, m), longer
than a block's default shared memory holds flags for. Copies of a function are
the same function, so the blocks of K are those of the distinct basis for the
density summed over the copies.

Bars: plain and erfc 1e-10 of max|K|, split 1e-12 (those of the distinct bases)."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import FockOracle
from oracle import tabulate as tab
from gpu_util import from_dev, relerr, to_dev, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,copies", [(1, 2), (3, 5), (3, 6)], ids=lambda v: str(v))
def test_exchange_of_repeated_functions(lmax, copies):
    torch = torch_cuda()
    b = tab.get_grid(30.0, 2, 4, 2.0)
    lv, mv = hg.angular_basis(lmax, lmax)
    nn, n, nang = 4, 5, len(lv)
    assert n == 2 * (nn - 1) - 1
    O = tab.build_atom(8, nn, b, lmax, lmax)
    A = hg.Atom(8, b, np.tile(lv, copies), np.tile(mv, copies), nnodes=nn)
    rng = np.random.default_rng(copies)
    C = rng.standard_normal((A.nbf, 4))
    P = C @ C.T / copies
    Psum = P.reshape(copies, nang * n, copies, nang * n).sum(axis=(0, 2))
    ref = np.tile(FockOracle(O).exchange(Psum), (copies, copies))
    Pd = to_dev(torch, P)
    for split, tol in ((False, 1e-10), (True, 1e-12)):
        for symmetric in (False, True):
            K = torch.full_like(Pd, np.nan)
            A.exchange(Pd, K, symmetric=symmetric, split=split)
            assert relerr(from_dev(K), ref) < tol, (split, symmetric)
    A.compute_erfc(0.4)
    one = hg.Atom(8, b, lv, mv, nnodes=nn)
    one.compute_erfc(0.4)
    Kone, K = to_dev(torch, np.zeros_like(Psum)), torch.full_like(Pd, np.nan)
    one.rs_exchange(to_dev(torch, Psum), Kone)
    A.rs_exchange(Pd, K)
    assert relerr(from_dev(K), np.tile(from_dev(Kone), (copies, copies))) < 1e-10
