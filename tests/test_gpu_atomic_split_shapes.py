"""Atomic split-precision exchange at the shapes where its compacted groups of
output blocks, its tiles and its scales can go wrong: the shortest and longest
elements, the last order the tensor-core form takes (16 nodes) and the first
it leaves to the float-pair form (17), l up to 3, densities with every block, with the m-diagonal ones, with one
block only and with none above the screen, general and symmetric modes, against
the oracle.

Bar: 1e-12 of max|K|, the split form's bar on the other bases."""
import numpy as np
import pytest

from oracle import FockOracle
from gpu_util import from_dev, make_pair, relerr, to_dev, torch_cuda

pytestmark = pytest.mark.gpu

CASES = [
    # Z, lmax, mmax, nelem, nnodes
    (4, 0, 0, 3, 3),
    (6, 1, 1, 2, 4),
    (10, 1, 0, 6, 16),
    (30, 2, 2, 3, 16),
    (18, 2, 1, 4, 9),
    (36, 3, 3, 3, 13),
    (20, 3, 0, 3, 8),
    (18, 2, 2, 2, 17),
]


def densities(A, O, seed):
    rng = np.random.default_rng(seed)
    n = O.nbf // len(A.lval)
    m = np.asarray(A.mval)
    C = rng.standard_normal((O.nbf, 5))
    full = C @ C.T
    same_m = np.kron((m[:, None] == m[None, :]).astype(float), np.ones((n, n)))
    one = np.zeros_like(full)
    one[-n:, -n:] = full[-n:, -n:]
    yield "dense", full
    yield "same m", full * same_m
    yield "one block", one
    yield "none", np.zeros_like(full)


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"Z{c[0]}_l{c[1]}m{c[2]}_e{c[3]}_n{c[4]}")
def test_split_exchange_shapes(case):
    torch = torch_cuda()
    A, O = make_pair(*case)
    F = FockOracle(O)
    for name, P in densities(A, O, case[0] + case[4]):
        ref = F.exchange(P)
        Pd = to_dev(torch, P)
        for symmetric in (False, True):
            K = torch.full_like(Pd, np.nan)
            A.exchange(Pd, K, symmetric=symmetric, split=True)
            torch.cuda.synchronize()
            got = from_dev(K)
            if name == "none":
                assert not got.any(), symmetric
            else:
                assert relerr(got, ref) < 1e-12, (name, symmetric, relerr(got, ref))
