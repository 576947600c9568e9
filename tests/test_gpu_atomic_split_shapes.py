"""Atomic exchange on the tensor cores, split-precision and FP64, at the
shapes where its compacted groups of output blocks, its tiles and its scales
can go wrong: the shortest and longest elements, the last order the form takes
(16 nodes) and the first it leaves to the other kernels (17), l up to 3,
densities with every block, with the m-diagonal ones, with one block only and
with none above the screen, general and symmetric modes, against the oracle.

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


# both sides of the line between the FP64 kernel and the FP64 form on the
# tensor cores, at its edges
CASES64 = [
    (6, 1, 1, 6, 13),
    (6, 1, 0, 6, 16),
    (30, 2, 2, 2, 13),
    (36, 3, 3, 2, 16),
    (36, 2, 2, 12, 10),
    (10, 1, 1, 16, 12),
    (6, 1, 0, 3, 10),
    (6, 1, 0, 3, 9),
    (6, 1, 0, 25, 10),
    (36, 2, 2, 11, 9),
    (10, 0, 0, 10, 15),
    (10, 0, 0, 11, 15),
    (4, 0, 0, 6, 14),
    (18, 1, 1, 6, 17),
]


@pytest.mark.parametrize("case", CASES64, ids=lambda c: f"Z{c[0]}_l{c[1]}m{c[2]}_e{c[3]}_n{c[4]}")
def test_fp64_exchange_shapes(case):
    """FP64 form: 1e-12 of max|K| (both sides sum in 53 bits or more; the
    tables of the two differ by their own rounding), at any scale of the
    density."""
    torch = torch_cuda()
    A, O = make_pair(*case)
    F = FockOracle(O)
    for name, P in densities(A, O, case[0] + case[4]):
        ref = F.exchange(P)
        for scale in (1.0, 2.0**600) if name == "dense" else (1.0,):
            Pd = to_dev(torch, P * scale)
            for symmetric in (False, True):
                K = torch.full_like(Pd, np.nan)
                A.exchange(Pd, K, symmetric=symmetric)
                torch.cuda.synchronize()
                got = from_dev(K) / scale
                if name == "none":
                    assert not got.any(), symmetric
                else:
                    assert relerr(got, ref) < 1e-12, (name, scale, symmetric, relerr(got, ref))


def test_fp64_exchange_nan_stays_in_its_tile():
    """A NaN of the density spoils the output of its element pair (through every
    multipole, so every output block that sees it) and of no other."""
    torch = torch_cuda()
    A, O = make_pair(10, 1, 1, 6, 13)
    _, P = next(densities(A, O, 1))
    n = O.nbf // len(A.lval)
    Pd = to_dev(torch, P)
    K0 = torch.empty_like(Pd)
    A.exchange(Pd, K0)
    for r, c in ((30, 54), (30, 30)):  # inside elements 2 and 4 (12 functions each), and 2 and 2
        Pn = Pd.clone()
        Pn[c, r] = np.nan
        K = torch.empty_like(Pd)
        A.exchange(Pn, K)
        k, k0 = from_dev(K), from_dev(K0)
        hit = np.isnan(k)
        rows, cols = np.where(hit)
        assert hit.any() and set(rows % n // 12) <= {r // 12, r // 12 - 1, r // 12 + 1}
        assert set(cols % n // 12) <= {c // 12, c // 12 - 1, c // 12 + 1}
        assert np.allclose(k[~hit], k0[~hit], rtol=0, atol=1e-12 * np.abs(k0).max())
