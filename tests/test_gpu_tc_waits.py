"""Completion waits of the tensor-core exchange kernels that run out (a limit of
no polls): the kernels end, K is NaN wherever the build was not finished, and
the handle's next build with the usual limit is what it was before."""
import pytest

import helfem_gb300 as hg
from gpu_util import make_pair, random_density, to_dev, torch_cuda

pytestmark = pytest.mark.gpu
DEFAULT = 1 << 17


# two groups of output blocks per element pair, many, diagonal tiles alone; fewer
# K steps than copy stages (split form only)
@pytest.mark.parametrize("case,split", [((10, 1, 1, 6, 13), False), ((10, 1, 1, 6, 13), True),
                                        ((36, 3, 3, 3, 13), False), ((36, 3, 3, 3, 13), True),
                                        ((18, 1, 1, 4, 17), False), ((18, 1, 1, 4, 17), True),
                                        ((4, 0, 0, 3, 4), True), ((10, 1, 1, 3, 4), True)],
                         ids=lambda c: f"l{c[1]}_e{c[3]}_n{c[4]}" if isinstance(c, tuple) else "split" if c else "plain")
@pytest.mark.parametrize("mix", [True, False], ids=["dense", "same_m"])
def test_atomic_wait_runs_out(case, split, mix):
    torch = torch_cuda()
    A, O = make_pair(*case)
    nn, n = case[4], O.nbf // len(A.lval)
    P = to_dev(torch, random_density(O.nbf, 5, seed=1))
    if not mix:  # the output blocks of different m are inactive, and zero
        m = torch.as_tensor(A.mval, device="cuda").repeat_interleave(n)
        P *= m[:, None] == m[None, :]
    g = torch.arange(n, device="cuda")
    inner = (g + 1) % (nn - 1) != 0  # not on a boundary between elements
    el = (g + 1) // (nn - 1)
    tiles = (inner[:, None] & inner[None, :]) & ((el[:, None] == el[None, :]) | (nn <= 16))
    tiles = tiles.repeat(len(A.lval), len(A.lval))
    for symmetric in (False, True):
        K0, K = torch.empty_like(P), torch.zeros_like(P)
        A.exchange(P, K0, symmetric=symmetric, split=split)
        A.tc_wait_limit(0)
        A.exchange(P, K, symmetric=symmetric, split=split)
        torch.cuda.synchronize()
        A.tc_wait_limit(DEFAULT)
        assert torch.isnan(K[tiles & (K0 != 0)]).all()
        assert torch.equal(K[~torch.isnan(K)], K0[~torch.isnan(K)])
        A.exchange(P, K, symmetric=symmetric, split=split)
        torch.cuda.synchronize()
        assert torch.isfinite(K0).all() and torch.equal(K, K0)


@pytest.mark.parametrize("split", [False, True], ids=["plain", "split"])
def test_diatomic_wait_runs_out(split):
    torch = torch_cuda()
    nn, nel = 10, 3
    d = hg.Diatomic.from_grid(3, 1, 3.0, nel, [4, 2], Rmax=12.0, nnodes=nn)
    P = to_dev(torch, random_density(d.nbf, 5, seed=1))
    n = nel * (nn - 1)  # functions of an m = 0 shell, the first of the basis
    g = torch.arange(n, device="cuda")
    el = g // (nn - 1)
    tiles = (el[:, None] == el[None, :]) & (g % (nn - 1) != 0)[:, None] & (g % (nn - 1) != 0)[None, :]
    for symmetric in (False, True):
        K0, K = torch.empty_like(P), torch.zeros_like(P)
        d.exchange(P, K0, symmetric=symmetric, split=split)
        d.tc_wait_limit(0)
        d.exchange(P, K, symmetric=symmetric, split=split)
        torch.cuda.synchronize()
        d.tc_wait_limit(1 << 20)
        assert torch.isnan(K[:n, :n][tiles]).all()
        assert torch.equal(K[~torch.isnan(K)], K0[~torch.isnan(K)])
        d.exchange(P, K, symmetric=symmetric, split=split)
        torch.cuda.synchronize()
        assert torch.isfinite(K0).all() and torch.equal(K, K0)


@pytest.mark.parametrize("split", [False, True], ids=["plain", "split"])
def test_wait_that_ran_out_is_reported_once(split):
    """By the host-pointer entries and the SCF driver themselves, after a
    device-pointer entry by the status query; then the handle works as before."""
    torch = torch_cuda()
    A, O = make_pair(10, 1, 1, 6, 13)
    d = hg.Diatomic.from_grid(3, 1, 3.0, 3, [4, 2], Rmax=12.0, nnodes=10)
    for h in (A, d):
        P = random_density(h.nbf, 4, seed=2)
        K0 = h.exchange_host(P, split=split)
        h.tc_wait_limit(0)
        with pytest.raises(hg.HfgError, match="ran out"):
            h.exchange_host(P, split=split)
        Pd = to_dev(torch, P)
        K = torch.zeros_like(Pd)
        h.exchange(Pd, K, split=split)
        with pytest.raises(hg.HfgError, match="ran out"):
            h.tc_status()
        h.tc_status()
        h.tc_wait_limit(DEFAULT if h is A else 1 << 20)
        assert (h.exchange_host(P, split=split) == K0).all()
    E = A.scf(5, 5, split=split)["Etot"]
    A.tc_wait_limit(0)
    with pytest.raises(hg.HfgError, match="ran out"):
        A.scf(5, 5, split=split)
    A.tc_wait_limit(DEFAULT)
    assert A.scf(5, 5, split=split)["Etot"] == pytest.approx(E, abs=1e-9)
