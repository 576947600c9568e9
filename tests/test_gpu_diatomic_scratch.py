"""Diatomic exchange with little scratch (one unit at a time, the FP64 in-element
kernels for lack of room) against the same handle's build with all it wants, and
the plain form's kernels, which stay what the handle's first plain call took.

Bars: 1e-12 of max|K| between the two plain forms; the same kernels in one and in
many passes make the same operations, bit for bit."""
import pytest

import helfem_gb300 as hg
from gpu_util import random_density, to_dev, torch_cuda

pytestmark = pytest.mark.gpu


def build(d, P, split):
    import torch
    K = torch.full_like(P, float("nan"))
    d.exchange(P, K, split=split)
    torch.cuda.synchronize()
    return K


@pytest.mark.parametrize("first", ["plain", "split"])
def test_little_scratch(first):
    torch = torch_cuda()
    args = (3, 1, 3.0, 4, [6, 5, 4])  # 21 shells, 441 output blocks
    full, tight = (hg.Diatomic.from_grid(*args, Rmax=12.0, nnodes=9) for _ in range(2))
    P = to_dev(torch, random_density(full.nbf, 5, seed=3))
    K0, K0s = build(full, P, False), build(full, P, True)
    tight.scratch_limit(1 << 20)
    big = K0.abs().max()
    if first == "plain":
        K = build(tight, P, False)
        assert (K - K0).abs().max() < 1e-12 * big
        tight.scratch_limit(0)
    Ks = build(tight, P, True)
    assert torch.equal(Ks, K0s)
    if first == "plain":  # the digit planes are there now, the form stays
        assert torch.equal(build(tight, P, False), K)
        assert not torch.equal(K, K0)
    else:
        assert torch.equal(build(tight, P, False), K0)
