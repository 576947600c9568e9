"""The engine's admission estimate of a DFT solve against that of the same solve
without a functional: what the XC build keeps on the device, per element, radial
point and pair of angular functions three densities and two potentials of each
spin, and the radial functions with their derivatives."""
import pytest

import helfem_gb300 as hg
from helfem_gb300 import workloads as wl
from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,nel", [(1, 8), (3, 12)])
def test_dft_footprint(lmax, nel):
    torch_cuda()
    lv, mv = wl.angular(lmax, lmax)
    nq, nn, pairs = 75, 15, len(lv) * (len(lv) + 1) // 2
    grid = 8 * nel * nq * (10 * pairs + 2 * nn)
    eng = hg.Engine(n_workers=1, hbm_budget_gb=40.0)
    fp = []
    for method in ("hf", "lda_x-lda_c_pw"):
        job = eng.submit(10, wl.grid(40.0, nel), lv, mv, 5, 5, method=method, symmetry=2,
                         l_occ=wl.l_occupations(5, 5, lmax))
        fp.append(eng.wait(job)["footprint_bytes"])
    eng.close()
    assert grid <= fp[1] - fp[0] <= 1.3 * grid
