"""GPU parity of the atomic XC kernels where their split can go wrong: grids
with an odd, a tiny (aliasing) or a large number of azimuthal or polar points
(several polar chunks per CTA), f shells, the shortest elements, densities
that mix m (azimuthal points differ) or do not (one azimuthal point stands for
all), and a density that is not symmetric.

Bar: the XC matrices within 1e-10 of max|oracle|, energies and electron counts
within 1e-10 relative, as for the default grids. For a density that is not
symmetric the gradient takes the derivative of the row function; the oracle
takes that of the column function, so it gets the transposed density."""
import numpy as np
import pytest

import helfem_gb300 as hg
from oracle import tabulate as tab
from oracle import xc as oxc
from gpu_util import random_density, relerr, torch_cuda

pytestmark = pytest.mark.gpu
TOL = 1e-10

CASES = [
    # lmax, mmax, nelem, nnodes, ldft, mdft, method, polarized, kind of density
    (1, 1, 2, 3, 7, 5, "gga_x_pbe-gga_c_pbe", True, "mixed"),
    (1, 1, 2, 3, 7, 1, "gga_x_pbe-gga_c_pbe", False, "mixed"),
    (2, 2, 2, 4, 9, 3, "gga_x_pbe-gga_c_pbe", False, "blocks"),
    (1, 1, 2, 5, 90, 2, "gga_x_pbe-gga_c_pbe", True, "mixed"),
    (1, 1, 2, 5, 4, 200, "lda_x-lda_c_vwn", True, "mixed"),
    (3, 3, 2, 4, 0, 0, "gga_x_pbe-gga_c_pbe", True, "blocks"),
    (3, 1, 2, 4, 0, 0, "lda_x-lda_c_pw", False, "mixed"),
    (2, 1, 3, 6, 0, 0, "gga_x_pbe-gga_c_pbe", True, "nonsymmetric"),
    (2, 2, 2, 17, 0, 0, "lda_x-gga_c_pbe", False, "blocks"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"l{c[0]}m{c[1]}_n{c[3]}_g{c[4]}x{c[5]}_{'u' if c[7] else 'r'}_{c[8]}")
def test_xc_grid_shapes(case):
    torch_cuda()
    lmax, mmax, nelem, nn, ldft, mdft, method, pol, kind = case
    b = tab.get_grid(30.0, nelem, 4, 2.0)
    lv, mv = hg.angular_basis(lmax, mmax)
    A = hg.Atom(8, b, lv, mv, nnodes=nn)
    A.dft_grid(ldft, mdft)
    O = tab.build_atom(8, nn, b, lmax, mmax)
    G = oxc.AtomGrid(O, ldft, mdft)
    names = oxc.parse_method(method)
    x, c = hg.parse_xc(method)
    nr = O.nbf // len(lv)

    def density(nocc, seed):
        P = random_density(O.nbf, nocc, seed=seed, S=O.S)
        ang = np.arange(O.nbf) // nr
        if kind == "blocks":
            P *= np.asarray(mv)[ang][:, None] == np.asarray(mv)[ang][None, :]
        if kind == "nonsymmetric":
            N = np.random.default_rng(seed).standard_normal(P.shape)
            P = P + 0.05 * np.abs(P).max() * (N - N.T)
        return P

    if pol:
        Pa = density(4, 3)
        Pb = 0.7 * Pa + 0.05 * density(4, 4)
        Ha, Hb, E, N = A.xc_host(x, c, Pa, Pb)
        Ra, Rb, Er, Nr = G.eval_Fxc(names, Pa.T, Pb.T)
        assert relerr(Hb, Rb) < TOL
    else:
        P = 2.0 * density(4, 3)
        Ha, _, E, N = A.xc_host(x, c, P)
        Ra, _, Er, Nr = G.eval_Fxc(names, 0.5 * P.T, 0.5 * P.T)
    assert relerr(Ha, Ra) < TOL
    assert abs(E - Er) < TOL * abs(Er)
    assert abs(N - Nr) < TOL * abs(Nr)
