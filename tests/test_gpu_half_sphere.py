"""The plane and z kernels compiled for a sphere of at most half the grid, and
their general forms, which a density cutoff below four times the
wavefunction's needs: H|psi> and the density against the FP64 oracle on both
sides of that line, with spheres smaller than the compiled bound."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_NL_RSPACE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu

# (grid, density cutoff, wavefunction cutoffs at, inside and beyond a quarter of it)
CASES = [(24, 48.0, 12.0), (24, 48.0, 7.0), (24, 48.0, 26.0), (24, 48.0, 44.0), (27, 66.0, 16.5), (27, 66.0, 40.0),
         (54, 255.0, 63.0), (54, 255.0, 30.0), (54, 255.0, 110.0), (96, 832.0, 207.0), (96, 832.0, 90.0),
         (96, 832.0, 300.0)]


@pytest.mark.parametrize("n,ecutdens,ecut", CASES)
@pytest.mark.parametrize("nl", [QX_NL_GSPACE, QX_NL_RSPACE])
def test_sphere_ratio(n, ecutdens, ecut, nl):
    need_gpu()
    nb = 3 if n > 27 else 5
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=6), ecut, ecutdens, nb, with_ewald=False)
    assert tuple(s.gs.grid) == (n, n, n)
    psi = cell.random_wavefunctions(s.gs.nplwex, nb)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    h = oracle.Ham(s, nl)
    ref, rho = h.hpsi(psi), h.softchg(psi, s.occ)
    # rounding of the transforms at each precision, as the other H|psi> tests
    for prec, tol in ((QX_PREC_MIXED, 2e-5), (QX_PREC_FP64, 1e-11)):
        ctx = Context(s, prec, nl)
        ctx.put_psi(psi)
        ctx.enonloc()
        assert relerr(ctx.get_hpsi(), ref) < tol
        assert relerr(ctx.softchg_host(psi), rho) < tol
        ctx.close()
