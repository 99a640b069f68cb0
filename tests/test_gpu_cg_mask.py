"""The projection of a batched CG sweep on the bands below: the mask on every
contraction that may apply it (tensor cores with K split and whole, CUDA cores
split and whole, FP64), and the active-band list beside the preconditioner."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import CgParm, Context, QX_NL_GSPACE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,env", [(QX_PREC_FP64, {}), (QX_PREC_MIXED, {}), (QX_PREC_MIXED, {"QX_TC_MIN_FLOPS": "0"})])
@pytest.mark.parametrize("ecut,nb", [(2.0, 1), (2.0, 7), (3.0, 33), (12.0, 5), (12.0, 66)])
def test_mask_routes(monkeypatch, prec, env, ecut, nb):
    need_gpu()
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=3), ecut, 4 * ecut, nb, with_ewald=False)
    psi = np.linalg.qr(cell.random_wavefunctions(s.gs.nplwex, nb).T)[0].T.copy()
    h = oracle.Ham(s, QX_NL_GSPACE)
    hc = h.hpsi(psi)
    _, ekib = h.ekinetic(psi)
    x_ref, _, eig_ref, _, nri_ref = h.eigen(psi, hc, ekib, noband=nb)
    ctx = Context(s, prec, QX_NL_GSPACE)
    x, _, eig = ctx.eigen_host(psi, hc, ekib, CgParm.defaults(nb))
    ctx.close()
    # rounding of the two precisions through one step (another order of the
    # bands moves x by 0.1 to 1)
    tol_e, tol_x = (1e-10, 1e-8) if prec == QX_PREC_FP64 else (1e-4, 1e-3)
    assert relerr(eig, eig_ref) < tol_e
    assert relerr(x, x_ref) < tol_x
