"""Real-space KB H|psi> through the plane kernels around the projectors
(k_plane_inv_r, k_plane_fwd_r) and the FP64 point sums (k_ptsum): plane shapes
with one and two warps of rows, odd pair counts and one to nine projectors per
atom, against the FP64 oracle, and against the shared-memory passes."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_RSPACE, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reps,ecut,nb,grid", [((1, 1, 1), 12.0, 5, (24, 24, 24)), ((1, 1, 1), 36.0, 3, (40, 40, 40)),
                                               ((2, 1, 1), 12.0, 18, (45, 24, 24)), ((2, 2, 1), 9.0, 33, (40, 40, 20)),
                                               ((1, 1, 1), 80.0, 2, (60, 60, 60))])
@pytest.mark.parametrize("lmx", [1, 4, 9])
def test_rspace_plane(monkeypatch, reps, ecut, nb, grid, lmx):
    need_gpu()
    s = cell.build_system(cell.diamond_si(reps, seed=4), ecut, 4 * ecut, nb, with_ewald=False)
    assert tuple(s.gs.grid) == grid
    # lmx projectors: the model's four with seeded values in the other columns
    kr = s.kb_r
    v = np.random.default_rng(5).standard_normal((kr.vnl.shape[0], 9)) * 0.05
    v[:, :4] = kr.vnl
    s.kb_r = cell.KBReal(off=kr.off, mesh=kr.mesh, vnl=np.ascontiguousarray(v[:, :lmx]),
                         clalp=np.linspace(0.3, 0.1, 9)[:lmx].copy(), rdelv=kr.rdelv)
    psi = cell.random_wavefunctions(s.gs.nplwex, nb)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    ref = oracle.Ham(s, QX_NL_RSPACE).hpsi(psi)
    got = []
    for env in ("1", "0"):
        monkeypatch.setenv("QX_PLANE", env)
        ctx = Context(s, QX_PREC_MIXED, QX_NL_RSPACE)
        ctx.put_psi(psi)
        ctx.enonloc()
        got.append(ctx.get_hpsi())
        ctx.close()
    # FP32 rounding of the transforms, as the other H|psi> tests of the mixed path
    assert relerr(got[0], ref) < 2e-5 and relerr(got[1], ref) < 2e-5
