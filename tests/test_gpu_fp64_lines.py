"""FP64 H|psi> at every grid whose z columns and planes have register kernels,
for full and half-empty band pairs: against the oracle and against the
shared-memory stage kernels."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_NONE, QX_PREC_FP64

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ecutdens", [(20, 32.5), (21, 40.0), (24, 47.5), (25, 55.0), (27, 65.0), (30, 75.0),
                                        (32, 85.0), (40, 122.5), (42, 152.5), (48, 200.0), (54, 235.0), (60, 295.0)])
def test_lines(monkeypatch, n, ecutdens):
    need_gpu()
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=6), ecutdens / 4, ecutdens, 5, with_ewald=False)
    assert tuple(s.gs.grid) == (n, n, n)
    psi = cell.random_wavefunctions(s.gs.nplwex, 5)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    h = oracle.Ham(s, QX_NL_NONE)
    ref, rho = h.hpsi(psi), h.softchg(psi, s.occ)
    out = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("QX_PLANE", mode)
        monkeypatch.setenv("QX_ZCOLS", mode)
        ctx = Context(s, QX_PREC_FP64, QX_NL_NONE)
        ctx.put_psi(psi)
        ctx.enonloc()
        out[mode] = ctx.get_hpsi()
        # the FP64 tolerance of the other H|psi> tests
        assert relerr(out[mode], ref) < 1e-11
        assert relerr(ctx.softchg_host(psi), rho) < 1e-11
        ctx.close()
    # log2(n^3) roundings each way on values of the same size
    assert relerr(out["1"], out["0"]) < 2 * 3 * np.log2(n) * 2.3e-16 * 10
