"""FP32 CUDA-core contractions with K split in clusters: <psi|hpsi> (H_sub) of
band counts at the edges of the tiles and of sphere sizes around the split's
threshold and its cluster counts, against the same sums in FP64."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ecut", [4.0, 6.0, 8.0, 12.0, 30.0])
@pytest.mark.parametrize("nb", [1, 2, 16, 31, 32, 33, 47, 65, 80, 81, 96])
def test_hmatrix_split(ecut, nb):
    _check(ecut, nb)


@pytest.mark.parametrize("ecut,nb", [(15.0, 385), (15.5, 384), (15.5, 385), (15.5, 450), (20.0, 1088), (20.0, 1089)])
def test_many_tiles(monkeypatch, ecut, nb):
    """36 to 324 output tiles on both sides of the sizes that split K (K of at
    least 1024, fewer than 296 tiles)."""
    monkeypatch.setenv("QX_TC_MIN_FLOPS", "1e18")
    _check(ecut, nb)


@pytest.mark.parametrize("nb", [16, 80, 81, 99, 128, 129, 161])
def test_row_tiles(monkeypatch, nb):
    """K P of H|psi> (2946 rows) with 32-, 48- and 64-row tiles, against the
    FP64 oracle."""
    need_gpu()
    monkeypatch.setenv("QX_TC_MIN_FLOPS", "1e18")
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=1), 30.0, 120.0, nb, with_ewald=False)
    assert s.gs.nplwex == 2946
    psi = cell.random_wavefunctions(s.gs.nplwex, nb)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    ctx = Context(s, QX_PREC_MIXED, QX_NL_GSPACE)
    ctx.put_psi(psi)
    ctx.enonloc()
    got = ctx.get_hpsi()
    ctx.close()
    # FP32 rounding of the transforms, as the other H|psi> tests of the mixed path
    assert relerr(got, oracle.Ham(s, QX_NL_GSPACE).hpsi(psi)) < 2e-5


def _check(ecut, nb):
    need_gpu()
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=1), ecut, 4 * ecut, nb, with_ewald=False)
    rng = np.random.default_rng(nb)
    x, y = (rng.standard_normal((nb, s.gs.nplwex)).astype(np.float32).astype(np.float64) for _ in range(2))
    x[:, 1] = y[:, 1] = 0.0
    ctx = Context(s, QX_PREC_MIXED, QX_NL_GSPACE)
    for _ in range(3):   # the counters of a launch start from what the last one left
        ctx.put_psi(x)
        ctx.put_hpsi(y)
        got = ctx.hmatrix()
    ctx.close()
    w = np.full(s.gs.nplwex, 2.0)
    w[0] = 1.0
    ref = (x * w) @ y.T
    ref = np.triu(ref) + np.triu(ref, 1).T
    # K + 2 roundings of FP32 sums of |x||y|
    bound = (s.gs.nplwex + 2) * 6e-8 * ((np.abs(x) * w) @ np.abs(y).T)
    bound = np.triu(bound) + np.triu(bound, 1).T
    assert np.all(np.abs(got - ref) <= bound)
