"""FP64 H|psi> at the cubic grids of silicon cells whose z columns and planes
have register kernels, for full and half-empty band pairs, and H|psi> of both
precisions at every plane shape and z length of their lists: against the oracle
and against the shared-memory stage kernels."""
import dataclasses

import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_NONE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu, relerr
from test_plane_shapes import plane64_grids, plane_grids, zcols64_lengths, zcols_lengths

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


def _box(grid, nband):
    """An atom in an orthorhombic box with edges in proportion to the grid, whose
    wavefunction sphere reaches a quarter of every axis."""
    edge = 0.35 * np.array(grid, dtype=np.float64)
    gmax = 2.0 * np.pi * 0.2499 / 0.35
    c = cell.Cell(rba=np.diag(edge), pos=np.array([[0.3, 0.4, 0.2]]) * edge)
    gs = cell.strvec(c.rba, gmax**2, 1.05 * gmax**2)
    k1, k2, k3 = grid

    def index(s):
        return (np.mod(s * gs.nga, k1) + (np.mod(s * gs.ngb, k2) + np.mod(s * gs.ngc, k3) * k2) * k1).astype(np.int32)
    gs = dataclasses.replace(gs, grid=grid, ijk_pos=index(1), ijk_neg=index(-1))
    rng = np.random.default_rng(k1 * 100 + k2)
    return cell.System(cell=c, gs=gs, pp=cell.ModelPP(), nband=nband, occ=cell.occupations(nband, c.nel),
                       vloc=rng.uniform(-1.0, 1.0, gs.kfft0), kb_g=np.zeros((gs.nplwex, 4)), vclalp=np.zeros(4),
                       kb_r=cell.KBReal(off=np.array([0, 1], dtype=np.int32), mesh=np.zeros(1, dtype=np.int32),
                                        vnl=np.zeros((1, 4)), clalp=np.zeros(4), rdelv=1.0), eewald=0.0)


SHAPES = sorted([(QX_PREC_FP64, a, b, 21) for a, b in plane64_grids()] +
                [(QX_PREC_FP64, 24, 24, n) for n in zcols64_lengths()] +
                [(QX_PREC_MIXED, a, b, 21) for a, b in plane_grids()] +
                [(QX_PREC_MIXED, 24, 24, n) for n in zcols_lengths()])


@pytest.mark.parametrize("prec,k1,k2,k3", SHAPES)
def test_listed_shapes(monkeypatch, prec, k1, k2, k3):
    need_gpu()
    s = _box((k1, k2, k3), 5)
    m = [int(np.max(np.abs(g[:s.gs.nplw + 1]))) for g in (s.gs.nga, s.gs.ngb, s.gs.ngc)]
    assert m == [(k - 1) // 4 for k in s.gs.grid]
    psi = cell.random_wavefunctions(s.gs.nplwex, 5)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    ref = oracle.Ham(s, QX_NL_NONE).hpsi(psi)
    for mode in ("1", "0"):
        monkeypatch.setenv("QX_PLANE", mode)
        monkeypatch.setenv("QX_ZCOLS", mode)
        ctx = Context(s, prec, QX_NL_NONE)
        ctx.put_psi(psi)
        ctx.enonloc()
        # the tolerances of the other H|psi> tests
        assert relerr(ctx.get_hpsi(), ref) < (1e-11 if prec == QX_PREC_FP64 else 2e-5)
        ctx.close()
