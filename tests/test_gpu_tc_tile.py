"""The default tile width of the tensor-core contractions: the rule itself on
the CPU, and H|psi> on both sides of it against both widths forced."""
import ctypes

import numpy as np
import pytest

from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_PREC_MIXED, lib

from gpu_util import need_gpu, relerr


@pytest.mark.parametrize("rows,nb,width", [
    (9316, 128, 80), (9316, 160, 80),          # one wave either way
    (9316, 161, 128), (9316, 256, 128),        # two waves of 80, one of 128
    (9473, 160, 80), (10252, 160, 80), (13134, 160, 80),   # two of either
    (13134, 128, 128), (10252, 256, 128),      # two to one, three to two
    (13572, 288, 80), (11494, 192, 80),        # three of either, two of either
    (13572, 350, 128), (48490, 1100, 128), (2048, 1100, 128), (256, 160, 80)])
def test_rule(rows, nb, width):
    f = lib()._ZN2qx15tc_tile_defaultEli   # qx::tc_tile_default(long, int)
    f.argtypes, f.restype = [ctypes.c_long, ctypes.c_int], ctypes.c_int
    assert f((rows + 127) // 128, nb) == width


@pytest.mark.gpu
@pytest.mark.parametrize("ecut,nb", [(16.0, 161), (17.0, 160), (20.0, 128), (17.0, 256)])
def test_widths_agree(monkeypatch, ecut, nb):
    need_gpu()
    s = cell.build_system(cell.diamond_si((2, 2, 2), seed=2), ecut, 4 * ecut, nb, with_ewald=False)
    psi = cell.random_wavefunctions(s.gs.nplwex, nb)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    out = []
    for tile in (None, "80", "128"):
        if tile:
            monkeypatch.setenv("QX_TC_TILE", tile)
        else:
            monkeypatch.delenv("QX_TC_TILE", raising=False)
        ctx = Context(s, QX_PREC_MIXED, QX_NL_GSPACE)
        ctx.put_psi(psi)
        ctx.enonloc()
        out.append(ctx.get_hpsi())
        ctx.close()
    # the same products in other sums: the tolerance of the mixed path's H|psi> tests
    assert relerr(out[0], out[1]) < 2e-5 and relerr(out[0], out[2]) < 2e-5
