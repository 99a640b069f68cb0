"""The FP64 full-grid transforms with lines of 36 to 64 points over two lanes,
and mixed with other lengths, against numpy and the shared-memory passes."""
import numpy as np
import pytest

from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_PREC_FP64

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ecutdens,n", [(47.5, 24), (122.5, 40), (152.5, 42), (200.0, 48), (235.0, 54), (295.0, 60)])
def test_lengths(monkeypatch, ecutdens, n):
    need_gpu()
    s = cell.build_system(cell.diamond_si((1, 1, 1), seed=1), ecutdens / 4, ecutdens, 4, with_ewald=False)
    assert tuple(s.gs.grid) == (n, n, n)
    _check(monkeypatch, s)


@pytest.mark.parametrize("index", [3, 6, 11, 20])
def test_mixed(monkeypatch, index):
    need_gpu()
    _check(monkeypatch, cell.batch_cell(index))


def _check(monkeypatch, s):
    k1, k2, k3 = s.gs.grid
    x = np.random.default_rng(5).standard_normal(s.gs.kfft0)
    ref = np.fft.fftn(x.reshape(k3, k2, k1)).ravel() / s.gs.kfft0
    out = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("QX_FULL_LINES", mode)
        ctx = Context(s, QX_PREC_FP64, QX_NL_GSPACE, nband=4)
        fx, fy = ctx.rfft3_host(1, x, np.zeros_like(x))
        bx, by = ctx.rfft3_host(2, fx, fy)
        ctx.close()
        # the tolerance of the other full-grid transforms
        assert relerr(fx + 1j * fy, ref) < 1e-13
        assert relerr(bx, x) < 1e-13
        out[mode] = fx + 1j * fy
    assert relerr(out["1"], out["0"]) < 1e-13
