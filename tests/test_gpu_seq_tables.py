"""The one-rank CG order after the real-space projector tables were replaced:
its captured loop must not go on with the tables of its capture."""
import numpy as np
import pytest

from qxmd_b200 import cell
from qxmd_b200.lib import CgParm, Context, QX_NL_GSPACE, QX_NL_RSPACE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


def _upload(ctx, kr):
    """qx_set_kb_r, as Context does it once."""
    rc = ctx.L.qx_set_kb_r(ctx.h, kr.off.size - 1, kr.vnl.shape[1], np.ascontiguousarray(kr.off, dtype=np.int32),
                           np.ascontiguousarray(kr.mesh, dtype=np.int32),
                           np.ascontiguousarray(kr.vnl, dtype=np.float64),
                           np.ascontiguousarray(kr.clalp, dtype=np.float64), kr.rdelv)
    assert rc == 0


def _sweep(ctx, psi):
    """H psi and one sweep of the one-rank order from psi."""
    ctx.put_psi(psi)
    ctx.enonloc()
    ctx.ekinetic()
    ctx.eigen(CgParm.defaults(16, sequential=1))
    return ctx.get_psi(), ctx.get_hpsi(), ctx.get_eig()


@pytest.mark.parametrize("prec", [QX_PREC_FP64, QX_PREC_MIXED])
@pytest.mark.parametrize("how", ["upload", "build"])
def test_replaced_tables(si8, si8_psi, prec, how):
    need_gpu()
    s = si8
    b = cell.kbr_builder_tables(s.gs, s.cell, s.pp)
    shift = np.random.default_rng(3).uniform(-0.3, 0.3, s.cell.pos.shape)
    moved = cell.kb_tables_r(s.gs, cell.Cell(rba=s.cell.rba, pos=s.cell.pos + shift), s.pp)
    satm = b["satm"] + shift @ np.linalg.inv(s.cell.rba).T

    def replace(ctx):
        if how == "upload":
            _upload(ctx, moved)
        else:
            ctx.set_kb_r_builder(b)
            ctx.build_kb_r(b["ityp"], satm)

    ctx = Context(s, prec, QX_NL_RSPACE)
    before = _sweep(ctx, si8_psi)
    replace(ctx)
    got = _sweep(ctx, si8_psi)
    ctx.close()
    fresh = Context(s, prec, QX_NL_RSPACE)
    replace(fresh)
    ref = _sweep(fresh, si8_psi)
    fresh.close()
    # every sum runs in a fixed order: the same tables give the same bits
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
    assert not np.allclose(got[2], before[2], rtol=1e-4)


def test_stream_switch(monkeypatch, si8, si8_psi):
    """QX_KB_STREAM between sweeps of one context: the projectors beside the
    transforms or behind them, to rounding (H psi of the entry sums the two
    parts in another order)."""
    need_gpu()
    ctx = Context(si8, QX_PREC_FP64, QX_NL_GSPACE)
    out = []
    for mode in ("1", "0", "1"):
        monkeypatch.setenv("QX_KB_STREAM", mode)
        out.append(_sweep(ctx, si8_psi))
    ctx.close()
    for r in out[1:]:
        for a, b in zip(r[:2], out[0][:2]):
            assert np.max(np.abs(a - b)) < 1e-11
