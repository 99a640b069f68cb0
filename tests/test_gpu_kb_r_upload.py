"""Real-space projector tables uploaded one after another into one context
(buffers that stay and grow): more and fewer points and projectors, atoms
without points, several points of an atom at one grid point, points in any
order and points before the first atom's, against the FP64 oracle and, bit for
bit, against a context that gets the tables first."""
import dataclasses

import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QxError, QX_NL_RSPACE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


def _tables(s):
    kr = s.kb_r
    rng = np.random.default_rng(2)
    nat, npts = s.cell.natom, int(kr.off[-1])

    def table(off, mesh, vnl):
        return cell.KBReal(off=np.asarray(off, dtype=np.int32), mesh=np.asarray(mesh, dtype=np.int32),
                           vnl=np.ascontiguousarray(vnl), clalp=np.linspace(0.3, 0.1, 9)[:vnl.shape[1]].copy(),
                           rdelv=kr.rdelv)
    wide = rng.standard_normal((npts, 9)) * 0.05
    yield table(kr.off, kr.mesh, kr.vnl)
    yield table(kr.off, kr.mesh, wide)                                  # nine projectors
    half = np.concatenate([np.arange(kr.off[a], (kr.off[a] + kr.off[a + 1]) // 2) for a in range(nat)])
    cut = np.concatenate([[0], np.cumsum([(kr.off[a] + kr.off[a + 1]) // 2 - kr.off[a] for a in range(nat)])])
    yield table(cut, kr.mesh[half], wide[half, :1])                     # fewer points, one projector
    yield table(np.concatenate([[0, 0], kr.off[2:]]), kr.mesh, kr.vnl)  # an atom without points
    rep = np.concatenate([np.tile(np.arange(kr.off[a], kr.off[a + 1]), 2) for a in range(nat)])
    yield table(2 * kr.off, kr.mesh[rep], wide[rep, :4])                # every point twice
    mix = np.concatenate([rng.permutation(np.arange(kr.off[a], kr.off[a + 1])) for a in range(nat)])
    yield table(kr.off, kr.mesh[mix], kr.vnl[mix])
    yield table(np.concatenate([[5], kr.off[1:]]), kr.mesh, kr.vnl)     # five points of no atom
    yield table(np.zeros(nat + 1), np.zeros(0), np.zeros((0, 4)))       # none at all


@pytest.mark.parametrize("prec,tol", [(QX_PREC_FP64, 1e-11), (QX_PREC_MIXED, 2e-5)])
def test_uploads(si8, si8_psi, prec, tol):
    need_gpu()

    def hpsi(ctx, kr):
        vnl = kr.vnl if kr.vnl.size else np.zeros((1, 4))
        mesh = kr.mesh if kr.mesh.size else np.zeros(1, dtype=np.int32)
        rc = ctx.L.qx_set_kb_r(ctx.h, si8.cell.natom, vnl.shape[1], kr.off, mesh, np.ascontiguousarray(vnl), kr.clalp,
                               kr.rdelv)
        assert rc == 0
        ctx.put_psi(si8_psi)
        ctx.enonloc()
        return ctx.get_hpsi()

    one = Context(si8, prec, QX_NL_RSPACE)
    for kr in _tables(si8):
        got = hpsi(one, kr)
        fresh = Context(si8, prec, QX_NL_RSPACE)
        assert np.array_equal(got, hpsi(fresh, kr))
        fresh.close()
        if kr.mesh.size:
            ref = oracle.Ham(dataclasses.replace(si8, kb_r=kr), QX_NL_RSPACE).hpsi(si8_psi)
            assert relerr(got, ref) < tol   # the tolerances of the other H|psi> tests
    bad = np.concatenate([[-1], si8.kb_r.off[1:]]).astype(np.int32)
    assert one.L.qx_set_kb_r(one.h, si8.cell.natom, 4, bad, np.ascontiguousarray(si8.kb_r.mesh, dtype=np.int32),
                             np.ascontiguousarray(si8.kb_r.vnl), si8.kb_r.clalp, si8.kb_r.rdelv) != 0
    one.close()


def test_forces_need_the_gradients_of_their_tables(si8, si8_psi):
    """Tables built without gradients after others with them: no forces from
    the gradients of the tables before; the builder alone changes nothing."""
    need_gpu()
    b = cell.kbr_builder_tables(si8.gs, si8.cell, si8.pp)
    plain = {k: v for k, v in b.items() if k != "dtabnl"}
    ctx = Context(si8, QX_PREC_FP64, QX_NL_RSPACE)
    ctx.put_psi(si8_psi)
    ctx.set_kb_r_builder(b)
    ctx.build_kb_r(b["ityp"], b["satm"])
    f = ctx.forces_nl_r()
    ctx.set_kb_r_builder(plain)
    assert np.array_equal(ctx.forces_nl_r(), f)
    ctx.build_kb_r(b["ityp"], b["satm"] + 0.01)
    with pytest.raises(QxError):
        ctx.forces_nl_r()
    ctx.set_kb_r_builder(b)
    ctx.build_kb_r(b["ityp"], b["satm"])
    assert np.array_equal(ctx.forces_nl_r(), f)
    ctx.close()
