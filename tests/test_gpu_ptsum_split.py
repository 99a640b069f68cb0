"""The projector point sums with an atom's points split over a cluster:
uneven atoms (none, one, a round of the warps and its neighbours, many) at
the point counts of every split, against the FP64 oracle."""
import dataclasses

import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_RSPACE, QX_PREC_FP64, QX_PREC_MIXED

from gpu_util import need_gpu, relerr

pytestmark = pytest.mark.gpu


# points by atom: on average below 256 (no split), 256 (two CTAs), 512 (four), 1024 and more (eight)
@pytest.mark.parametrize("counts", [(0, 1, 127, 128, 129, 255, 256, 1000), (0, 1, 127, 128, 129, 255, 256, 1152),
                                    (0, 1, 127, 128, 129, 600, 1111, 2000), (0, 1, 129, 130, 1023, 1024, 1025, 4860),
                                    (0, 3, 5000, 1025, 4097, 9000, 7, 8192)])
@pytest.mark.parametrize("lmx,nb", [(1, 2), (4, 17), (9, 32)])
@pytest.mark.parametrize("prec,tol", [(QX_PREC_FP64, 1e-11), (QX_PREC_MIXED, 2e-5)])
def test_split(si8, counts, lmx, nb, prec, tol):
    need_gpu()
    rng = np.random.default_rng(sum(counts) + lmx)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    kr = cell.KBReal(off=off, mesh=rng.integers(0, si8.gs.kfft0, off[-1]).astype(np.int32),
                     vnl=rng.standard_normal((off[-1], lmx)) * 0.05, clalp=np.linspace(0.3, 0.1, 9)[:lmx].copy(),
                     rdelv=si8.kb_r.rdelv)
    s = dataclasses.replace(si8, kb_r=kr)
    psi = cell.random_wavefunctions(s.gs.nplwex, nb)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    ctx = Context(s, prec, QX_NL_RSPACE, nband=nb)
    ctx.put_psi(psi)
    ctx.enonloc()
    got = ctx.get_hpsi()
    ctx.close()
    # the tolerances of the other H|psi> tests
    assert relerr(got, oracle.Ham(s, QX_NL_RSPACE).hpsi(psi)) < tol
