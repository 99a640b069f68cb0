"""Gram-Schmidt (Cholesky and inverse of the overlap) at the edges of the
blocked kernel: one 8 x 8 tile, 16-column blocks and their remainders, the
largest size one CTA takes and the first beyond it, against the oracle, and
the pivot test."""
import numpy as np
import pytest

import oracle
from qxmd_b200 import cell
from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_PREC_FP64, QxError

from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 80, 81, 159, 160, 161, 192, 193, 207, 208, 209])
def test_schmidt_sizes(si8, n):
    need_gpu()
    x = cell.random_wavefunctions(si8.gs.nplwex, n)
    ref, _, rc = oracle.schmidt(x.copy())
    assert rc == 0
    ctx = Context(si8, QX_PREC_FP64, QX_NL_GSPACE, nband=n)
    got = ctx.schmidt_host(x)
    ctx.close()
    # both are FP64 solves of the same system: n eps times the condition of the overlap
    w = np.full(si8.gs.nplwex, 2.0)
    w[0] = 1.0
    cond = np.linalg.cond((x * w) @ x.T)
    assert np.max(np.abs(got - ref)) <= 8 * n * 2.3e-16 * cond * np.max(np.abs(ref))


@pytest.mark.parametrize("n,row", [(5, 3), (40, 0), (40, 17), (160, 159), (208, 100)])
def test_schmidt_dependent_band(si8, n, row):
    """A zero band stops the factorisation at its row."""
    need_gpu()
    x = cell.random_wavefunctions(si8.gs.nplwex, n)
    x[row] = 0.0
    ctx = Context(si8, QX_PREC_FP64, QX_NL_GSPACE, nband=n)
    with pytest.raises(QxError, match="at band %d" % row):
        ctx.schmidt_host(x)
    ctx.close()
