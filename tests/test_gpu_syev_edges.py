"""The subspace eigenproblem at the edges of its kernels' ranges: remainders of
the four-step sweeps of the inverse iteration, and sizes around those of the
kernels that take over for larger matrices; and matrices with columns that need
no reflector."""
import numpy as np
import pytest

from qxmd_b200.lib import Context, QX_NL_GSPACE, QX_PREC_FP64

from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [2, 3, 4, 5, 6, 7, 8, 33, 129, 160, 161, 255, 256, 257])
def test_edges(si8, nb):
    need_gpu()
    npw = si8.gs.nplwex
    rng = np.random.default_rng(nb)
    # orthonormal in the Gamma metric: 2 sum c c' = 1, no G = 0 part
    q = np.linalg.qr(rng.standard_normal((npw - 2, nb)))[0].T / np.sqrt(2.0)
    psi = np.concatenate([np.zeros((nb, 2)), q], axis=1)
    v = np.linalg.qr(rng.standard_normal((nb, nb)))[0]
    lam = np.sort(rng.uniform(-1, 1, nb))
    hm = (v * lam) @ v.T
    ctx = Context(si8, QX_PREC_FP64, QX_NL_GSPACE, nband=nb)
    ctx.put_psi(psi)
    ctx.put_hpsi(hm @ psi)
    ctx.hmatrix()
    ev = ctx.untryt()
    ctx.untryhc()
    x, hx = ctx.get_psi(), ctx.get_hpsi()
    ctx.close()
    # n eps |H| for the values; the vectors' residual and orthogonality likewise,
    # with the factor of the reduction's n steps
    eps = 2.3e-16
    assert np.max(np.abs(ev - lam)) < 20 * (nb + 10) * eps
    assert np.max(np.abs(2.0 * x @ x.T - np.eye(nb))) < 200 * (nb + 10) * eps
    assert np.max(np.abs(2.0 * x @ hx.T - np.diag(ev))) < 200 * (nb + 10) * eps


@pytest.mark.parametrize("kind", ["diagonal", "tridiagonal", "blocks"])
@pytest.mark.parametrize("nb", [2, 3, 4, 5, 33, 79, 80, 81, 159, 160, 161])
def test_columns_already_reduced(si8, nb, kind):
    """Columns whose part below the subdiagonal is zero already (no reflector),
    the last ones among them, at odd and even sizes: unit vectors for psi, so
    that the zeros of H_sub are exact."""
    need_gpu()
    npw = si8.gs.nplwex
    rng = np.random.default_rng(nb)
    hm = np.diag(rng.permutation(np.linspace(-1.0, 1.0, nb)) + 0.1)
    if kind == "tridiagonal":
        hm += np.diag(rng.uniform(0.1, 0.3, nb - 1), 1)
    elif kind == "blocks":   # dense rows first, then pairs, the last row alone
        m = nb // 2
        hm[:m, :m] += rng.uniform(-0.2, 0.2, (m, m))
        for i in range(m, nb - 2, 2):
            hm[i, i + 1] = 0.25
    hm = np.triu(hm) + np.triu(hm, 1).T
    psi = np.zeros((nb, npw))
    psi[np.arange(nb), 2 + np.arange(nb)] = np.sqrt(0.5)
    ctx = Context(si8, QX_PREC_FP64, QX_NL_GSPACE, nband=nb)
    ctx.put_psi(psi)
    ctx.put_hpsi(hm @ psi)
    ctx.hmatrix()
    ev = ctx.untryt()
    ctx.untryhc()
    x, hx = ctx.get_psi(), ctx.get_hpsi()
    ctx.close()
    # the bounds of test_edges
    eps = 2.3e-16
    assert np.max(np.abs(ev - np.linalg.eigvalsh(hm))) < 20 * (nb + 10) * eps
    assert np.max(np.abs(2.0 * x @ x.T - np.eye(nb))) < 200 * (nb + 10) * eps
    assert np.max(np.abs(2.0 * x @ hx.T - np.diag(ev))) < 200 * (nb + 10) * eps
