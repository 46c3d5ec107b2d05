"""The CG update that takes the scalar step itself (k_cg_update): lattices with
1, 4, 256 and 272 block partials, on both sides of the limit up to which FP64
takes it, for iteration limits that end a solve at every place of a batch of
queued iterations.  The iterates are those of BQCD's cg: FP64, 1e-12 after at
most 21 iterations of a well-conditioned operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("L", [(2, 2, 2, 2), (4, 4, 4, 4), (8, 8, 8, 32), (8, 8, 8, 34)],
                         ids=lambda L: "x".join(map(str, L)))
def test_truncated_cg(oracle, bq, L):
    g = oracle.Geom(L, (1, 1, 1, -1))
    oracle.ranset(5)
    uf = g.flip_bc(g.hot())
    para = bq.HmcPara(kappa=0.1, csw=0.0, rho=0.1)
    b = g.gauss_spinor(0)
    with bq.Lattice(L, (1, 1, 1, -1)) as lat:
        lat.load_gauge(uf, flipped=True)
        for n in (1, 2, 3, 4, 5, 12, 13, 21):
            xr, itr, _, _ = g.cg("w_dagger_w", np.zeros_like(b), b, uf, None, 0.1, 0.0, 0.0, 0.1, rest=1e-30,
                                 maxiter=n, log=2)
            x, it, info = lat.cg(np.zeros_like(b), b, para, rest=1e-30, maxiter=n, log=2)
            assert it == itr == n and info.converged == 0
            assert rel(x, xr) < 1e-12


@pytest.mark.parametrize("L", [(12, 12, 12, 32), (12, 12, 14, 28)], ids=lambda L: "x".join(map(str, L)))
def test_mixed_on_both_sides(oracle, bq, L):
    """216 and 221 block partials of the int16 iterations: the true residual
    that the solve reports and stops at, by the oracle's operator.  A x is
    rounded by about 2^-53 |A| |x| with |A| |x| < 10 |b|, which is 1e-6 of |r|
    at |r|/|b| = 1e-9; 1e-5 leaves a factor 10."""
    g = oracle.Geom(L, (1, 1, 1, -1))
    oracle.ranset(6)
    uf = g.flip_bc(g.hot())
    para = bq.HmcPara(kappa=0.1, csw=0.0, rho=0.1)
    b = g.gauss_spinor(0)
    with bq.Lattice(L, (1, 1, 1, -1)) as lat:
        lat.load_gauge(uf, flipped=True)
        x, info = lat.solve(np.zeros_like(b), b, para, precision=bq.PREC_HALF, tol=1e-9)
    assert info.converged
    r = b - g.op("w_dagger_w", x, uf, None, 0.1, 0.0, 0.0, 0.1)
    true = np.linalg.norm(r) / np.linalg.norm(b)
    assert true < 1e-9 * (1 + 1e-5)
    assert abs(np.sqrt(info.rtr) / np.linalg.norm(b) - true) < 1e-5 * true
