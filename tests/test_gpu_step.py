"""The CG update that takes the scalar step itself (k_cg_update): lattices with
1, 4, 256 and 272 block partials, on both sides of the limit up to which it is
taken, for iteration limits that end a solve at every place of a batch of
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
