"""The FP64 passes with four threads per site (dslash_split.cu) against the
CPU oracle: a single CTA with idle lanes (8 sites), a remainder of 8 sites in
the last CTA, and lattices on each side of every bound of split_sites (14208,
18944 and 28416 sites of a parity; beyond, the one-thread passes in one wave and
in two), with every term of the operators.
Relative norm-wise agreement to 1e-13: some 1,400 FP64 operations per site and
pass, rounding to 2^-53 each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICES = [(2, 2, 2, 2), (6, 6, 6, 6), (12, 12, 12, 16), (12, 12, 10, 20), (12, 12, 12, 22), (12, 12, 16, 24),
            (14, 14, 14, 22), (16, 16, 16, 18), (20, 16, 16, 16)]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module", params=LATTICES, ids=lambda L: "x".join(map(str, L)))
def setup(request, oracle, bq):
    L = request.param
    g = oracle.Geom(L, (1, 1, 1, -1))
    oracle.ranset(11)
    u = g.hot()
    uf = g.flip_bc(u.copy())
    csw, kappa = 1.9192, 0.12
    clov = g.clover_init(u, csw * kappa)
    with bq.Lattice(L, (1, 1, 1, -1)) as lat:
        lat.load_gauge(uf, flipped=True)
        lat.load_clover(*clov)
        yield dict(g=g, uf=uf, clov=clov, lat=lat, kappa=kappa, csw=csw)


@pytest.mark.parametrize("name", ["w_mult", "w_mult_dag", "w_dagger_w"])
@pytest.mark.parametrize("csw,h", [(1.9192, 0.0), (0.0, 0.0), (0.0, 0.2)], ids=["clover", "wilson", "wilson_h"])
def test_operators(setup, bq, name, csw, h):
    g, rho = setup["g"], 0.15
    para = bq.HmcPara(kappa=setup["kappa"], csw=csw, rho=rho, h=h)
    psi = g.gauss_spinor(0)
    ref = g.op(name, psi, setup["uf"], setup["clov"] if csw else None, setup["kappa"], para.csw_kappa, h, rho)
    assert rel(getattr(setup["lat"], name)(psi, para), ref) < 1e-13


@pytest.mark.parametrize("csw", [1.9192, 0.0], ids=["clover", "wilson"])
def test_cg(setup, bq, csw):
    """The sums over the CTAs and the CG scalars: iterations and solution of BQCD's cg."""
    g = setup["g"]
    para = bq.HmcPara(kappa=setup["kappa"], csw=csw, rho=0.1)
    b = g.gauss_spinor(0)
    rest = np.float32(1e-16 * 12 * g.volh)
    xr, itr, _, rc = g.cg("w_dagger_w", np.zeros_like(b), b, setup["uf"], setup["clov"] if csw else None,
                          setup["kappa"], para.csw_kappa, 0.0, 0.1, rest=rest, maxiter=2000, log=0)
    assert rc == 0
    x, it, info = setup["lat"].cg(np.zeros_like(b), b, para, rest=rest, maxiter=2000, log=0)
    assert abs(it - itr) <= 1 and info.converged
    assert rel(x, xr) < 1e-8    # both stop at |r|^2 of the same size, 1e-16 |b|^2
