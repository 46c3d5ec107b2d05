"""Force and clover-construction kernels at the sizes where their indexing can
go wrong: extents of 2 (both neighbours of a site are the same), site counts
below a warp and not a multiple of 32 or 128, and the dispatch of the clover
force between one parity of sigma planes and both.

Tolerance: an entry sums at most 3 planes x 16 products of up to six 3x3
matrices, about 2000 rounded operations; with random signs that is sqrt(2000)
x 1.1e-16 = 5e-15 of the force's own size, and 1e-13 leaves a factor 20."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-13
LATTICES = [(2, 2, 2, 2), (4, 2, 6, 2), (2, 6, 4, 10), (6, 10, 2, 14), (10, 4, 6, 4)]


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.fixture(scope="module", params=LATTICES, ids=lambda L: "x".join(map(str, L)))
def setup(request, oracle, bq):
    L = request.param
    g = oracle.Geom(L, (1, 1, 1, -1))
    oracle.ranset(4711)
    u = g.hot()
    kappa, csw = 0.13, 1.9192
    clov = g.clover_init(u, csw * kappa)
    lat = bq.Lattice(L, (1, 1, 1, -1))
    lat.load_gauge(u, flipped=False)
    lat.clover_init(csw * kappa)
    yield dict(g=g, u=u, clov=clov, lat=lat, kappa=kappa, csw=csw)
    lat.close()


def test_clover_blocks(setup):
    for got, want in zip(setup["lat"].get_clover(), setup["clov"]):
        assert rel(got, want) < TOL


def test_gauge_force(setup):
    g, lat = setup["g"], setup["lat"]
    p0 = g.gauss_momenta()
    want = g.dsg(p0.copy(), setup["u"], 0.05, 5.29) - p0
    lat.mom_set(p0)
    lat.dsg_dev(0.05, 5.29)
    assert rel(lat.mom_get() - p0, want) < TOL


@pytest.mark.parametrize("kappa", [0.13, 0.0])
def test_dsf_both_parities_and_one(setup, bq, kappa):
    """kappa = 0 leaves the even sigma planes only (s2 = 0)."""
    g, lat, u = setup["g"], setup["lat"], setup["u"]
    csw_kappa = setup["csw"] * setup["kappa"]
    a, b = g.gauss_spinor(0), g.gauss_spinor(0)
    p0 = g.gauss_momenta()
    want = g.dsf(p0.copy(), g.flip_bc(u.copy()), setup["clov"], 0.037, kappa, csw_kappa, a, b) - p0
    got = lat.dsf(p0.copy(), 0.037, bq.Params(kappa, csw_kappa, 0.0, 0.0), a, b) - p0
    assert rel(got, want) < TOL


@pytest.mark.parametrize("eo", [0, 1])
def test_one_parity_forces(setup, eo):
    g, lat, u = setup["g"], setup["lat"], setup["u"]
    a, b = g.gauss_spinor(eo), g.gauss_spinor(eo)
    p0 = g.gauss_momenta()
    want = g.clover_dsf(eo, p0.copy(), b, a, -0.0123, u) - p0
    assert rel(lat.clover_dsf(eo, p0.copy(), b, a, -0.0123) - p0, want) < TOL
    want = g.clover_dsd(eo, p0.copy(), setup["clov"][2], -0.0211, u) - p0
    assert rel(lat.clover_dsd(eo, p0.copy(), -0.0211) - p0, want) < TOL
