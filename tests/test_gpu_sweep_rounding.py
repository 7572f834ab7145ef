"""Rounding of one pair in the boundary SDPD sweep.  Two particles at rest on an
axis, P = rho = m = 1, no noise: f = 2 F(r) x with F = fnorm (1 - r)^3, where
r = sqrt(fl(x^2)) correctly rounded is off by 1.5 u (u the unit roundoff), so
1 - r by 1.5 u r / (1 - r) + u, its cube by three times that and three
products, and the constant, the factor x and the sum by one each:
|df| <= (4.5 r / (1 - r) + 9) u |f|."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


def test_pair_near_the_cutoff(cuda_device):
    from gpucell_gb300.host import ParticleSystem
    rng = np.random.default_rng(4)
    m, gap = 16, 2.5
    centre = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * gap
    k = len(centre)
    axis = rng.integers(0, 3, k)
    a, b = centre.copy(), centre.copy()
    a[np.arange(k), axis] += rng.integers(0.45 * 2 ** 18, 0.495 * 2 ** 18, k) / 2.0 ** 18
    b[np.arange(k), axis] -= rng.integers(0.45 * 2 ** 18, 0.495 * 2 ** 18, k) / 2.0 ** 18
    x = np.concatenate([a, b])   # multiples of 2^-18 below 64: differences are exact
    assert np.array_equal(x.astype(np.float32), x)
    n = 2 * k
    L = m * gap
    cfg = gen.Config(name="pairs", bbox=np.array([0, L] * 3, np.float32), pmask=7, n_b1=0, n_b2=0, n_fluid=n,
                     coor=x.astype(np.float32), velhalf=np.zeros((n, 3), np.float32), den_init=1.0,
                     phys=gen.Physics(ext_force=0.0))
    ps = ParticleSystem(cfg, noise=False)
    ps.set_state(vel=np.zeros((n, 3)), rho=np.ones(n), press=np.ones(n))
    ps.sdpd_force()
    f = ps.fetch()["force"].astype(np.float64)
    d = (a - b)[np.arange(k), axis]
    want = 2 * 210 / np.pi * (1 - d) ** 3 * d
    err = np.abs(f[np.arange(k), axis] / want - 1)
    assert np.array_equal(f[:k], -f[k:])
    assert (err <= (4.5 * d / (1 - d) + 9) * 2.0 ** -24).all(), (err / ((4.5 * d / (1 - d) + 9) * 2.0 ** -24)).max()
