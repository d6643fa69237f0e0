"""Particle transfers keep the upload order whatever order the device holds the particles in: exact round
trips, and a step and the property table from permuted uploads, bit for bit."""
import numpy as np
import pytest

from dns_gkm_lpt_b200 import ic
from dns_gkm_lpt_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 5003])
def test_transfers_keep_the_upload_order(count):
    n = 16
    rng = np.random.default_rng(count)
    P = ic.Params(n=n, gam=1.4, den0=1.0, Mt=0.3, Re=30.0, mu0=0.9, p0=86100.0, t0=0.01)
    vel = rng.normal(0.0, 60.0, (3, n, n, n))
    rho = np.ones((n, n, n))
    W0 = ic.embed_ghost(np.stack([rho, *vel, P.p0 / 0.4 + 0.5 * (vel**2).sum(0)]))
    pos = rng.uniform(0.0, 2.0 * np.pi, (count, 3))
    U = rng.normal(size=(count, 3))
    perm = rng.permutation(count)
    results = []
    for order in (np.arange(count), perm):
        with Solver(P, cfl=0.5, max_particles=count + 3) as s:
            s.upload_state(W0)
            s.particles_upload(pos[order], U[order])
            back = s.particles_download()
            assert np.array_equal(back[0], pos[order]) and np.array_equal(back[1], U[order])
            s.step(3)
            results.append((*s.particles_download(), s.particle_props()))
    for a, b in zip(*results):
        assert np.isfinite(a).all()
        assert np.array_equal(a[perm], b)
