"""Particle steps with the order renewed only at times: counts on both sides of the one from which particles
are ordered, over enough steps for the order to be renewed, against particles carried in small groups that
never are, bit for bit; uploads begin anew."""
import numpy as np
import pytest

from dns_gkm_lpt_b200 import ic
from dns_gkm_lpt_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,graphs", [(49_999, True), (50_000, True), (60_001, False)])
def test_order_of_particles_does_not_show(count, graphs):
    n, steps = 16, 19
    rng = np.random.default_rng(count)
    P = ic.Params(n=n, gam=1.4, den0=1.0, Mt=0.3, Re=30.0, mu0=0.9, p0=86100.0, t0=0.01)
    vel = rng.normal(0.0, 60.0, (3, n, n, n))
    W0 = ic.embed_ghost(np.stack([np.ones_like(vel[0]), *vel, P.p0 / 0.4 + 0.5 * (vel**2).sum(0)]))
    pos = rng.uniform(0.0, 2.0 * np.pi, (count, 3))
    U = rng.normal(size=(count, 3))
    with Solver(P, cfl=0.5, max_particles=count, use_graphs=graphs) as s:
        s.upload_state(W0)
        s.particles_upload(pos, U)
        s.step(3)
        s.evolve_particles()
        s.upload_state(W0)
        s.particles_upload(pos, U)
        s.step(steps)
        got = s.particles_download()
    some = rng.choice(count, 700, replace=False)
    with Solver(P, cfl=0.5, max_particles=700) as s:
        s.upload_state(W0)
        s.particles_upload(pos[some], U[some])
        s.step(steps)
        want = s.particles_download()
    for a, b in zip(got, want):
        assert np.isfinite(a).all()
        assert np.array_equal(a[some], b)
