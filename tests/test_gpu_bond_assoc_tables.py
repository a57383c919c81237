"""The bond-associated step with its per-particle weight matrices: families of
every size around a group of four bonds and one warp (no bond, 1 .. 32, and past
32, where the other kernel runs), and tables re-formed when a reset restores
bonds that broke under earlier, classic parameters; against the oracle."""
import numpy as np
import pytest

from conftest import normwise

pytestmark = pytest.mark.gpu
TOL = 1e-12  # as tests/test_gpu_bond_assoc.py: the weights' exp and pow differ in the last bits


def _ctx(pdg, x, vol, cutoff, n1=10.0, n2=10.0, s_c=0.0):
    ctx = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, s_c=s_c, n1=n1, n2=n2,
                                                weight_len=3.0))
    ctx.set_particles(x, vol)
    ctx.build_families(cutoff)
    return ctx


def _sim(po, ctx, x, vol, n1=10.0, n2=10.0):
    rp, col = ctx.families()
    return po.OracleSim(x, vol, rp, col, E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, n1=n1, n2=n2, wlen=3.0)


@pytest.mark.parametrize("nx,ny,cutoff", [(1, 1, 3.0), (2, 1, 3.0), (3, 2, 3.0), (7, 1, 3.0), (5, 5, 1.1), (8, 7, 3.03),
                                          (9, 9, 3.17), (11, 9, 3.7)])
def test_bond_assoc_family_sizes_match_oracle(pdg, po, nx, ny, cutoff):
    r = np.random.default_rng(2)
    n = nx * ny
    x = np.stack([np.arange(n) % nx, np.arange(n) // nx], axis=1) + 0.02 * r.random((n, 2))
    vol = 1.0 + 0.2 * r.random(n)
    ctx = _ctx(pdg, x, vol, cutoff)
    sim = _sim(po, ctx, x, vol)
    u = 1e-4 * r.standard_normal((n, 2))
    ctx.set_state(u, np.zeros_like(u), np.zeros_like(u))
    sim.u[:] = u
    for steps in (1, 3):
        ctx.step(steps)
        sim.step(steps)
        gu, gv, gf = ctx.state()
        if n > 1:
            assert normwise(gv, sim.v) < TOL and normwise(gf, sim.f) < TOL and normwise(gu, sim.u) < TOL
        else:
            assert not gf.any() and not gv.any()
    ctx.close()


def test_bond_assoc_tables_follow_a_reset(pdg, po):
    """Bonds break under classic parameters, then the bond-associated model is
    set (its tables hold the cut families), then a reset restores the bonds."""
    r = np.random.default_rng(4)
    x = np.stack([np.arange(72) % 9, np.arange(72) // 9], axis=1).astype(np.float64)
    vol = np.ones(72)
    ctx = _ctx(pdg, x, vol, 3.03, n1=0.0, n2=0.0, s_c=1e-3)
    u = 1e-2 * r.standard_normal(x.shape)
    ctx.set_state(u, np.zeros_like(u), np.zeros_like(u))
    ctx.step(1)
    assert ctx.counters()["bonds_broken"] > 0
    ctx.set_params(s_c=0.0, n1=10.0, n2=10.0)
    ctx.reset()
    fresh = _ctx(pdg, x, vol, 3.03)
    sim = _sim(po, fresh, x, vol)
    sim.u[:] = u
    sim.step(2)
    for c in (ctx, fresh):
        c.set_state(u, np.zeros_like(u), np.zeros_like(u))
        c.step(2)
    for a, b, o in zip(ctx.state(), fresh.state(), (sim.u, sim.v, sim.f)):
        assert np.array_equal(a, b) and normwise(a, o) < TOL
    ctx.close()
    fresh.close()
