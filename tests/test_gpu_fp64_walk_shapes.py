"""The FP64 passes' bond walk equals the oracle bit for bit at every chunk width
modulo its groups (lines and strips: 0 to ~20 bonds), with and without bond
breaking and the penalty, and on either side of 60,000 particles, where the
passes change how they hand over to one another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(pdg, po, p, s_c, k_hg, steps):
    ctx = p.context(s_c=s_c, k_hg=k_hg)
    rp, col = po.build_families(p.x, p.cutoff, p.cracks)
    m = p.material
    sim = po.OracleSim(p.x, p.vol, rp, col, E=m.E, nu=m.nu, rho=m.rho, dt=p.dt, s_c=s_c, k_hg=k_hg,
                       damage_fail=p.damage_fail, bc=p.group_of, group_kind=p.group_kind, group_val=p.group_val)
    r = np.random.default_rng(1)
    u = 4e-4 * p.x + 1e-8 * r.standard_normal(p.x.shape)
    u[r.random(p.n) < 0.01] += 2e-6  # bonds that break
    f = 1e6 * r.standard_normal(p.x.shape)
    ctx.set_state(u, np.zeros_like(u), f)
    sim.u[:], sim.f[:] = u, f
    ctx.step(steps)
    sim.step(steps)
    assert np.array_equal(ctx.bond_mask(), sim.mask)
    assert np.array_equal(ctx.damage(), sim.damage)
    for a, b in zip(ctx.state(), (sim.u, sim.v, sim.f)):
        assert np.array_equal(a, b)
    ctx.close()


@pytest.mark.parametrize("s_c", [0.0, 5e-4])
@pytest.mark.parametrize("penalty", [False, True])
@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (3, 1), (4, 1), (9, 1), (2, 2), (3, 2), (7, 2), (33, 2), (5, 3), (40, 3),
                                   (17, 4), (33, 5), (65, 33)])
def test_every_walk_width_matches_oracle(pdg, po, shape, penalty, s_c):
    p = pdg.plates.make_plate(shape[0], shape[1], seed=11, jitter=0.01)
    _compare(pdg, po, p, s_c, p.k_hg if penalty else 0.0, 3)


@pytest.mark.parametrize("s_c", [0.0, 5e-4])
@pytest.mark.parametrize("shape", [(245, 244), (245, 245)])
def test_hand_over_by_size_matches_oracle(pdg, po, shape, s_c):
    p = pdg.plates.make_plate(shape[0], shape[1], seed=12, crack="centre-half")
    _compare(pdg, po, p, s_c, p.k_hg, 4)


@pytest.mark.parametrize("penalty", [False, True])
@pytest.mark.parametrize("shape", [(125001, 2), (62501, 4), (501, 500)])
def test_tests_ahead_of_the_sums_match_oracle(pdg, po, shape, penalty):
    """From 250,000 particles on, bonds are tested before a particle's sums: narrow and wide chunks."""
    p = pdg.plates.make_plate(shape[0], shape[1], seed=13)
    _compare(pdg, po, p, 5e-4, p.k_hg if penalty else 0.0, 2)


@pytest.mark.parametrize("penalty", [False, True])
@pytest.mark.parametrize("part", [0.05, 0.4, 1.0])
def test_warps_with_few_intact_bonds_match_oracle(pdg, po, part, penalty):
    """501 x 500 particles (the last warp is partial), of which some to all lose most of their bonds."""
    p = pdg.plates.make_plate(501, 500, seed=14)
    k_hg = p.k_hg if penalty else 0.0
    ctx = p.context(s_c=5e-4, k_hg=k_hg)
    rp, col = po.build_families(p.x, p.cutoff, p.cracks)
    m = p.material
    sim = po.OracleSim(p.x, p.vol, rp, col, E=m.E, nu=m.nu, rho=m.rho, dt=p.dt, s_c=5e-4, k_hg=k_hg,
                       damage_fail=p.damage_fail, bc=p.group_of, group_kind=p.group_kind, group_val=p.group_val)
    r = np.random.default_rng(2)
    u = 1e-9 * r.standard_normal(p.x.shape)
    hit = np.arange(p.n) >= (1.0 - part) * p.n  # a contiguous part, the last warp in it
    u[hit] += 4e-6 * r.standard_normal((int(hit.sum()), 2))
    z = np.zeros_like(u)
    ctx.set_state(u, z, z)
    sim.u[:] = u
    ctx.step(2)
    sim.step(2)
    assert (sim.mask == 0).sum() > 0.2 * part * sim.mask.size
    assert np.array_equal(ctx.bond_mask(), sim.mask) and np.array_equal(ctx.damage(), sim.damage)
    for a, b in zip(ctx.state(), (sim.u, sim.v, sim.f)):
        assert np.array_equal(a, b, equal_nan=True)
    ctx.close()
