"""Bonds at the critical stretch: the FP64 form's mask, damage, forces and
state equal the oracle's bit for bit where the FP32 stretch test cannot decide
(stretches within rounding of s_c), where it decides either way, and under a
rigid translation that is large against the bonds' elongations; with one, some
and all of a warp's particles (16 per warp) losing bonds in a step; and either
side of 250,000 particles, from where on the tests run ahead of the sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 3), (33, 7), (64, 40)])
@pytest.mark.parametrize("rel", [-1e-3, -2e-6, -1e-7, -1e-12, 0.0, 1e-15, 1e-9, 5e-7, 3e-6, 1e-2])
@pytest.mark.parametrize("shift", [0.0, 3e-2])
def test_bonds_at_the_critical_stretch_match_oracle(pdg, po, shape, rel, shift):
    s_c = 5e-4
    p = pdg.plates.make_plate(shape[0], shape[1], seed=7, jitter=0.0 if rel == 0.0 else 0.01)
    r = np.random.default_rng(3)
    half = p.x[:, 0] > np.median(p.x[:, 0])  # (one half is compressed: bonds that a bound on |d| alone cannot clear)
    s = np.where(half, s_c * (1.0 + rel), -2.0 * s_c)[:, None]
    u = s * p.x + shift
    u[r.random(p.n) < 0.02] += 2e-6  # a few particles out of line
    ctx = p.context(s_c=s_c)
    rp, col = po.build_families(p.x, p.cutoff, p.cracks)
    m = p.material
    sim = po.OracleSim(p.x, p.vol, rp, col, E=m.E, nu=m.nu, rho=m.rho, dt=p.dt, s_c=s_c, k_hg=p.k_hg,
                       damage_fail=p.damage_fail, bc=p.group_of, group_kind=p.group_kind, group_val=p.group_val)
    ctx.set_state(u, np.zeros_like(u), np.zeros_like(u))
    sim.u[:] = u
    ctx.step(2)
    sim.step(2)
    gu, gv, gf = ctx.state()
    assert np.array_equal(ctx.bond_mask(), sim.mask)
    assert np.array_equal(ctx.damage(), sim.damage)
    assert np.array_equal(gu, sim.u) and np.array_equal(gv, sim.v) and np.array_equal(gf, sim.f)
    assert ctx.counters()["bonds_broken"] == int((sim.mask == 0).sum())
    ctx.close()


@pytest.mark.parametrize("shape", [(499, 501), (500, 500)])
@pytest.mark.parametrize("rel", [-1e-12, 0.0, 5e-7, 1e-2])
def test_tests_ahead_of_the_sums_match_oracle(pdg, po, shape, rel):
    test_bonds_at_the_critical_stretch_match_oracle(pdg, po, shape, rel, 3e-2)
