"""Pass A's update of particles that lost bonds, from a few of a warp's
particles to all of them (each form of the update): the state equals that of a
context restored from a checkpoint taken after the losses, whose K^-1 is formed
afresh from the mask, and for FP64 the oracle's, bit for bit, with the counters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(p, part):
    r = np.random.default_rng(8)
    u = 1e-9 * r.standard_normal(p.x.shape)
    hit = r.random(p.n) < part
    u[hit] += 3e-6 * r.standard_normal((int(hit.sum()), 2))  # their bonds stretch past s_c, one by one
    return u, np.zeros_like(u), 1e5 * r.standard_normal(u.shape)


@pytest.mark.parametrize("part", [0.002, 0.01, 0.03, 0.08, 0.3, 1.0])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("shape", [(64, 48), (101, 37)])
def test_losses_of_part_of_a_warp_to_all_of_it(pdg, po, shape, mixed, part):
    nat = pdg.native
    p = pdg.plates.make_plate(shape[0], shape[1], seed=6)
    prec = nat.PD_MIXED if mixed else nat.PD_FP64
    state = _state(p, part)
    a, b = p.context(precision=prec), p.context(precision=prec)
    a.set_state(*state)
    a.step(1)
    c = a.counters()
    assert c["bonds_broken"] == int((a.bond_mask() == 0).sum()) > 0
    b.restore(a.checkpoint())
    for ctx in (a, b):
        ctx.step(1)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y, equal_nan=True)
    assert np.array_equal(a.bond_mask(), b.bond_mask()) and np.array_equal(a.damage(), b.damage())
    if not mixed:
        rp, col = po.build_families(p.x, p.cutoff, p.cracks)
        m = p.material
        sim = po.OracleSim(p.x, p.vol, rp, col, E=m.E, nu=m.nu, rho=m.rho, dt=p.dt, s_c=m.s_c, k_hg=p.k_hg,
                           damage_fail=p.damage_fail, bc=p.group_of, group_kind=p.group_kind, group_val=p.group_val)
        sim.u[:], sim.v[:], sim.f[:] = state
        sim.step(2)
        assert np.array_equal(a.bond_mask(), sim.mask) and np.array_equal(a.damage(), sim.damage)
        for x, y in zip(a.state(), (sim.u, sim.v, sim.f)):
            assert np.array_equal(x, y, equal_nan=True)
    a.close()
    b.close()
