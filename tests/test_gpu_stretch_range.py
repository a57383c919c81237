"""Critical stretches at the ends of FP32's range, where the FP32 stretch test's error
bound does not hold and the FP64 test decides: the mask, damage and state equal the
oracle's bit for bit with every bond near its limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s_c,dx", [(1e-41, 1e7), (3e-42, 1e8), (1e-15, 1.0), (1e-16, 1.0), (900.0, 1e-18), (1100.0, 1e-18),
                                    (1e5, 1e-19)])
@pytest.mark.parametrize("rel", [-3e-5, -1e-5, -3e-6, 3e-6, 1e-5, 3e-5])
def test_stretches_at_the_ends_of_fp32(pdg, po, s_c, dx, rel):
    p = pdg.plates.make_plate(33, 12, dx=dx, seed=7, v_load=0.0)
    u = s_c * (1.0 + rel * np.random.default_rng(3).random(p.n))[:, None] * p.x
    ctx = p.context(s_c=s_c)
    rp, col = po.build_families(p.x, p.cutoff, p.cracks)
    assert np.array_equal(rp, ctx.families()[0])
    m = p.material
    sim = po.OracleSim(p.x, p.vol, rp, col, E=m.E, nu=m.nu, rho=m.rho, dt=p.dt, s_c=s_c, k_hg=p.k_hg,
                       damage_fail=p.damage_fail, bc=p.group_of, group_kind=p.group_kind, group_val=p.group_val)
    ctx.set_state(u, np.zeros_like(u), np.zeros_like(u))
    sim.u[:] = u
    ctx.step(1)
    sim.step(1)
    assert np.array_equal(ctx.bond_mask(), sim.mask) and 0 < int((sim.mask == 0).sum()) < rp[-1]
    assert np.array_equal(ctx.damage(), sim.damage)
    for a, b in zip(ctx.state(), (sim.u, sim.v, sim.f)):
        assert np.array_equal(a, b, equal_nan=True)
    ctx.close()
