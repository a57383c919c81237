"""The persistent batch kernel stages in each phase the indices that its own earlier
phases marked broken: with bonds breaking in every step its state equals that of the
single-plate passes (a launch each, handed over on either side of the limits on their
blocks per SM), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(61, 43), (32, 2432), (32, 2433), (300, 300), (32, 3648), (32, 3649)])
def test_persistent_kernel_with_bonds_breaking_equals_single_passes(pdg, nx, ny):
    nat = pdg.native
    p = pdg.plates.make_plate(nx, ny, seed=3, crack="centre-half")
    r = np.random.default_rng(4)
    u = 4e-4 * p.x * [0.0, 1.0] + 1e-8 * r.standard_normal(p.x.shape)
    v = 0.5 * r.standard_normal(p.x.shape)  # neighbours drift apart: losses from the first steps on
    a, b = p.context(precision=nat.PD_MIXED), p.context(precision=nat.PD_MIXED)
    for c in (a, b):
        c.set_state(u, v, np.zeros_like(u))
    bt = nat.Batch(nat.PD_MIXED)
    bt.add(b)
    bt.set_config(persistent=1)
    broken = [0]
    for steps in (3, 4, 5):
        a.step(steps)
        bt.step(steps)
        bt.synchronize()
        for x, y in zip(a.state(), b.state()):
            assert np.array_equal(x, y, equal_nan=True)
        assert np.array_equal(a.bond_mask(), b.bond_mask())
        broken.append(a.counters()["bonds_broken"])
    assert 0 < broken[1] < broken[2] < broken[3] < a.nnz
    assert b.counters()["bonds_broken"] == broken[3] and a.counters()["device_error"] == 0
    bt.remove(b)
    bt.close()
    a.close()
    b.close()
