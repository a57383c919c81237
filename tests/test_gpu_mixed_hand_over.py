"""The mixed passes hand over to one another in two ways, by the number of their
blocks per SM: on either side of the two limits the state after many steps equals
that of the persistent batch kernel (grid barriers instead), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(32, 2432), (32, 2433), (300, 300), (32, 3648), (32, 3649)])  # 304 .. 457 tiles
def test_hand_over_equals_grid_barriers(pdg, nx, ny):
    nat = pdg.native
    p = pdg.plates.make_plate(nx, ny, seed=3, crack="centre-half")
    p.material.s_c = 2e-4
    r = np.random.default_rng(4)
    u = 1e-4 * p.x * [0.0, 1.0] + 1e-9 * r.standard_normal(p.x.shape)
    z = np.zeros_like(u)
    a, b = p.context(precision=nat.PD_MIXED), p.context(precision=nat.PD_MIXED)
    for c in (a, b):
        c.set_state(u, z, z)
    bt = nat.Batch(nat.PD_MIXED)
    bt.add(b)
    bt.set_config(persistent=1)
    for _ in range(3):
        a.step(40)
        bt.step(40)
    bt.synchronize()
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y, equal_nan=True)
    assert np.array_equal(a.bond_mask(), b.bond_mask())
    bt.remove(b)
    bt.close()
    a.close()
    b.close()
