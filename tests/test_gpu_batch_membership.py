"""A context stepped alone, as a member of a batch, alone again and back in it: its step
graphs are those of its place (alone, small plates' passes hand over at their blocks'
exit), and the run equals an uninterrupted one, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed,nx,ny", [(False, 61, 43), (False, 244, 245), (False, 245, 245),  # 60,000 particles
                                         (True, 61, 43), (True, 300, 300)])
def test_steps_alone_and_in_a_batch(pdg, mixed, nx, ny):
    nat = pdg.native
    prec = nat.PD_MIXED if mixed else nat.PD_FP64
    p = pdg.plates.make_plate(nx, ny, seed=3, crack="centre-half")
    r = np.random.default_rng(4)
    state = 4e-4 * p.x * [0.0, 1.0] + 1e-8 * r.standard_normal(p.x.shape), 0.3 * r.standard_normal(p.x.shape), 0.0 * p.x
    a, b = p.context(precision=prec), p.context(precision=prec)
    for c in (a, b):
        c.set_state(*state)
    bt = nat.Batch(prec)
    for round_ in range(2):
        b.step(4)
        bt.add(b)
        bt.step(4)
        bt.synchronize()
        bt.remove(b)
        b.step(4)
    a.step(24)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y, equal_nan=True)
    assert np.array_equal(a.bond_mask(), b.bond_mask()) and a.counters() == b.counters()
    assert a.counters()["bonds_broken"] > 0
    bt.close()
    a.close()
    b.close()
