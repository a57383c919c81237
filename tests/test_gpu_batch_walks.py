"""Mixed batches in every mode, whose pass A takes another number of bonds at a time than
the single-plate one: rows of one bond to wide ones (every remainder), graded volumes, a plate
whose blocks are not staged, and bonds breaking; equal to the plates alone, bit for bit."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plates(pdg):
    mk = pdg.plates.make_plate
    out = [mk(40, 17, seed=2, horizon=h) for h in (1.015, 1.5, 2.015, 2.3, 3.015, 3.5, 4.6)] + [mk(1, 1), mk(37, 1), mk(48, 48)]
    r = np.random.default_rng(1)
    out += [dataclasses.replace(p, vol=p.vol * (1.0 + 0.2 * r.random(p.n))) for p in out[4:6]]
    p = mk(120, seed=5, crack="centre-half")  # shuffled, with two far particles: its blocks are not staged
    perm = r.permutation(p.n)
    far = np.array([[-5.0, -5.0], [5.0, 5.0]])
    out.append(dataclasses.replace(
        p, x=np.ascontiguousarray(np.vstack([p.x[perm], far])), vol=np.concatenate([p.vol[perm], p.vol[:2]]),
        group_of=np.ascontiguousarray(np.concatenate([p.group_of[perm], np.zeros(2, p.group_of.dtype)]))))
    return out


@pytest.mark.parametrize("persistent,blocks_per_sm", [(0, 1), (1, 1), (1, 4), (2, 1)])
def test_batch_walks_equal_single_plates(pdg, persistent, blocks_per_sm):
    nat = pdg.native
    plates = _plates(pdg)
    r = np.random.default_rng(6)
    b = nat.Batch(nat.PD_MIXED)
    pairs = []
    for p in plates:
        u = 3e-4 * p.x * [0.0, 1.0] + 1e-8 * r.standard_normal(p.x.shape)
        u[r.random(p.n) < 0.05] += 1.5e-6  # bonds that break
        pair = p.context(precision=nat.PD_MIXED), p.context(precision=nat.PD_MIXED)
        for c in pair:
            c.set_state(u, 0.1 * p.x * 0.0, 0.0 * p.x)
        b.add(pair[1])
        pairs.append(pair)
    assert pairs[-1][0].counters()["unstaged_blocks"] > 0
    b.set_config(persistent=persistent, blocks_per_sm=blocks_per_sm)
    b.step(2)
    b.step(5)
    b.synchronize()
    broken = []
    for one, member in pairs:
        one.step(7)
        for x, y in zip(one.state(), member.state()):
            assert np.array_equal(x, y, equal_nan=True)
        assert np.array_equal(one.bond_mask(), member.bond_mask()) and one.counters() == member.counters()
        broken.append(one.counters()["bonds_broken"])
    assert sum(n > 0 for n in broken) >= 9 and broken[-1] > 0
    b.close()
    for pair in pairs:
        for c in pair:
            c.close()
