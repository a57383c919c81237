"""pd_step_host and pd_compute_velocity on either side of the sizes where they
change from one stream to the slab pipelines (FP64 220,000 particles, mixed
900,000), and step counts around the 16-step graph of the one-stream route:
equal to pd_set_state + pd_step + pd_get_state (or the call on pageable
buffers), bit for bit, with bonds breaking."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(p, seed):
    r = np.random.default_rng(seed)
    u = 4e-4 * p.x * [0.0, 1.0] + 1e-8 * r.standard_normal(p.x.shape)
    u[np.abs(p.x - p.x[p.n // 3]).max(axis=1) < 5e-3, 1] += 2e-6  # bonds that break
    return u, 0.1 * r.standard_normal(p.x.shape), 1e6 * r.standard_normal(p.x.shape)


@pytest.mark.parametrize("mixed,nx,ny,counts", [(False, 1, 1, (1, 2)), (False, 61, 43, (1, 2, 16, 17, 18, 33, 40)),
                                                (False, 470, 467, (1, 3)), (False, 471, 470, (1, 3)),
                                                (True, 1, 1, (1, 2)), (True, 61, 43, (1, 2, 16, 17, 18, 33, 40)),
                                                (True, 949, 947, (1, 3)), (True, 951, 949, (1, 3))])
def test_step_host_routes_equal_staged_steps(pdg, mixed, nx, ny, counts):
    nat = pdg.native
    p = pdg.plates.make_plate(nx, ny, seed=3, crack="centre-half" if nx > 1 else None)
    prec = nat.PD_MIXED if mixed else nat.PD_FP64
    a, b = p.context(precision=prec), p.context(precision=prec)
    bufs = [nat.PinnedArray((p.n, 2)) for _ in range(6)]
    hin, hout = [x.array for x in bufs[:3]], [x.array for x in bufs[3:]]
    for seed, steps in enumerate(counts):
        for h, s in zip(hin, _state(p, seed)):
            h[:] = s
        a.set_state(*hin)
        a.step(steps)
        want = a.state()
        b.step_host(steps, *hin, *hout)
        for w, h in zip(want, hout):
            assert np.array_equal(w, h), steps
        b.step_host(steps, *hin)  # in place, once more (with the bonds that broke)
        a.set_state(*_state(p, seed))
        a.step(steps)
        for w, h in zip(a.state(), hin):
            assert np.array_equal(w, h), steps
    ca, cb = a.counters(), b.counters()
    assert ca["bonds_broken"] == cb["bonds_broken"] and ca["steps"] == cb["steps"]
    if nx > 1:
        assert ca["bonds_broken"] > 0
    a.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (61, 43), (471, 470)])
def test_compute_velocity_routes_equal_pageable(pdg, nx, ny):
    nat = pdg.native
    p = pdg.plates.make_plate(nx, ny, seed=5)
    a, b = p.context(), p.context()
    u, v, acc = _state(p, 1)
    bufs = [nat.PinnedArray((p.n, 2)) for _ in range(4)]
    hu, hv, ha, hf = (x.array for x in bufs)
    hu[:], hv[:], ha[:] = u, v, acc
    for _ in range(2):
        fa = a.compute_velocity(u, v, acc)
        b.compute_velocity(hu, hv, ha, netf=hf)
        assert np.array_equal(v, hv) and np.array_equal(acc, ha) and np.array_equal(fa, hf)
    a.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(837, 836), (837, 837), (1013, 991)])
def test_slab_plans_equal_staged_steps(pdg, nx, ny):
    """Either side of 700,000 particles, where the even slabs get finer, and the most slabs."""
    test_step_host_routes_equal_staged_steps(pdg, False, nx, ny, (1, 3))


@pytest.mark.parametrize("nx,ny,order", [(480, 480, "reversed"), (480, 480, "shuffled"), (840, 840, "reversed"),
                                         (840, 840, "shuffled")])
def test_slab_plans_other_numberings(pdg, nx, ny, order):
    """Numberings in which the slabs' neighbours lie in earlier, or in all, slabs."""
    import dataclasses
    p = pdg.plates.make_plate(nx, ny, seed=9, crack="centre-half")
    perm = np.arange(p.n)[::-1] if order == "reversed" else np.random.default_rng(2).permutation(p.n)
    p = dataclasses.replace(p, x=np.ascontiguousarray(p.x[perm]), vol=np.ascontiguousarray(p.vol[perm]),
                            group_of=np.ascontiguousarray(p.group_of[perm]))
    a, b = p.context(), p.context()
    bufs = [nat.PinnedArray((p.n, 2)) for nat in [pdg.native] * 3]
    h = [x.array for x in bufs]
    for seed, steps in enumerate((1, 2, 1)):
        state = _state(p, seed)
        for x, y in zip(h, state):
            x[:] = y
        a.set_state(*state)
        a.step(steps)
        b.step_host(steps, *h)
        for w, x in zip(a.state(), h):
            assert np.array_equal(w, x), steps
    assert a.counters()["bonds_broken"] == b.counters()["bonds_broken"] > 0
    a.close()
    b.close()
