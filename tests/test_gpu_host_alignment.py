"""pd_step_host and pd_compute_velocity on page-locked buffers of which some begin
8 bytes into a 16-byte element: taken, and equal to the calls on aligned buffers,
bit for bit, in every mode and on either side of the sizes where the routes change."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _buffers(pdg, n, odd):
    """Page-locked [n][2] arrays; those of odd begin 8 bytes past a 16-byte boundary."""
    keep = [pdg.native.PinnedArray(2 * n + 1) for _ in odd]
    out = [k.array[o:2 * n + o].reshape(n, 2) for k, o in zip(keep, odd)]
    for a, o in zip(out, odd):
        assert a.ctypes.data % 16 == 8 * o
    return keep, out


def _state(x, seed):
    r = np.random.default_rng(seed)
    return (4e-4 * x * [0.0, 1.0] + 1e-8 * r.standard_normal(x.shape), 0.1 * r.standard_normal(x.shape),
            1e6 * r.standard_normal(x.shape))


def _check(make, pdg, x, steps, odd):
    a, b = make(), make()
    keep, bufs = _buffers(pdg, x.shape[0], odd)
    state = _state(x, steps)
    for h, s in zip(bufs, state):
        h[:] = s
    a.set_state(*state)
    a.step(steps)
    b.step_host(steps, *bufs)
    want = a.state()
    for w, got, s, h in zip(want, bufs[3:], state, bufs):
        assert np.array_equal(w, got) and np.array_equal(s, h)
    b.step_host(steps, *bufs[3:])  # in place
    a.set_state(*want)
    a.step(steps)
    for w, got in zip(a.state(), bufs[3:]):
        assert np.array_equal(w, got)
    assert a.counters() == b.counters()
    a.close()
    b.close()
    del bufs


@pytest.mark.parametrize("odd", [o for o in itertools.product((0, 1), repeat=6) if sum(o) in (0, 1, 6)])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_step_host_on_views(pdg, mode, odd):
    nat = pdg.native
    p = pdg.plates.make_plate(41, 37, seed=3, crack="centre-half")
    _check(lambda: p.context(precision=nat.PD_MIXED if mode == "mixed" else nat.PD_FP64), pdg, p.x, 2, odd)


@pytest.mark.parametrize("odd", [(0, 0, 0, 0, 0, 0), (1, 0, 1, 0, 0, 0), (0, 0, 0, 0, 1, 0)])
@pytest.mark.parametrize("mode,side", [("fp64", 480), ("mixed", 951)])
def test_step_host_on_views_slab_pipelines(pdg, mode, side, odd):
    nat = pdg.native
    p = pdg.plates.make_plate(side, seed=3, crack="centre-half")
    for steps in (1, 3):
        _check(lambda: p.context(precision=nat.PD_MIXED if mode == "mixed" else nat.PD_FP64), pdg, p.x, steps, odd)


@pytest.mark.parametrize("odd", [(0, 0, 0, 0, 0, 0), (1, 0, 0, 0, 0, 0), (0, 1, 0, 1, 0, 1)])
def test_step_host_on_views_bond_associated(pdg, odd):
    x = np.stack([np.arange(72) % 9, np.arange(72) // 9], axis=1).astype(np.float64)

    def make():
        ctx = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, n1=10.0, n2=10.0,
                                                    weight_len=3.0))
        ctx.set_particles(x, np.ones(72))
        ctx.build_families(3.03)
        return ctx

    _check(make, pdg, x, 2, odd)


@pytest.mark.parametrize("odd", [o for o in itertools.product((0, 1), repeat=4) if sum(o) in (0, 1, 4)])
@pytest.mark.parametrize("side", [37, 480])
def test_compute_velocity_on_views(pdg, side, odd):
    p = pdg.plates.make_plate(side, seed=5)
    a, b = p.context(), p.context()
    u, v, acc = _state(p.x, 1)
    keep, (hu, hv, ha, hf) = _buffers(pdg, p.n, odd)
    hu[:], hv[:], ha[:] = u, v, acc
    for _ in range(2):
        fa = a.compute_velocity(u, v, acc)
        b.compute_velocity(hu, hv, ha, netf=hf)
        assert np.array_equal(v, hv) and np.array_equal(acc, ha) and np.array_equal(fa, hf)
    a.close()
    b.close()
    del hu, hv, ha, hf
