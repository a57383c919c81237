"""The bond-associated tables and reverse slots follow the bond mask whatever
changed it, and under whichever weights: formed over families that classic steps
had cut, then set aside for the classic weights, under which a reset or a restore
brings the bonds back, then set again.  Against a fresh context over the same
bonds, bit for bit, and for whole families the oracle.  (Of cut families some hold
one or two bonds, whose shape tensors are singular to rounding: volumes off by
3e-16 move the oracle's own forces by 7e-8 there.)"""
import numpy as np
import pytest

from conftest import normwise

pytestmark = pytest.mark.gpu
TOL = 1e-12  # as tests/test_gpu_bond_assoc.py: the weights' exp and pow differ in the last bits
BA, CLASSIC = dict(s_c=0.0, n1=10.0, n2=10.0), dict(s_c=1e-3, n1=0.0, n2=0.0)


def _ctx(pdg, x, vol, cutoff, **kw):
    ctx = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, weight_len=3.0, **kw))
    ctx.set_particles(x, vol)
    ctx.build_families(cutoff)
    return ctx


@pytest.mark.parametrize("cutoff", [3.03, 3.7])  # families of up to 32 bonds, and wider ones
@pytest.mark.parametrize("back", ["reset", "restore", "restore-cut", "steps"])
def test_tables_follow_the_mask_under_classic_weights(pdg, po, back, cutoff):
    r = np.random.default_rng(4)
    x = np.stack([np.arange(72) % 9, np.arange(72) // 9], axis=1) + 0.02 * r.random((72, 2))
    vol = 1.0 + 0.2 * r.random(72)
    ctx = _ctx(pdg, x, vol, cutoff, **CLASSIC)
    z = np.zeros_like(x)

    def cut(seed, part):
        d = 1e-2 * np.random.default_rng(seed).standard_normal(x.shape) * (x[:, :1] < part)
        before = ctx.counters()["bonds_broken"]
        ctx.set_state(d, z, z)
        ctx.step(1)
        assert ctx.counters()["bonds_broken"] > before

    whole = ctx.checkpoint()
    cut(1, 3.5)
    partly = ctx.checkpoint()
    cut(2, 6.5)
    ctx.set_params(**BA)
    ctx.step(1)
    ctx.set_params(**CLASSIC)
    if back == "reset":
        ctx.reset()
    elif back == "restore":
        ctx.restore(whole)
    elif back == "restore-cut":
        ctx.restore(partly)
    else:
        cut(3, 99.0)
    mask = ctx.bond_mask().astype(bool)
    assert mask.all() == (back in ("reset", "restore"))
    ctx.set_params(**BA)
    # the reference: the same bonds as the families of a new context
    rp, col = ctx.families()
    row = np.repeat(np.arange(72), np.diff(rp))
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(row[mask], minlength=72))]).astype(np.int64)
    fresh = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, weight_len=3.0, **BA))
    fresh.set_particles(x, vol)
    fresh.set_families(rp2, col[mask])
    sim = po.OracleSim(x, vol, rp2, col[mask], E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, n1=10.0, n2=10.0, wlen=3.0)
    u = 1e-4 * r.standard_normal(x.shape)
    sim.u[:] = u
    sim.step(3)
    for c in (ctx, fresh):
        c.set_state(u, z, z)
        c.step(3)
    for a, b, o in zip(ctx.state(), fresh.state(), (sim.u, sim.v, sim.f)):
        assert np.array_equal(a, b) and (not mask.all() or normwise(a, o) < TOL)
    ctx.close()
    fresh.close()
