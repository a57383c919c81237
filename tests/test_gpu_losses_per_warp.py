"""Every number of a warp's particles losing a bond in one step, from none to all
of them, through both forms of pass A's K^-1 update (by the whole warp; each lane
its own): the two threads of an FP64 particle take the same new K^-1, which the
state, mask and damage show against the oracle, bit for bit.

Each particle under test ("head") has six neighbours of its own ("anchors", with
no family), one of which is moved away for the heads that are to lose a bond."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_MOD, NU, RHO, S_C, DX, ANCHORS = 72e9, 0.33, 2440.0, 5e-4, 1e-3, 6


def _heads(n_heads, lose, pad, seed):
    """Positions, volumes, families and state: ids 0 .. n_heads are the heads, their
    anchors follow, then pad particles without bonds."""
    r = np.random.default_rng(seed)
    side = 64
    h = np.stack([np.arange(n_heads) % side, np.arange(n_heads) // side], axis=1) * DX
    ang = 2.0 * np.pi * (np.arange(ANCHORS) / ANCHORS + 0.05 * r.random((n_heads, ANCHORS)))
    rad = 100 * DX * (1.0 + 0.2 * r.random((n_heads, ANCHORS)))  # past the heads, which fill their tiles alone
    anchors = h[:, None, :] + rad[..., None] * np.stack([np.cos(ang), np.sin(ang)], axis=2)
    m = n_heads * (1 + ANCHORS)
    x = np.concatenate([h, anchors.reshape(-1, 2),
                        np.stack([np.arange(pad) % 500, -5.0 - np.arange(pad) // 500], axis=1) * DX])
    row_ptr = np.zeros(m + pad + 1, np.int64)
    row_ptr[1:n_heads + 1] = ANCHORS * np.arange(1, n_heads + 1)
    row_ptr[n_heads + 1:] = ANCHORS * n_heads
    col = np.arange(n_heads, m, dtype=np.int32)
    vol = 1e-9 * (1.0 + 0.2 * r.random(m + pad))
    u = np.zeros_like(x)
    u[:m] = 1e-9 * r.standard_normal((m, 2))
    moved = n_heads + ANCHORS * np.flatnonzero(lose) + r.integers(0, ANCHORS, int(lose.sum()))
    which = (moved - n_heads) // ANCHORS
    u[moved] += 3.0 * S_C * (x[moved] - x[which])
    return x, vol, row_ptr, col, u


@pytest.mark.parametrize("pad", [0, 250000])  # (the tests among the sums; ahead of them)
@pytest.mark.parametrize("seed", [1, 2])
def test_every_number_of_losing_particles_fp64(pdg, po, pad, seed):
    per_warp = 16  # two threads per particle
    r = np.random.default_rng(seed)
    lose = np.concatenate([r.permutation(np.arange(per_warp) < k) for k in range(per_warp + 1)])
    x, vol, row_ptr, col, u = _heads(lose.size, lose, pad, seed)
    k_hg = 1e20
    ctx = pdg.native.Context(pdg.native.default_params(E=E_MOD, nu=NU, rho=RHO, dt=1e-7, s_c=S_C, k_hg=k_hg))
    ctx.set_particles(x, vol)
    ctx.set_families(row_ptr, col)
    sim = po.OracleSim(x, vol, row_ptr, col, E=E_MOD, nu=NU, rho=RHO, dt=1e-7, s_c=S_C, k_hg=k_hg)
    ctx.set_state(u, np.zeros_like(u), np.zeros_like(u))
    sim.u[:] = u
    for _ in range(3):
        ctx.step(1)
        sim.step(1)
        assert np.array_equal(ctx.bond_mask(), sim.mask) and np.array_equal(ctx.damage(), sim.damage)
        for a, b in zip(ctx.state(), (sim.u, sim.v, sim.f)):
            assert np.array_equal(a, b)
    lost = (sim.mask.reshape(-1, ANCHORS) == 0).any(axis=1)
    assert np.array_equal(lost, lose) and np.isfinite(sim.f).all()
    assert ctx.counters()["bonds_broken"] == int(lose.sum())
    ctx.close()


@pytest.mark.parametrize("part", [0.03, 0.2, 0.4, 0.5, 0.9])  # 32 particles per warp; one lane each from 15 on
@pytest.mark.parametrize("uniform", [False, True])
@pytest.mark.parametrize("n_heads", [4096, 4100])
def test_numbers_of_losing_particles_mixed(pdg, part, uniform, n_heads):
    """As a context restored after the losses, whose K^-1 is formed afresh from the mask."""
    r = np.random.default_rng(5)
    lose = r.random(n_heads) < part
    x, vol, row_ptr, col, u = _heads(n_heads, lose, 0, 5)
    if uniform:
        vol[:] = 1e-9
    a, b = (pdg.native.Context(pdg.native.default_params(precision=pdg.native.PD_MIXED, E=E_MOD, nu=NU, rho=RHO,
                                                         dt=1e-7, s_c=S_C, k_hg=1e20)) for _ in range(2))
    for c in (a, b):
        c.set_particles(x, vol)
        c.set_families(row_ptr, col)
    a.set_state(u, np.zeros_like(u), np.zeros_like(u))
    a.step(1)
    mask = a.bond_mask()
    assert np.array_equal((mask.reshape(-1, ANCHORS) == 0).any(axis=1), lose)
    assert a.counters()["bonds_broken"] == int(lose.sum())
    b.restore(a.checkpoint())
    for c in (a, b):
        c.step(2)
    for p, q in zip(a.state(), b.state()):
        assert np.isfinite(p).all() and np.array_equal(p, q)
    assert np.array_equal(a.bond_mask(), b.bond_mask()) and np.array_equal(a.damage(), b.damage())
    a.close()
    b.close()
