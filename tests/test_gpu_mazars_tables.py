"""Mazars damage with bond-associated weights where the update's weight table
changes hands: families at and past its 32 bonds (those are evaluated in every
update), one particle and a partial block, loading and unloading, and weights
changed by pd_set_params after the table was formed; against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-12  # GPU and oracle differ by their exp / pow in the last bits (as tests/test_gpu_mazars.py)


@pytest.mark.parametrize("nx,ny,horizon,widest", [(1, 1, 3.0, 0), (9, 7, 3.0, 28), (12, 11, 3.17, 36), (10, 9, 4.0, 48)])
def test_mazars_bond_associated_tables_match_oracle(pdg, po, nx, ny, horizon, widest):
    r = np.random.default_rng(5)
    n = nx * ny
    x = np.stack([np.arange(n) % nx, np.arange(n) // nx], axis=1).astype(np.float64)
    vol = 1.0 + 0.2 * r.random(n)
    E, nu, rho, dt, k0 = 3.5e4, 0.2, 2.5e-6, 1e-9, 8e-5
    ctx = pdg.native.Context(pdg.default_params(E=E, nu=nu, rho=rho, dt=dt, s_c=0.0, n1=10.0, n2=10.0, weight_len=3.0))
    ctx.set_particles(x, vol)
    ctx.build_families(1.01 * horizon)
    rp, col = ctx.families()
    assert int(np.diff(rp).max(initial=0)) == widest
    ctx.mazars_init(kappa0=k0)
    thr, bd = np.full(int(rp[-1]), k0), np.zeros(int(rp[-1]))
    u = np.stack([-4e-5 * x[:, 0], 1.2e-4 * x[:, 1]], axis=1) + 2e-5 * r.random((n, 2))
    for n1, n2, scale in ((10.0, 10.0, 1.0), (10.0, 10.0, 0.5), (4.5, 2.5, 1.3)):
        if n1 != 10.0:
            ctx.set_params(n1=n1, n2=n2)
        sim = po.OracleSim(x, vol, rp, col, E=E, nu=nu, rho=rho, dt=dt, n1=n1, n2=n2, wlen=3.0)
        sim.u[:] = scale * u
        st = sim.mazars(thr, bd, k0)
        ctx.set_state(u=scale * u)
        ctx.mazars_update()
        gthr, gbd, gst = ctx.mazars()
        if n > 1:
            assert np.abs(gthr - thr).max() < TOL * np.abs(thr).max()
            assert np.abs(gbd - bd).max() < TOL and np.abs(gst - st).max() < TOL
        else:
            assert not gst.any()
    ctx.close()
