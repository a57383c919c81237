"""pd_compute_velocity_noalloc at the edges of its two forms (16 lanes per
particle up to 4,096 particles, two threads per particle above): one particle,
partial warps and blocks, both sides of the limit, the largest call, families
past 16 and 32 bonds, rows of unequal length, a captured call, and a bad index
in either form; bit for bit against pd_compute_velocity."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(pdg, torch, n, bufs, params, stream=None):
    err = ctypes.create_string_buffer(256)
    rc = pdg.native.lib().pd_compute_velocity_noalloc(n, *(ctypes.c_void_p(b.data_ptr()) for b in bufs),
                                                      ctypes.byref(params), ctypes.c_void_p(stream), err, 256)
    assert rc == 0, err.value


@pytest.mark.parametrize("nx,ny,horizon", [(1, 1, 3.015), (2, 1, 3.015), (5, 3, 3.015), (17, 9, 4.6), (64, 64, 3.015),
                                           (241, 17, 3.015), (83, 51, 4.6), (256, 256, 3.015)])
def test_noalloc_shapes_match_compute_velocity(pdg, nx, ny, horizon):
    torch = pytest.importorskip("torch")
    p = pdg.plates.make_plate(nx, ny, seed=9, horizon=horizon)
    r = np.random.default_rng(1)
    n = p.n
    vol = p.vol * (1.0 + 0.2 * r.random(n))
    ctx = pdg.native.Context(p.params(s_c=0.0))
    ctx.set_particles(p.x, vol)
    ctx.build_families(p.cutoff)
    rp, col = ctx.families()
    u, v, acc = (1e-7 * r.standard_normal((n, 2)) for _ in range(3))
    d = torch.device("cuda", 0)
    t = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(d, dt)
    col_t = t(col if col.size else np.zeros(1, np.int32), torch.int32)
    bufs = [t(p.x), t(vol), t(rp, torch.int64), col_t, t(u), t(v), t(acc), torch.zeros((n, 2), dtype=torch.float64, device=d)]
    hv, hacc = v.copy(), acc.copy()
    _call(pdg, torch, n, bufs, p.params(s_c=0.0))
    torch.cuda.synchronize()
    hf = ctx.compute_velocity(u, hv, hacc)
    for dev, host in zip(bufs[5:], (hv, hacc, hf)):
        assert np.array_equal(dev.cpu().numpy(), host)
    if nx == 64:  # and captured in a graph
        bufs[5].copy_(t(v))
        bufs[6].copy_(t(acc))
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            _call(pdg, torch, n, bufs, p.params(s_c=0.0), torch.cuda.current_stream().cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(bufs[5].cpu().numpy(), hv) and np.array_equal(bufs[7].cpu().numpy(), hf)
    ctx.close()


@pytest.mark.parametrize("nx,ny,horizon", [(4097, 1, 1.015), (4111, 1, 2.015), (4099, 1, 3.015), (2051, 2, 1.015),
                                           (2051, 2, 2.015), (1400, 3, 2.015), (1401, 3, 3.015), (90, 47, 3.5)])
def test_noalloc_rows_past_whole_groups_match_compute_velocity(pdg, nx, ny, horizon):
    """Rows of 1 to ~36 bonds: whole groups of four and 0 .. 3 bonds past them."""
    test_noalloc_shapes_match_compute_velocity(pdg, nx, ny, horizon)


@pytest.mark.parametrize("side", [40, 70])
def test_noalloc_bad_index_poisons_its_particle(pdg, side):
    torch = pytest.importorskip("torch")
    p = pdg.plates.make_plate(side, seed=4)
    n, bad = p.n, p.n // 2
    ctx = pdg.native.Context(p.params(s_c=0.0))
    ctx.set_particles(p.x, p.vol)
    ctx.build_families(p.cutoff)
    rp, col = ctx.families()
    reach = np.unique(np.append(col[rp[bad]:rp[bad + 1]], bad))
    col = col.copy()
    col[rp[bad + 1] - 1] = -3  # the last of its row
    d = torch.device("cuda", 0)
    t = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(d, dt)
    z = lambda: torch.zeros((n, 2), dtype=torch.float64, device=d)
    u = 1e-7 * np.random.default_rng(2).standard_normal((n, 2))
    bufs = [t(p.x), t(p.vol), t(rp, torch.int64), t(col, torch.int32), t(u), z(), z(), z()]
    _call(pdg, torch, n, bufs, p.params(s_c=0.0))
    torch.cuda.synchronize()
    f = bufs[7].cpu().numpy()
    nan = np.flatnonzero(np.isnan(f).any(axis=1))
    assert bad in nan and np.isin(nan, reach).all()
    ctx.close()
