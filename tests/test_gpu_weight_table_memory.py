"""The bond-associated weight tables by the device memory that is free: a table takes
at most a quarter of it, the step falls back to its triangles and then to evaluated
weights, the Mazars update to evaluated weights, with the same results bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GB = 1 << 30


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_tables_by_free_memory(pdg):
    torch = pytest.importorskip("torch")
    side, widest = 520, 28
    n = side * side
    x = np.stack([np.arange(n) % side, np.arange(n) // side], axis=1).astype(np.float64)
    r = np.random.default_rng(3)
    u = np.stack([-4e-5 * x[:, 0], 1.2e-4 * x[:, 1]], axis=1) + 2e-5 * r.random((n, 2))
    z = np.zeros_like(u)
    slots = -(-n // 32) * 32 * widest
    buffers, matrices, triangles = 88 * slots + 8 * n, 8192 * n, 4224 * n  # per slot and per particle
    mazars = 16384 * n + 32 * slots
    want = None
    for room, table, damage_table in ((None, matrices, mazars), (6 * GB, triangles, 0),
                                      (buffers + triangles // 2, 0, 0)):
        ctx = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, weight_len=3.0))
        ctx.set_particles(x, np.ones(n))
        ctx.build_families(3.03)
        assert int(np.diff(ctx.families()[0]).max()) == widest
        torch.zeros(1, device="cuda")
        hog = None if room is None else torch.empty(_free(torch) - room, dtype=torch.uint8, device="cuda")
        before = _free(torch)
        ctx.set_params(n1=10.0, n2=10.0)
        after = _free(torch)
        assert abs(before - after - buffers - table) < 0.05 * triangles
        ctx.mazars_init(kappa0=8e-5)
        with_damage = _free(torch)
        assert abs(after - with_damage - damage_table - 16 * slots - 8 * n) < 0.05 * triangles
        ctx.set_state(u, z, z)
        ctx.mazars_update()
        ctx.step(2)
        ctx.mazars_update()
        assert with_damage - _free(torch) < 0.05 * triangles  # (kernels' code and the step graph: a few MB)
        got = (*ctx.state(), *ctx.mazars())
        assert np.abs(got[4]).max() > 0.0  # bonds are damaged
        want = got if want is None else want
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        ctx.close()
        del hog
        torch.cuda.empty_cache()
