"""The Mazars weight table is made by the calls that set the damage or its weights up
(pd_mazars_init, pd_set_params), whichever comes last, and let go with the history; an
update allocates nothing.  The updates equal those of a context set up at once, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDE = 150
N = SIDE * SIDE
TABLE = 16384 * N  # bytes


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _taken(torch, call):
    before = _free(torch)
    call()
    return before - _free(torch)


def test_table_comes_with_the_set_up(pdg):
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    x = np.stack([np.arange(N) % SIDE, np.arange(N) // SIDE], axis=1).astype(np.float64)
    u = np.stack([-4e-5 * x[:, 0], 1.2e-4 * x[:, 1]], axis=1) + 2e-5 * np.random.default_rng(3).random((N, 2))

    def make(**kw):
        ctx = pdg.native.Context(pdg.default_params(E=3.5e4, nu=0.2, rho=2.5e-6, dt=1e-9, weight_len=3.0, **kw))
        ctx.set_particles(x, np.ones(N))
        ctx.build_families(3.03)
        ctx.set_state(u=u)
        return ctx

    def update(ctx):
        assert _taken(torch, ctx.mazars_update) < 0.05 * TABLE
        return ctx.mazars()

    a = make(n1=10.0, n2=10.0)  # the weights first, then the damage
    assert _taken(torch, lambda: a.mazars_init(kappa0=8e-5)) > 0.95 * TABLE
    want = update(a)
    assert (want[1] > 0.0).any()
    assert _taken(torch, lambda: a.mazars_init(kappa0=8e-5)) < 0.05 * TABLE  # once
    again = update(a)
    b = make()  # the damage first
    no_history = b.checkpoint()
    assert _taken(torch, lambda: b.mazars_init(kappa0=8e-5)) < 0.2 * TABLE
    assert _taken(torch, lambda: b.set_params(n1=10.0, n2=10.0)) > 0.95 * TABLE
    late = update(b)
    for p, q, r in zip(want, again, late):
        assert np.array_equal(p, q) and np.array_equal(p, r)
    b.set_params(n1=4.5, n2=2.5)  # other weights: the table follows
    c = make(n1=4.5, n2=2.5)
    c.mazars_init(kappa0=8e-5)
    b.mazars_init(kappa0=8e-5)
    for p, q in zip(update(b), update(c)):
        assert np.array_equal(p, q)
    b.set_params(n1=0.0, n2=0.0)
    assert _taken(torch, lambda: b.restore(no_history)) < -0.95 * TABLE  # a blob without the history
    for ctx in (a, b, c):
        ctx.close()
