"""pd_compute_velocity_noalloc and a bad index or row in the caller's families, in either
form of its pass A: every particle whose family holds the bad one gets NaN (pass A's scratch
carries it: their own rows are sound), and no other particle does."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [40, 64, 70])
@pytest.mark.parametrize("fault", ["first", "last", "past-the-end", "row"])
def test_bad_particle_poisons_its_reach_and_nothing_else(pdg, side, fault):
    torch = pytest.importorskip("torch")
    p = pdg.plates.make_plate(side, seed=4)
    n, bad = p.n, p.n // 2 + 3
    ctx = pdg.native.Context(p.params(s_c=0.0))
    ctx.set_particles(p.x, p.vol)
    ctx.build_families(p.cutoff)
    rp, col = ctx.families()
    ctx.close()
    refused = [bad]
    rp, col = rp.copy(), col.copy()
    rows = {k: col[rp[k]:rp[k + 1]].copy() for k in (bad - 1, bad)}
    if fault == "first":
        col[rp[bad]] = n
    elif fault == "last":
        col[rp[bad + 1] - 1] = -3
    elif fault == "past-the-end":
        col[rp[bad] + 5] = np.iinfo(np.int32).max
    else:  # the two rows that share this bound are not ranges of the families
        rp[bad] = rp[n] + 7
        refused = [bad - 1, bad]
    reach = np.zeros(n, bool)
    for k in refused:  # (the families are symmetric: who is in a row holds the row's particle)
        reach[rows[k]] = True
        reach[k] = True
    d = torch.device("cuda", 0)
    t = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(d, dt)
    z = lambda: torch.zeros((n, 2), dtype=torch.float64, device=d)
    u = 1e-7 * np.random.default_rng(2).standard_normal((n, 2))
    bufs = [t(p.x), t(p.vol), t(rp, torch.int64), t(col, torch.int32), t(u), z(), z(), z()]
    err = ctypes.create_string_buffer(256)
    params = p.params(s_c=0.0)
    rc = pdg.native.lib().pd_compute_velocity_noalloc(n, *(ctypes.c_void_p(b.data_ptr()) for b in bufs),
                                                      ctypes.byref(params), None, err, 256)
    assert rc == 0, err.value
    torch.cuda.synchronize()
    for b in bufs[5:]:
        nan = np.isnan(b.cpu().numpy())
        assert np.array_equal(nan.any(axis=1), nan.all(axis=1)) and np.array_equal(nan.any(axis=1), reach)
