"""The far-field sum at the edges of its chunks, warps and shape-factor forms,
against the oracle."""
import numpy as np
import pytest

from test_gpu_fill import GROUNDS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(nb):
    from gpu_helpers import Engine
    e = Engine(nb.lib)
    yield e
    e.close()


# segments of 0.004 to 0.4 wavelengths (the polynomial shape factors up to
# 1/(2 pi)), one chunk of 256 segments and two, one direction and several per
# warp, the last warp incomplete
@pytest.mark.parametrize("n,length,ndir,ground", [
    (2, 0.8, 1, "free"), (5, 2.0, 7, "free"), (6, 0.9, 33, "perfect"), (255, 4.0, 63, "free"),
    (256, 1.0, 65, "reflection"), (257, 20.0, 17, "perfect"), (257, 120.0, 9, "free"), (31, 4.0, 2369, "free"),
    (33, 9.0, 2403, "reflection")])
def test_pattern_at_edges(nb, oracle, engine, n, length, ndir, ground):
    """Both field components to 1e-12 of the larger one's maximum: a sum of n
    terms whose arguments carry a few roundings of up to 2 pi times the
    antenna's extent each (120 wavelengths: 1e-13)."""
    ctx = nb.nec_create()
    assert nb.nec_wire(ctx, 1, n, 0.1, -0.4 * length, 1.0, 0.2, 0.4 * length, 1.0 + 0.6 * length, 1e-4, 1.0, 1.0) == 0
    assert nb.nec_geometry_complete(ctx, 0) == 0
    if GROUNDS[ground]:
        assert nb.nec_gn_card(ctx, *GROUNDS[ground]) == 0
    assert nb.nec_ex_card(ctx, 0, 1, (n + 1) // 2, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0) == 0
    st = nb.structure(ctx, 299.8)
    rhs = nb.rhs(ctx)
    nb.nec_delete(ctx)
    engine.set_structure(st)
    engine.fill()
    engine.factor(0)
    _, abc = engine.solve(rhs)
    rng = np.random.default_rng(ndir)
    th = rng.uniform(0.0, 1.55, ndir)
    ph = rng.uniform(0.0, 6.28, ndir)
    et, ep = engine.pattern(th, ph)
    some = np.unique(np.concatenate([np.arange(min(ndir, 40)), np.arange(max(0, ndir - 40), ndir)]))
    ref = np.array([oracle.ffld(st, abc, th[k], ph[k]) for k in some])
    scale = np.max(np.abs(ref))
    assert np.max(np.abs(et[some] - ref[:, 0])) <= 1e-12 * scale
    assert np.max(np.abs(ep[some] - ref[:, 1])) <= 1e-12 * scale
