"""Which tiles a query goes to (a warp's, several warps', a CTA's) and the bins that
they sum in: every route against the FP64 oracle, with the tolerances of the other
EM tests."""
import numpy as np
import pytest

from massiveclicks_gb300 import api
from oracle import bindings

pytestmark = pytest.mark.gpu

PARAM_RTOL = 1e-5
PARAM_ATOL = 1e-6


def _sessions(queries, seed):
    """queries: (documents, sessions), each document shown, three sessions in four clicked."""
    rng = np.random.default_rng(seed)
    query, pidx, clicks, base = [], [], [], 0
    for k, (pool, n) in enumerate(queries):
        cover = np.minimum(np.arange(-(-pool // 10))[:, None] * 10, pool - 10)
        n = max(n, len(cover))
        first = rng.integers(0, pool - 9, (n, 1))
        first[:len(cover)] = cover
        mask = (rng.random((n, 10)) < 0.2) @ (1 << np.arange(10))
        mask[rng.random(n) < 0.15] = 0
        query.append(np.full(n, k))
        pidx.append(base + first + np.arange(10))
        clicks.append(mask)
        base += pool
    pidx = np.concatenate(pidx).astype(np.int32)
    return api.SessionSet(np.concatenate(query).astype(np.int32), pidx, pidx, np.concatenate(clicks).astype(np.uint16)), base


def _fit_and_check(model, queries, seed, iters, values=None):
    sessions, n_qd = _sessions(queries, seed)
    cm = api.ClickModel.create(model)
    cm.upload(sessions, n_qd)
    assert cm.fused_path()[0] == "tiles"
    f = bindings.OracleFit("f64", model, 0, sessions.query, sessions.pidx, sessions.click, n_qd)
    if values:
        v = cm.get_parameters()
        for name, x in values.items():
            v[name][:] = x
        cm.set_parameters(v)
        f.set_values(v)
    cm.em(iters)
    f.run(iters)
    got = cm.get_parameters()
    for name, ref in f.values().items():
        err = np.abs(got[name].astype(np.float64) - ref)
        assert np.all(err <= PARAM_RTOL * np.abs(ref) + PARAM_ATOL), f"m{model} {name}: {err.max():.3g}"


@pytest.mark.parametrize("queries", [[(20, 90)] * 40 + [(30, 1300)], [(680, 300)] * 5 + [(900, 1500)]], ids=["narrow", "wide"])
def test_float_bins(queries):
    """Continuations near 1 leave CCM's terms too large for fixed-point bins."""
    _fit_and_check(api.CCM, queries, 1, 2, {"continuation": [0.9, 0.9999, 0.999]})


ROUTES = {
    # both sides of the windows and sessions at which a query is cut (64 sessions per narrow tile in fits this small)
    "limits": [(w, n) for w in (40, 41, 80, 81) for n in (60, 75, 76, 77, 90, 148, 150, 152, 170, 900)],
    # runs of wide queries with narrow ones before, between and after them
    "runs": [(14, 20), (700, 100), (12, 3), (12, 300), (690, 90), (15, 40), (1500, 160), (700, 80), (1200, 150), (11, 2)] * 5,
    # queries of several blocks, cut or a CTA's, staged and direct
    "heads": [(30, 3000), (64, 2500), (65, 2500), (300, 2500), (12, 5), (700, 4200), (1600, 2500), (1536, 5000)],
}


@pytest.mark.parametrize("model", [api.CCM, api.DBN])
@pytest.mark.parametrize("route", ROUTES)
def test_routes(model, route):
    _fit_and_check(model, ROUTES[route], len(route), 4)


@pytest.mark.parametrize("block", [64, 96, 160, 256])
def test_blocks_of_other_sizes(block):
    queries = ROUTES["runs"][:10] + ROUTES["heads"][:3]
    sessions, n_qd = _sessions(queries, 9)
    values = []
    for b in (256, block):
        cm = api.DBNModel()
        cm.configure(0, 0, b)
        cm.upload(sessions, n_qd)
        cm.em(3)
        values.append(cm.get_parameters())
    for name in values[0]:
        np.testing.assert_allclose(values[1][name], values[0][name], rtol=PARAM_RTOL, atol=PARAM_ATOL, err_msg=name)
