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
