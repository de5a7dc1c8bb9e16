"""Batches whose fits have wide and direct tiles (a CTA each): more of them than
CTAs, so that a CTA goes from one fit's tiles to another's, and with fewer chunks
of 32 sessions than the CTA has warps, so that some warps have no chunk of a fit.
Each fit against the FP64 oracle, with the tolerances of the other EM tests."""
import numpy as np
import pytest

from massiveclicks_gb300 import api
from oracle import bindings

pytestmark = pytest.mark.gpu

PARAM_RTOL = 1e-5
PARAM_ATOL = 1e-6
WINDOW = 704  # queries of more documents are direct


def _sessions(queries, seed):
    """queries: (documents, sessions, share of sessions with clicks), each document shown."""
    rng = np.random.default_rng(seed)
    query, pidx, clicks, base = [], [], [], 0
    for k, (pool, n, clicked) in enumerate(queries):
        cover = np.minimum(np.arange(-(-pool // 10))[:, None] * 10, pool - 10)
        n = max(n, len(cover))
        first = rng.integers(0, pool - 9, (n, 1))
        first[:len(cover)] = cover
        mask = (rng.random((n, 10)) < 0.25) @ (1 << np.arange(10))
        mask[rng.random(n) >= clicked] = 0
        query.append(np.full(n, k))
        pidx.append(base + first + np.arange(10))
        clicks.append(mask)
        base += pool
    pidx = np.concatenate(pidx).astype(np.int32)
    return api.SessionSet(np.concatenate(query).astype(np.int32), pidx, pidx, np.concatenate(clicks).astype(np.uint16)), base


def _upload(model, sessions, n_qd):
    cm = api.ClickModel.create(model)
    cm.configure(0, WINDOW, 0)
    cm.upload(sessions, n_qd)
    assert cm.fused_path()[0] == "tiles"
    return cm


def _check(cm, model, sessions, n_qd, iters, what):
    f = bindings.OracleFit("f64", model, 0, sessions.query, sessions.pidx, sessions.click, n_qd)
    f.run(iters)
    got = cm.get_parameters()
    for name, ref in f.values().items():
        err = np.abs(got[name].astype(np.float64) - ref)
        assert np.all(err <= PARAM_RTOL * np.abs(ref) + PARAM_ATOL), f"{what} {name}: {err.max():.3g}"


@pytest.mark.parametrize("models", [(api.DBN,), (api.CCM,), (api.DBN, api.CCM)])
def test_more_wide_tiles_than_ctas_over_many_fits(models):
    fits = []
    for k in range(300):
        rng = np.random.default_rng(k)
        sessions, n_qd = _sessions([(680 + k % 5, int(rng.integers(70, 200)), 0.7), (12, 3, 1.0),
                                    (690 + k % 4, int(rng.integers(70, 120)), 0.0 if k % 7 == 0 else 0.5),
                                    (720 + k % 3, int(rng.integers(73, 200)), 0.8)], k)
        fits.append((models[k % len(models)], sessions, n_qd))
    batch_models = [_upload(*f) for f in fits]
    batch = api.Batch(batch_models)
    batch.em(4)
    for k, (f, cm) in enumerate(zip(fits, batch_models)):
        _check(cm, *f, 4, f"fit {k}")
    batch.close()


def test_em_after_a_refused_shape_is_an_error():
    """A window that no CTA holds: configure refuses it, and EM has no tiles to
    run over until another shape is set."""
    sessions, n_qd = _sessions([(40, 90, 0.8), (12, 30, 0.5)], 1)
    cm = _upload(api.DBN, sessions, n_qd)
    with pytest.raises(api._capi.MCError):
        cm.configure(0, 16384, 0)
    for call in (lambda: cm.em(1), lambda: cm.em_trace(1)):
        with pytest.raises(api._capi.MCError):
            call()
    cm.configure(0, WINDOW, 0)
    cm.em(3)
    _check(cm, api.DBN, sessions, n_qd, 3, "after a refused shape")


def _mixed_fits():
    """DBN and CCM fits with windows between a DBN and a CCM warp's memory, and a
    DBN fit so large that a batch with it takes more sessions per tile."""
    small = [(660, 90, 0.8), (410, 60, 0.7), (25, 300, 0.6), (12, 5, 1.0)]
    large = [(20, 150, 0.9)] * 2000
    return [(m, *_sessions(q, k)) for k, (m, q) in enumerate([(api.DBN, small), (api.CCM, small), (api.CCM, small[1:]), (api.DBN, large)])]


def test_models_alone_after_a_mixed_batch():
    fits = _mixed_fits()
    models = [_upload(*f) for f in fits]
    batch = api.Batch(models)
    batch.em(2)
    for f, cm in zip(fits, models):
        cm.em(2)
        cm.em_trace(1)
        _check(cm, *f, 5, "alone after a batch")
    batch.em(1)
    for f, cm in zip(fits, models):
        _check(cm, *f, 6, "batch after alone")
    batch.close()


def test_overlapping_batches_keep_their_tiles():
    fits = _mixed_fits()
    models = [_upload(*f) for f in fits]
    first = api.Batch(models[:2])
    second = api.Batch(models)
    third = api.Batch(models[1:])
    first.em(1)
    second.em(2)
    third.em(1)
    first.em(1)
    for k, (f, cm) in enumerate(zip(fits, models)):
        _check(cm, *f, 2 + 2 * (k < 2) + (k > 0), f"overlapping batches, fit {k}")
    second.close()
    first.em(1)
    third.em(1)
    for k, (f, cm) in enumerate(zip(fits, models)):
        _check(cm, *f, 2 + 3 * (k < 2) + 2 * (k > 0), f"after one was closed, fit {k}")
    first.close()
    third.close()
