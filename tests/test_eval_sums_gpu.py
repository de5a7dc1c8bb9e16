"""The evaluation's sums: no less exact than FP64 over many sessions, and sessions
with probabilities outside (0, 1] next to others."""
import numpy as np
import pytest

from massiveclicks_gb300 import api

pytestmark = pytest.mark.gpu


def _model(attractiveness):
    """A PBM fit over ten documents with examination 1 at every rank."""
    docs = np.arange(10, dtype=np.int32)[None]
    cm = api.PBMModel()
    cm.upload(api.SessionSet(np.zeros(1, np.int32), docs, docs, np.ones(1, np.uint16)), 10)
    cm.set_parameters({"examination": np.ones(10, np.float32), "attractiveness": np.asarray(attractiveness, np.float32)})
    return cm


def _evaluate(cm, pidx, clicks):
    cm.upload_test(api.SessionSet(None, None, pidx, clicks))
    return cm.evaluate(1)


@pytest.mark.parametrize("seed", [0, 1])
def test_many_like_sessions(seed):
    """16M copies of one session whose terms span seven decades: its sums times
    the number.  A thread's sum is exact; 621 FP64 additions (5 between lanes, 8
    between warps, 608 between blocks) of like signs round by at most 2^-53 each."""
    n = 16_000_000
    rng = np.random.default_rng(seed)
    a = 10.0 ** rng.uniform(-7, -1, 10)
    a[3] = 1e-4
    cm = _model(a)
    one = _evaluate(cm, np.arange(10, dtype=np.int32)[None], np.full(1, 1 << 3, np.uint16))
    got = _evaluate(cm, np.tile(np.arange(10, dtype=np.int32), (n, 1)), np.full(n, 1 << 3, np.uint16))
    np.testing.assert_allclose(got.llh_sum, n * one.llh_sum, rtol=622 * 2.0**-53)
    np.testing.assert_allclose(got.log2_sums, n * one.log2_sums, rtol=622 * 2.0**-53)


@pytest.mark.parametrize("n", [1, 33, 10007, 700_001])
def test_probabilities_outside_the_unit_interval(n):
    """Document 1's attractiveness of 1.5 makes a click's probability 1.5, document
    2's of 1 one of exactly 1; the FP32 logarithms are within 2 ulp, 2.4e-7."""
    a = np.array([0.25, 1.5, 1.0, 0.5, 0.3, 1e-6, 0.9, 0.75, 0.125, 0.6], np.float32)
    cm = _model(a)
    rng = np.random.default_rng(n)
    pidx = np.argsort(rng.random((n, 10)), axis=1).astype(np.int32)
    pidx[::3][pidx[::3] == 1] = -1  # unseen: attractiveness 1/2
    clicks = rng.integers(0, 1024, n).astype(np.uint16)
    clicks |= (((pidx == 1) | (pidx == 2)) @ (1 << np.arange(10))).astype(np.uint16)
    got = _evaluate(cm, pidx, clicks)
    value = np.where(pidx < 0, np.float32(0.5), a[pidx])
    clicked = (clicks[:, None] >> np.arange(10)) & 1
    p = np.where(clicked == 1, value, np.float32(1) - value).astype(np.float64)
    np.testing.assert_allclose(got.llh_sum, np.log(p).sum() / 10, rtol=0, atol=2.4e-7 * np.abs(np.log(p)).sum() / 10)
    np.testing.assert_allclose(got.log2_sums, np.log2(p).sum(0), rtol=0, atol=2.4e-7 * np.abs(np.log2(p)).sum(0).max())


def test_nan_parameters_stay_nan():
    cm = _model([0.5, np.nan, 2.0] + [0.25] * 7)
    got = _evaluate(cm, np.tile(np.arange(10, dtype=np.int32), (50, 1)), np.zeros(50, np.uint16))
    assert np.isnan(got.llh_sum) and np.isnan(got.log2_sums[1:3]).all()
    assert np.isfinite(got.log2_sums[[0] + list(range(3, 10))]).all()
