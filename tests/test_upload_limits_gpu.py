"""An upload of test sessions that the device cannot hold leaves the model without
test sessions, and usable."""
import ctypes as C

import numpy as np
import pytest

from massiveclicks_gb300 import api, _capi

pytestmark = pytest.mark.gpu


def test_refused_test_sessions():
    docs = np.tile(np.arange(10, dtype=np.int32), (40, 1))
    clicks = np.arange(40).astype(np.uint16)
    sessions = api.SessionSet(np.zeros(40, np.int32), docs, docs, clicks)
    cm = api.DBNModel()
    cm.upload(sessions, 10)
    cm.upload_test(sessions)
    held = cm.memory()
    cm.em(1)
    n = 10**11  # 4 TB of indices: refused before the host's rows are read
    rc = _capi.load().mc_model_upload_test(cm._h, n, docs.ctypes.data_as(C.c_void_p), clicks.ctypes.data_as(C.c_void_p), None)
    assert rc == 4
    assert cm.evaluate(1).n_sessions == 0
    assert np.isfinite(cm.evaluate(0).llh)
    assert cm.memory() < held
    cm.upload_test(sessions)
    assert cm.memory() == held
    np.testing.assert_allclose(cm.evaluate(1).llh, cm.evaluate(0).llh, rtol=1e-12)
