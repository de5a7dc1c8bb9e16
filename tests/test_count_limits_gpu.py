"""The count kernels with parameters at 1, as a caller may set them: a rank at
which a pair has no unclicked occurrence adds nothing, even where 1 - a e is 0.
One iteration against the FP64 oracle from the same parameters, with the
tolerances of the other EM tests."""
import numpy as np
import pytest

from massiveclicks_gb300 import api
from oracle import bindings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [45, 2000, 70000])  # PBM counts in bytes, in 16 bits, and beyond the dense table
@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("model", [api.PBM, api.UBM])
def test_certain_clicks(model, batched, n):
    """Document 0 is attractive for certain; it is clicked at rank 0, whose
    examination is certain too, and passed over at rank 1 now and then."""
    docs = np.tile(np.arange(10, dtype=np.int32), (n, 1))
    clicks = np.full(n, 1, np.uint16)
    docs[3::5, :2] = [1, 0]
    clicks[3::5] = 0
    clicks[::7] |= 1 << 4
    train = api.SessionSet(np.zeros(n, np.int32), docs, docs, clicks)
    cm = api.ClickModel.create(model)
    cm.upload(train, 10)
    assert cm.fused_path()[0] == ("dense" if model == api.PBM and n < 65536 else "counts")
    values = cm.get_parameters()
    values["examination"][:] = np.linspace(0.3, 0.7, len(values["examination"]))
    # rank 0; for UBM its slot, and the first of the table, which no rank has
    values["examination"][[0, 9] if model == api.UBM else [0]] = 1.0
    values["attractiveness"][0] = 1.0
    cm.set_parameters(values)
    if batched:
        batch = api.Batch([cm])
        batch.em(1)
        batch.close()
    else:
        cm.em(1)
    f = bindings.OracleFit("f64", model, 0, train.query, train.pidx, train.click, 10)
    f.set_values(values)
    f.run(1)
    got = cm.get_parameters()
    for name, ref in f.values().items():
        np.testing.assert_allclose(got[name], ref, rtol=1e-5, atol=1e-6, err_msg=name)
