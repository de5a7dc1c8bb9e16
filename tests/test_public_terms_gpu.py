"""Continuation parameters of fits whose documents are all attractive: what
remains after a long unclicked tail, R, is small, and the numerators are sums of
g R h.  One iteration against the FP64 oracle from the same parameters.

R is a recursion of nine steps with two FP32 roundings each, whose relative errors
grow by at most 1 / (1 - g): 9 x 2 x 2^-24 x 10 = 1.1e-5 at g = 0.9, and a term
adds a few roundings of its own."""
import numpy as np
import pytest

from massiveclicks_gb300 import api
from oracle import bindings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [api.DBN, api.CCM])
@pytest.mark.parametrize("clicks", ["first", "any"])
def test_attractive_documents(model, clicks):
    rng = np.random.default_rng(model)
    n, queries, pool = 20000, 100, 30
    query = np.repeat(np.arange(queries, dtype=np.int32), n // queries)
    docs = np.argsort(rng.random((n, pool)), axis=1)[:, :10].astype(np.int32)
    first = 0 if clicks == "first" else rng.integers(0, 4, n)
    train = api.SessionSet(query, docs, query[:, None] * pool + docs, np.full(n, 1, np.uint16) << np.uint16(first))
    cm = api.ClickModel.create(model)
    cm.upload(train, queries * pool)
    values = cm.get_parameters()
    values["attractiveness"][:] = rng.uniform(0.999, 0.9995, queries * pool)
    values["continuation"][:] = 0.9
    if model == api.DBN:
        values["satisfaction"][:] = rng.uniform(0.05, 0.1, queries * pool)
    cm.set_parameters(values)
    cm.em(1)
    f = bindings.OracleFit("f64", model, 0, train.query, train.pidx, train.click, queries * pool)
    f.set_values(values)
    f.run(1)
    np.testing.assert_allclose(cm.get_parameters()["continuation"], f.values()["continuation"], rtol=1.2e-5, atol=0)
