"""Option factored of a server reaches its FP64 cases: in 3-D it chooses between
the operator in parts and the stored blocks, and a served case gives the bits
of the same setting stepped alone."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine, serving
from mphimplicit_gb300.cabi import PRECISION_FP64

pytestmark = pytest.mark.gpu


def test_served_fp64_case_takes_the_operator_asked_for(engine_lib):
    parts = casegen.dam_case(3, (11, 9, 10), (15, 11, 13), 0.005, seed=4)
    params = casegen.baseline_params(3, 0.005, 5.0e-5)
    alone = {}
    for factored in (1, 0):
        g = engine.Case(params, parts, 3, precision=PRECISION_FP64)
        g.set_option("factored", factored)
        g.step(2)
        alone[factored] = g.fields(("id", "vel"))
        g.close()
    assert not np.array_equal(alone[0]["vel"], alone[1]["vel"])   # two orders of sums
    for factored in (1, 0):
        srv = serving.Server(int(4e9), workers=2)
        srv.set_option("factored", factored)
        srv.submit(params, parts, 3, 2, precision=PRECISION_FP64)
        got = []
        for _ in range(300):
            got += srv.poll(wait_ms=100)
            if got:
                break
        srv.close()
        assert got[0]["status"] == 0, got[0]["error"]
        assert np.array_equal(got[0]["fields"]["id"], alone[factored]["id"])
        assert np.array_equal(got[0]["fields"]["vel"], alone[factored]["vel"])
