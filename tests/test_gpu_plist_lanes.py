"""P-list passes with one and with four threads a row (the line lies at 65,536
particles): density, source vector, right-hand side and C against the oracle,
beside the line on either side in 2-D and 3-D, and the mixed solve refined to
1e-10 in the oracle's own system.

FP64 sums of some twenty terms in another order: the parity tests' bounds for
the same arrays, 1e-12 for the density and 1e-11 for p and b."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import rel, vec_proj

pytestmark = pytest.mark.gpu

CASES = [(3, (32, 32, 30), (49, 36, 38)), (3, (33, 33, 31), (41, 37, 39)), (2, (320, 193), (350, 233)), (2, (320, 194), (350, 234))]


@pytest.mark.parametrize("dim,fluid,interior", CASES, ids=["x".join(map(str, c[1])) for c in CASES])
def test_lanes(engine_lib, oracle_built, dim, fluid, interior):
    parts = casegen.dam_case(dim, fluid, interior, 0.005 if dim == 3 else 0.01, seed=3)
    params = casegen.baseline_params(dim, 0.005 if dim == 3 else 0.01, 5.0e-5 if dim == 3 else 1.0e-4)
    o = oracle_built.Oracle(params, parts, dim, threads=8)
    o.init()
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(outer_rel_residual=1e-10)
    for st in ("step_begin", "cellsort", "neighbors", "explicit", "assemble"):
        getattr(o, st)()
        g.stage(st)
    nf = g.fluid_count
    print(parts.count, nf)
    assert rel(g.export("VolStrainP"), o.array("VolStrainP")) <= 1e-12
    assert rel(g.export("VectorP"), o.array("VectorP")) <= 1e-11
    assert rel(g.export("VectorB"), vec_proj(o.array("VectorB"), dim).ravel()) <= 1e-11
    g.stage("mg_build")
    g.stage("solve")
    assert g.solve_stats()["status"] == 0
    ptr, ind, val = o.array("CsrPtrA"), o.array("CsrIndA"), o.array("CsrCofA")
    x = np.zeros((nf, 3))
    x[:, :dim] = vec_proj(g.export("Velocity"), dim)[:nf]
    rows = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))
    b = o.array("VectorB")[:3 * nf]
    r = b - np.bincount(rows, weights=val * x.ravel()[ind], minlength=len(ptr) - 1)
    # 1e-10 of the engine's own residual and the FP32 pair coefficients (6e-10
    # of the operator), as the parity tests of the mixed form hold it
    assert np.linalg.norm(r) <= 1e-9 * np.linalg.norm(b)
