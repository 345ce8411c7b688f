"""FP64 form in 3-D: the operator in parts (pairs in two floats, C Lambda C^T
over the P-lists) against the stored blocks (option factored 0).

Both are FP64 solves of one system to 1e-13, where each is converged to its
rounding (stopped at 1e-10, two solves differ by what the stop leaves, also
those on the blocks of the two assemblies: 5e-11).  They differ by the
rounding of the applications: 2^-46 of a pair part that is at most a tenth of
the inertia, below 2^-49 of a row, grown by at most the condition (1e3):
1e-11 holds the velocities with room.  Cases: one and two fluids of different
density and viscosity with moving walls, a fluid that reaches over the
periodic boundary, row counts beside a slice and a block."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from parity_util import small_cases, vec_proj

pytestmark = pytest.mark.gpu


def _case(name):
    if name in ("cube3d", "surface3d"):
        return next((p, parts) for n, d, p, parts in small_cases() if n == name)
    l0 = 0.005
    fluid, interior = {"small": ((5, 5, 4), (6, 6, 7)), "edge": ((8, 8, 2), (9, 9, 6)), "odd": ((11, 13, 9), (13, 14, 12)),
                       "mixed": ((9, 8, 7), (11, 10, 9)), "wrap": ((9, 8, 7), (11, 10, 9))}[name]
    n = int(np.prod(fluid))
    types = (np.arange(n) % 2).astype(np.int32) if name == "mixed" else None
    parts = casegen.dam_case(3, fluid, interior, l0, seed=4, fluid_types=types)
    p = casegen.baseline_params(3, l0, 5.0e-5)
    if name == "mixed":
        p.density = (1000.0, 300.0, 1000.0, 1000.0)
        p.shear_viscosity = (0.1, 0.02, 0.1, 0.1)
    if name == "wrap":   # the whole arrangement shifted by half a box: the fluid crosses the boundary
        lo, w = parts.domain_min, parts.domain_max - parts.domain_min
        parts.pos = lo + (parts.pos - lo + 0.5 * w) % w
    return p, parts


@pytest.mark.parametrize("name", ["cube3d", "surface3d", "small", "edge", "odd", "mixed", "wrap"])
def test_parts_against_blocks(engine_lib, name):
    params, parts = _case(name)
    out = []
    for factored in (1, 0):
        c = engine.Case(params, parts, 3)
        c.set_option("factored", factored)
        c.set_solver(outer_rel_residual=1e-13)
        c.step(2)
        out.append((c.export("ParticleIndex"), vec_proj(c.export("Velocity"), 3)[:c.fluid_count], c.solve_stats()))
    (ia, va, sa), (ib, vb, sb) = out
    err = float(np.linalg.norm(va - vb) / np.linalg.norm(vb))
    print(name, c.fluid_count, sa["iter"], err)
    assert sa["status"] == 0 and sb["status"] == 0
    assert np.array_equal(ia, ib)
    assert abs(sa["iter"] - sb["iter"]) <= 0.02 * sb["iter"]
    assert err <= 1e-11
