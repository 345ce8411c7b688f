"""FP64 form: the small multigrid levels applied as one matrix, against the
oracle's level by level V-cycle (main.cpp:3243-3546).

(b, M b) and (r, M r) are what one V-cycle gives; the oracle's system agrees
with the engine's to 1e-11 (the parity tests' bound), and M is applied to it
linearly, so 1e-10 holds it.  Sizes: the matrix from level 0 on, from level 1
on with one and with several blocks of rows, from level 2 on (3-D), long
grids, odd cell counts; and the sort's network at the edges of its tiles, on
the same particles (the permutation is bit for bit the reference's)."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine

pytestmark = pytest.mark.gpu

# (dim, fluid lattice, interior lattice): particles with their walls cross
# 2^11 .. 2^14, the tile being 2^12
CASES = [(2, (7, 7), (10, 9)), (2, (41, 33), (50, 40)), (2, (83, 30), (90, 33)), (2, (160, 7), (170, 12)),
         (2, (78, 78), (82, 80)), (3, (9, 8, 7), (10, 9, 9)), (3, (25, 9, 8), (27, 10, 9)), (3, (16, 17, 15), (17, 18, 18))]


@pytest.mark.parametrize("dim,fluid,interior", CASES, ids=["x".join(map(str, c[1])) for c in CASES])
def test_tail_matrix_and_sort(engine_lib, oracle_built, dim, fluid, interior):
    l0 = 0.01 if dim == 2 else 0.005
    parts = casegen.dam_case(dim, fluid, interior, l0, seed=2)
    params = casegen.baseline_params(dim, l0, 1.0e-4 if dim == 2 else 5.0e-5)
    o = oracle_built.Oracle(params, parts, dim, threads=8)
    o.init()
    g = engine.Case(params, parts, dim)
    o.step_begin(); g.stage("step_begin")
    o.cellsort(); g.stage("cellsort")
    for n in ("CellIndex", "CellParticle", "ParticleIndex"):
        assert np.array_equal(g.export(n), o.array(n)), n
    o.neighbors(); g.stage("neighbors")
    for n in ("NeighborPtr", "NeighborPtrP"):
        assert np.array_equal(g.export(n), o.array(n)), n
    o.explicit(); o.assemble(); o.mg_build(); o.solve()
    for st in ("explicit", "assemble", "mg_build", "solve"):
        g.stage(st)
    so, sg = o.solve_stats(), g.solve_stats()
    print(parts.count, sg["iter"], sg["rs0"] / so["rs0"] - 1.0)
    assert abs(sg["rs0"] / so["rs0"] - 1.0) <= 1e-10
    assert abs(sg["iter"] - so["iter"]) <= 1
