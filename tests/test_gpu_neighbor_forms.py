"""The cell-bucket neighbour search's block forms: small blocks in 2-D up to 32
particles a cell, large ones beyond and in 3-D, per-thread walks where a pass
has more candidates than a block has room for (1536).  The lists are the
oracle's bit for bit with each, for walls and fluid, wide radii and packed
fluids, walks that wrap and walks that do not."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine

pytestmark = pytest.mark.gpu

# (dim, fluid lattice, interior lattice, radius ratio of A and V, packing, shift by half a box)
CASES = [(2, (48, 48), (60, 60), 4.5, 1.0, True), (2, (48, 48), (60, 60), 5.6, 1.0, False), (2, (48, 48), (60, 60), 8.5, 1.0, False), (2, (48, 48), (60, 60), 12.0, 1.0, True), (2, (90, 50), (100, 60), 15.5, 1.0, False),
         (3, (14, 13, 12), (16, 15, 14), 3.5, 1.25, False), (3, (14, 13, 12), (16, 15, 14), 3.5, 1.7, True),
         (3, (17, 16, 15), (19, 18, 17), 5.5, 1.0, False)]


@pytest.mark.parametrize("dim,fluid,interior,ratio,pack,shift", CASES)
def test_lists_of_every_form(engine_lib, oracle_built, dim, fluid, interior, ratio, pack, shift):
    l0 = 0.01 if dim == 2 else 0.005
    parts = casegen.dam_case(dim, fluid, interior, l0, seed=6)
    params = casegen.baseline_params(dim, l0, 1.0e-4 if dim == 2 else 5.0e-5)
    params.radius_ratio_a = params.radius_ratio_v = ratio
    fl = parts.types < 2
    c = parts.pos[fl].mean(axis=0)
    parts.pos[fl] = c + (parts.pos[fl] - c) / pack
    room = 4 * ratio * l0                       # a grid of several cells an axis around the walls
    parts.domain_min[:dim] -= room
    parts.domain_max[:dim] += room
    if shift:
        lo, w = parts.domain_min[:dim], (parts.domain_max - parts.domain_min)[:dim]
        parts.pos[:, :dim] = lo + (parts.pos[:, :dim] - lo + 0.5 * w) % w
    o = oracle_built.Oracle(params, parts, dim, threads=8)
    o.init()
    g = engine.Case(params, parts, dim)
    cells = g.export("CellIndex")[:parts.count]
    print(parts.count, np.bincount(cells).max(), g.export("NeighborCount").max())
    for n in ("NeighborCount", "NeighborFluidCount", "NeighborCountP", "NeighborPtr", "NeighborInd", "NeighborPtrP", "NeighborIndP"):
        assert np.array_equal(g.export(n), o.array(n)), n
