"""2-D cell-bucket neighbour search around its shared-memory capacity (512
candidates a pass, 256 particles a bucket): a fluid packed to a fraction of
its spacing, so that the cells' walks hold fewer, about as many and more
candidates; the lists are the oracle's bit for bit on both paths."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pack", [1.0, 2.0, 2.4, 2.6, 4.0, 6.0])
def test_packed_2d_lists(engine_lib, oracle_built, pack):
    parts = casegen.dam_case(2, (48, 48), (60, 60), 0.01, seed=6)
    fluid = parts.types < 2
    c = parts.pos[fluid].mean(axis=0)
    parts.pos[fluid] = c + (parts.pos[fluid] - c) / pack
    params = casegen.baseline_params(2, 0.01, 1.0e-4)
    o = oracle_built.Oracle(params, parts, 2, threads=4)
    o.init()
    g = engine.Case(params, parts, 2)
    for n in ("NeighborCount", "NeighborFluidCount", "NeighborCountP", "NeighborPtr", "NeighborInd", "NeighborPtrP", "NeighborIndP"):
        assert np.array_equal(g.export(n), o.array(n)), n
