"""The stage entry points between which a caller sets options or reads arrays:
what a step's assembly built decides what its solve runs on, and an array is
read from the step it belongs to or refused."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED

pytestmark = pytest.mark.gpu

BEFORE_SOLVE = ("step_begin", "cellsort", "neighbors", "explicit", "assemble", "mg_build")


def _parts(dim, seed=4):
    if dim == 2:
        parts = casegen.dam_case(2, (23, 17), (40, 26), 0.01, seed=seed)
        params = casegen.baseline_params(2, 0.01, 1.0e-4)
    else:
        parts = casegen.dam_case(3, (11, 9, 10), (15, 11, 13), 0.005, seed=seed)
        params = casegen.baseline_params(3, 0.005, 5.0e-5)
    fl = parts.types < 2
    parts.vel[fl, :dim] = np.random.default_rng(seed).uniform(-0.05, 0.05, size=(int(fl.sum()), dim))
    return params, parts


def _mixed(params, parts, dim):
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(1e-10, 1e-3, 50)
    return g


@pytest.mark.parametrize("at_assembly", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_staging_is_the_assemblys(engine_lib, dim, at_assembly):
    """Option inner_local set between the assembly and the solve: the solve
    runs on what the assembly built (staged and gathering blocks give the same
    bits), and the new setting acts from the next step on."""
    params, parts = _parts(dim)
    a, b = _mixed(params, parts, dim), _mixed(params, parts, dim)
    b.step(1)
    a.set_option("inner_local", at_assembly)
    for s in BEFORE_SOLVE:
        a.stage(s)
    a.set_option("inner_local", 1 - at_assembly)
    a.stage("solve")
    a.stage("step_end")
    for want in (at_assembly, 1 - at_assembly):
        assert (a.solve_stats()["inner_local_blocks"] > 0) == bool(want)
        assert np.array_equal(a.export("Velocity"), b.export("Velocity"))
        a.step(1)
        b.step(1)
