"""The frame fields of cases with surface tension (the pressure-A and
diffuse-interface terms of the virial, and the forces), 2D and 3D, against
the oracle: the kernel forms every pair's virial as one factor times
q (x) q, the reference term by term.  Once after a whole step and once after
its explicit stage, before any solve.

Tolerances: the fields are linear in the solved velocities, which two solves
stopped at 1e-6 share to 2e-5; before a solve only FP64 rounding of sums of
at most some 200 terms is left, below 1e-11 of the field's largest value."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from parity_util import rel, small_cases, vec_proj

pytestmark = pytest.mark.gpu

CASES = [c for c in small_cases() if c[0].startswith("surface")]
# two fluids spanning several cells an axis, so that blocks of 128 particles end inside a cell
_p = casegen.baseline_params(3, 0.005, 5.0e-5)
_p.surface_tension = (0.072, 0.03, 0.0, 0.0)
_p.interaction_ratio = ((1.0, 0.8, 1.0, 1.0), (0.9, 1.0, 0.7, 1.0), (1.0,) * 4, (1.0,) * 4)
CASES.append(("surface3d_9", 3, _p, casegen.dam_case(3, (9, 8, 11), (12, 11, 14), 0.005, seed=6,
                                                     fluid_types=(np.arange(9 * 8 * 11) % 2).astype(np.int32))))
FIELDS = ("DivergenceP", "PressureP", "VirialPressureAtParticle")


@pytest.mark.parametrize("steps", [0, 1])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_frame_fields_with_surface_tension(engine_lib, oracle_built, case, steps):
    name, dim, params, parts = case
    parts = casegen.Particles(parts.time, parts.spacing, parts.domain_min, parts.domain_max, parts.types, parts.pos,
                              parts.vel.copy())
    rng = np.random.default_rng(1)
    fl = parts.types < 2
    parts.vel[fl, :dim] = rng.uniform(-0.05, 0.05, size=(int(fl.sum()), dim))
    o = oracle_built.Oracle(params, parts, dim, threads=1)
    o.init()
    g = engine.Case(params, parts, dim)
    if steps:
        o.step(steps)
        g.step(steps)
    else:
        o.step_begin(); o.cellsort(); o.neighbors(); o.explicit()
        for st in ("step_begin", "cellsort", "neighbors", "explicit"):
            g.stage(st)
    o.output_fields()
    g.stage("output_fields")
    tol = 2e-5 if steps else 1e-11
    for n in FIELDS:
        assert rel(g.export(n), o.array(n)) <= tol, n
    assert rel(vec_proj(g.export("Force"), dim), vec_proj(o.array("Force"), dim)) <= tol
    assert rel(g.export("VolStrainP"), o.array("VolStrainP")) <= 1e-13


def test_frame_without_surface_tension_needs_no_density_pass(engine_lib, oracle_built):
    """Without surface tension the frame forms no DensityA; a reader that asks
    for it afterwards gets it, and VolStrainP keeps its bits."""
    name, dim, params, parts = small_cases()[2]
    o = oracle_built.Oracle(params, parts, dim, threads=1)
    o.init()
    o.step(1)
    o.output_fields()
    g = engine.Case(params, parts, dim)
    g.step(1)
    g.stage("output_fields")
    assert rel(g.export("VolStrainP"), o.array("VolStrainP")) <= 1e-13
    assert rel(g.export("DensityA"), o.array("DensityA")) <= 1e-13
    assert rel(g.export("VirialPressureAtParticle"), o.array("VirialPressureAtParticle")) <= 2e-5
