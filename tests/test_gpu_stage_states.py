"""The stage entry points between which a caller sets options or reads arrays:
what a step's assembly built decides what its solve runs on, and an array is
read from the step it belongs to or refused."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import csr_blocks_oracle, rel

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


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_levels_are_the_assemblys(engine_lib, dim, pairs):
    """Option mg_depth set to 0 between an assembly without multigrid levels
    and the solve: the step keeps point Jacobi (levels would be built from
    stencils that the assembly did not write), the next one has its levels.
    pairs: the pair-term operator (two particles close together)."""
    params, parts = _parts(dim)
    if pairs:
        parts.pos[1] = parts.pos[0] + 1e-3 * parts.spacing * np.array([0.6, 0.8, 0.0])
        parts.vel[1] = parts.vel[0]
    a, b = _mixed(params, parts, dim), _mixed(params, parts, dim)
    for s in BEFORE_SOLVE[:5]:
        a.stage(s)
    a.set_option("mg_depth", 0)
    for s in ("mg_build", "solve"):
        a.stage(s)
    with pytest.raises(engine.MphError):
        a.export("MultiGridCsrCofA:0")
    a.stage("step_end")
    b.step(1)
    assert a.solve_stats()["status"] == 0
    assert np.array_equal(a.export("Velocity"), b.export("Velocity"))
    a.step(1)
    assert a.solve_stats()["status"] == 0 and len(a.export("MultiGridCsrCofA:0")) > 0


@pytest.mark.parametrize("dim", [2, 3])
def test_c_of_the_mixed_form(engine_lib, oracle_built, dim):
    """C as the point-Jacobi mixed form's assembly writes it with four threads
    a row, own slots (the sum of a row's others) included, against the
    oracle's, to the bound of the FP64 form's parity tests."""
    params, parts = _parts(dim)
    o = oracle_built.Oracle(params, parts, dim, threads=1)
    o.init()
    g = _mixed(params, parts, dim)
    for s in BEFORE_SOLVE[:5]:
        getattr(o, s)()
        g.stage(s)
    want = csr_blocks_oracle(o.array("CsrPtrC"), o.array("CsrCofC"), g.fluid_count, g.export("NeighborCountP"), dim, per_block=False)
    assert rel(g.export("CsrCofC"), want) <= 1e-12


@pytest.mark.parametrize("dim", [2, 3])
def test_diagonal_is_of_its_step_or_refused(engine_lib, dim):
    """InvDiagA of the point-Jacobi form is formed when it is read, from the
    step's lists and C: the same values from the assembly to the end of the
    step, and refused where positions or lists are newer (a later step's first
    stages, a new state)."""
    params, parts = _parts(dim)
    g = _mixed(params, parts, dim)
    for s in BEFORE_SOLVE[:5]:
        g.stage(s)
    want = g.export("InvDiagA")
    for s in ("mg_build", "solve", "step_end"):
        g.stage(s)
        assert np.array_equal(g.export("InvDiagA"), want), s
    for s in BEFORE_SOLVE[:4]:
        g.stage(s)
        with pytest.raises(engine.MphError) as e:
            g.export("InvDiagA")
        assert e.value.status == 9, s
    g.stage("assemble")
    assert len(g.export("InvDiagA")) == len(want)
    g.set_state(parts)
    with pytest.raises(engine.MphError):
        g.export("InvDiagA")


@pytest.mark.parametrize("dim", [2, 3])
def test_reading_the_density_changes_nothing(engine_lib, dim):
    """Without surface tension DensityA, GravityCenter and PressureA are formed
    when they are read; VolStrainP and the step's result keep their bits."""
    params, parts = _parts(dim)
    a, b = engine.Case(params, parts, dim), engine.Case(params, parts, dim)
    first = a.export("VolStrainP")
    a.export("DensityA")
    a.stage("output_fields")
    assert np.array_equal(a.export("VolStrainP"), first)
    for s in BEFORE_SOLVE[:4]:
        a.stage(s)
        b.stage(s)
    vsp = a.export("VolStrainP")
    for n in ("DensityA", "GravityCenter", "PressureA"):
        a.export(n)
    assert np.array_equal(a.export("VolStrainP"), vsp)
    for s in ("assemble", "mg_build", "solve", "step_end", "output_fields"):
        a.stage(s)
        b.stage(s)
    for n in ("VectorB", "Velocity", "VolStrainP", "PressureP"):
        assert np.array_equal(a.export(n), b.export(n)), n
