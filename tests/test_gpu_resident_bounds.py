"""The resident CR iteration's bounds: a launch that ends at its iteration bound
is followed by another that goes on with the solve, and a grid barrier whose
wait runs out ends the solve with an error status, after which the same case
steps as a new one does."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import vec_proj

pytestmark = pytest.mark.gpu


def _case(dim):
    if dim == 2:
        parts = casegen.dam_case(2, (61, 43), (80, 60), 0.01, seed=1)
        params = casegen.baseline_params(2, 0.01, 1.0e-4)
    else:
        parts = casegen.dam_case(3, (13, 11, 12), (20, 14, 15), 0.005, seed=4)
        params = casegen.baseline_params(3, 0.005, 5.0e-5)
    fl = parts.types < 2
    parts.vel[fl, :dim] = np.random.default_rng(9).uniform(-0.02, 0.02, size=(int(fl.sum()), dim))
    return params, parts


def _new(dim, **options):
    params, parts = _case(dim)
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(1e-10, 1e-3, 50)
    for k, v in options.items():
        g.set_option(k, v)
    return g, parts


@pytest.mark.parametrize("bound", [40, 16, 5])
@pytest.mark.parametrize("dim", [2, 3])
def test_launch_bound(engine_lib, dim, bound):
    """The directions carry on from launch to launch while the FP64 residual
    replaces the recursive one, as between phases, so a bounded launch costs
    no iterations beyond a few and the solve ends at the same tolerance (1e-8
    of the velocities, as the other forms' tests)."""
    a, _ = _new(dim)
    b, _ = _new(dim, launch_iterations=bound)
    a.step(1)
    b.step(1)
    sa, sb = a.solve_stats(), b.solve_stats()
    print(dim, bound, sa["iter"], sa["outer"], sb["iter"], sb["outer"])
    assert sa["status"] == 0 and sb["status"] == 0 and sb["rr"] / sb["rr0"] < 1e-20
    va, vb = (vec_proj(c.export("Velocity"), dim)[:c.fluid_count] for c in (a, b))
    assert np.linalg.norm(vb - va) <= 1e-8 * np.linalg.norm(va)
    assert sb["iter"] <= 1.1 * sa["iter"] + 5


@pytest.mark.parametrize("dim", [2, 3])
def test_wait_runs_out(engine_lib, dim):
    """One poll a wait: a block that arrives before the others gives up, every
    block leaves, the step fails with a status that the host reads, and the
    case given its state again steps to a new case's bits."""
    g, parts = _new(dim, wait_polls=1)
    with pytest.raises(engine.MphError) as e:
        g.step(1)
    assert "barrier" in str(e.value)
    g.set_option("wait_polls", 1 << 21)
    g.set_state(parts)
    h, _ = _new(dim)
    h.set_state(parts)
    for _ in range(2):
        g.step(1)
        h.step(1)
        assert g.solve_stats()["status"] == 0
    assert np.array_equal(g.export("ParticleIndex"), h.export("ParticleIndex"))
    assert np.array_equal(g.export("Velocity"), h.export("Velocity"))


def test_bounds_are_checked(engine_lib):
    g, _ = _new(2)
    for name, value in (("launch_iterations", 0), ("launch_iterations", 4097), ("launch_iterations", 2.5), ("wait_polls", 0),
                        ("wait_polls", float("nan")), ("wait_polls", 2097153)):
        with pytest.raises(engine.MphError) as e:
            g.set_option(name, value)
        assert e.value.status == 1
