"""The mixed form where two particles are close together: its inner operator
takes C from fixed-point positions, whose rounding turns a close pair's
direction, and leaves the viscous pairs, which grow as 1 / r, to the FP64
residual.  Refined to 1e-10 the velocities must be the FP64 form's on stored
blocks within 1e-8 (the bound of the other inner operators), in about the
iterations of the same particles with none close together (half as many again
at most: a refinement phase more)."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import vec_proj

pytestmark = pytest.mark.gpu


def _case(dim, distance, mu):
    if dim == 2:
        l0, dt, u = 0.01, 1e-4, (0.6, 0.8, 0.0)
        parts = casegen.dam_case(2, (15, 12), (20, 18), l0, seed=3)
    else:
        l0, dt, u = 0.005, 5e-5, (0.48, 0.6, 0.64)
        parts = casegen.dam_case(3, (9, 8, 7), (11, 10, 10), l0, seed=3)
    fl = parts.types < 2
    rng = np.random.default_rng(3)
    parts.vel[fl, :dim] = rng.uniform(-0.02, 0.02, size=(int(fl.sum()), dim))
    a, b = np.argsort(((parts.pos[fl] - parts.pos[fl].mean(axis=0)) ** 2).sum(axis=1))[:2]   # two in the middle
    parts.vel[b] = parts.vel[a]
    parts.pos[b] = parts.pos[a] + distance * l0 * np.array(u)
    return casegen.baseline_params(dim, l0, dt, mu=mu), parts


def _solve(dim, distance, mu, **kw):
    params, parts = _case(dim, distance, mu)
    c = engine.Case(params, parts, dim, **kw)
    if not kw:
        c.set_option("factored", 0)
    c.set_solver(1e-10 if kw else 1e-12, 1e-3, 50)
    c.step(1)
    return vec_proj(c.export("Velocity"), dim)[:c.fluid_count], c.solve_stats()


@pytest.mark.parametrize("distance", [0.3, 0.1, 0.03, 0.015, 0.01, 1e-3, 1e-4, 1e-6])
@pytest.mark.parametrize("dim", [2, 3])
def test_direction(engine_lib, dim, distance):
    """Hardly viscous: what the positions' rounding does."""
    v, s = _solve(dim, distance, 1e-5, precision=PRECISION_MIXED)
    _, apart = _solve(dim, 1.0, 1e-5, precision=PRECISION_MIXED)
    want, f = _solve(dim, distance, 1e-5)
    print(dim, distance, s["iter"], s["outer"], apart["iter"])
    assert s["status"] == 0 and f["status"] == 0
    assert np.linalg.norm(v - want) <= 1e-8 * np.linalg.norm(want)
    assert s["iter"] <= 1.5 * apart["iter"]


@pytest.mark.parametrize("mu", [0.1, 1.0])
@pytest.mark.parametrize("distance", [0.3, 0.1, 0.03, 0.015, 0.01])
@pytest.mark.parametrize("dim", [2, 3])
def test_viscous_pair(engine_lib, dim, distance, mu):
    """A pair that is stiff against the inertia (f / inertia up to 0.1)."""
    v, s = _solve(dim, distance, mu, precision=PRECISION_MIXED)
    _, apart = _solve(dim, 1.0, mu, precision=PRECISION_MIXED)
    want, f = _solve(dim, distance, mu)
    print(dim, distance, mu, s["iter"], s["outer"], apart["iter"])
    assert s["status"] == 0 and f["status"] == 0
    assert np.linalg.norm(v - want) <= 1e-8 * np.linalg.norm(want)
    assert s["iter"] <= 1.5 * apart["iter"]


@pytest.mark.parametrize("dim", [2, 3])
def test_footprint_with_a_close_pair(engine_lib, dim):
    """A step that meets a pair too close for the penalty operator assembles the
    pair terms beside what that operator had: the admission bound holds both."""
    torch = pytest.importorskip("torch")
    from mphimplicit_gb300 import serving
    torch.cuda.init()
    l0, dt = (0.01, 1e-4) if dim == 2 else (0.005, 5e-5)
    parts = casegen.dam_case(dim, (100, 100) if dim == 2 else (30, 30, 30), (120, 110) if dim == 2 else (33, 33, 33), l0, seed=3)
    params = casegen.baseline_params(dim, l0, dt)
    parts.pos[1] = parts.pos[0] + 1e-3 * l0 * np.array([0.6, 0.8, 0.0])
    fp = serving.footprint(params, parts, dim, PRECISION_MIXED)
    free0, _ = torch.cuda.mem_get_info()
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(1e-10, 1e-3, 50)
    g.step(2)
    free1, _ = torch.cuda.mem_get_info()
    s = g.solve_stats()
    g.close()
    print(dim, free0 - free1, fp)
    assert s["inner_kernel"] == 0
    assert free0 - free1 <= fp
