"""The inner operator of the point-Jacobi mixed form (k_penalty.cu): inertia
and C Lambda C^T from the P-lists, C evaluated from fixed-point positions, the
viscous pairs left to the FP64 outer residual.

Refined to 1e-10 the velocity must be the FP64 form's solved to 1e-12 within
1e-8 (the bound the other inner operators are held to), whatever form and block
shape the particle count selects (all iterations of a phase in one resident
kernel, or a kernel each for lists too long for its shared memory and beyond
155,648 particles, with remainders), with periodic images in the lists, and where the fluid is viscous enough for
the part left out to set the refinement's pace; and every block gathering by
column must give the bits of the staged blocks."""
import numpy as np
import pytest

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import vec_proj

pytestmark = pytest.mark.gpu


def _periodic(dim, n, l0, seed):
    """Fluid filling a periodic box of n cells an axis: every face couples to the opposite one."""
    rng = np.random.default_rng(seed)
    ax = [(np.arange(k) + 0.5) * l0 for k in n] + [np.zeros(1)] * (3 - dim)
    pos = np.stack([g.ravel() for g in np.meshgrid(*ax, indexing="ij")], axis=1)
    pos[:, :dim] += rng.uniform(-0.02 * l0, 0.02 * l0, size=(len(pos), dim))
    hi = np.array([k * l0 for k in n] + [0.5 * l0] * (3 - dim))
    lo = np.array([0.0] * dim + [-0.5 * l0] * (3 - dim))
    return casegen.Particles(0.0, l0, lo, hi, np.zeros(len(pos), np.int32), pos, np.zeros_like(pos))


def _cases():
    out = []
    for name, dim, parts, mu in (
            ("resident-2d-small", 2, casegen.dam_case(2, (41, 33), (80, 50), 0.01, seed=1), 0.1),
            ("resident-2d", 2, casegen.dam_case(2, (171, 163), (340, 200), 0.01, seed=2), 0.3),
            ("resident-2d-wide-blocks", 2, casegen.dam_case(2, (281, 277), (500, 320), 0.01, seed=3), 0.1),
            ("beyond-resident-2d", 2, casegen.dam_case(2, (417, 373), (600, 420), 0.01, seed=10), 0.1),
            ("resident-3d-small", 3, casegen.dam_case(3, (13, 11, 12), (20, 14, 15), 0.005, seed=4), 0.1),
            ("resident-3d", 3, casegen.dam_case(3, (27, 25, 24), (40, 29, 28), 0.005, seed=5), 0.1),
            ("long-lists-3d", 3, casegen.dam_case(3, (12, 13, 12), (16, 15, 15), 0.005, seed=11), 0.1),
            ("viscous-3d", 3, casegen.dam_case(3, (13, 11, 12), (20, 14, 15), 0.005, seed=6), 1.5),
            ("periodic-2d", 2, _periodic(2, (23, 17), 0.01, 7), 0.1),
            ("periodic-3d", 3, _periodic(3, (15, 12, 13), 0.005, 8), 0.1)):
        l0, dt = (0.01, 1e-4) if dim == 2 else (0.005, 5e-5)
        params = casegen.baseline_params(dim, l0, dt, mu=mu)
        if name.startswith("long-lists"):   # some 380 P-neighbours a row
            params.radius_ratio_a, params.radius_ratio_p, params.radius_ratio_v = 9.4, 4.5, 9.4
            parts.domain_min[:] -= 8 * l0
            parts.domain_max[:] += 8 * l0
        fl = parts.types < 2
        rng = np.random.default_rng(9)
        parts.vel[fl, :dim] = rng.uniform(-0.02, 0.02, size=(int(fl.sum()), dim))
        out.append((name, dim, params, parts))
    return out


CASES = _cases()


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_solution_and_staging(engine_lib, case):
    name, dim, params, parts = case
    got = {}
    for local in (1, 0):
        g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
        g.set_solver(1e-10, 1e-3, 50)
        g.set_option("inner_local", local)
        g.step(1)
        s = g.solve_stats()
        assert s["status"] == 0 and s["inner_form"] == 2 and s["rr"] / s["rr0"] < 1e-20
        # (64 rows of the long lists have more distinct neighbours than a block stages)
        assert (s["inner_local_blocks"] > 0) == (local == 1 and not name.startswith("long-lists"))
        got[local] = (g.export("ParticleIndex"), g.export("Velocity"), s["iter"], s["outer"])
    assert np.array_equal(got[1][1], got[0][1]) and got[1][2:] == got[0][2:]
    f = engine.Case(params, parts, dim)
    f.set_solver(1e-12, 1e-3, 50)
    f.step(1)
    assert np.array_equal(f.export("ParticleIndex"), got[1][0])
    nf = f.fluid_count
    vf, vm = vec_proj(f.export("Velocity"), dim)[:nf], vec_proj(got[1][1], dim)[:nf]
    err = float(np.linalg.norm(vm - vf) / np.linalg.norm(vf))
    print(f"{name}: {got[1][2]} iterations, {got[1][3]} phases, velocity {err:.1e} from the FP64 form at 1e-12")
    assert err <= 1e-8
