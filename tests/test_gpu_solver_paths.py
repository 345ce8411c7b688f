"""The mixed solve's ways beside the resident kernel, on cases that take them
(solve_stats()["inner_kernel"] says which): a kernel each for the parts of an
iteration (lists too long for the resident kernel, some staged and some
gathered, and a case beyond its particle count) replayed as graphs or launched
directly, with any chunk, driven by the device, and together with other cases;
and the pair-term operator (mg_depth 0, or particles too close together) with
its record formats, block widths and fused slicing.

What runs the same kernels in the same order gives the same bits; what sums in
another order or rounds the inner operator otherwise agrees within the
refinement's tolerance (1e-10, velocities to 1e-8 as the other forms' tests)."""
import numpy as np
import pytest

from mphimplicit_gb300 import autotune, casegen, engine, serving
from mphimplicit_gb300.cabi import PRECISION_MIXED
from parity_util import rel, small_cases, vec_proj

pytestmark = pytest.mark.gpu


def _start(params, parts, dim, seed=9):
    fl = parts.types < 2
    parts.vel[fl, :dim] = np.random.default_rng(seed).uniform(-0.02, 0.02, size=(int(fl.sum()), dim))
    return dim, params, parts


def _long2(n, seed):
    """Some 95 P-neighbours a row in 2-D."""
    parts = casegen.dam_case(2, n, (n[0] + 20, n[1] + 8), 0.01, seed=seed)
    params = casegen.baseline_params(2, 0.01, 1.0e-4)
    params.radius_ratio_a = params.radius_ratio_v = 11.5
    params.radius_ratio_p = 5.5
    parts.domain_min[:2] -= 0.25
    parts.domain_max[:2] += 0.25
    return _start(params, parts, 2)


def _long3(n, seed):
    """Some 380 in 3-D."""
    parts = casegen.dam_case(3, n, tuple(k + 4 for k in n), 0.005, seed=seed)
    params = casegen.baseline_params(3, 0.005, 5.0e-5)
    params.radius_ratio_a, params.radius_ratio_p, params.radius_ratio_v = 9.4, 4.5, 9.4
    parts.domain_min[:] -= 0.04
    parts.domain_max[:] += 0.04
    return _start(params, parts, 3)


def _beyond():
    return _start(casegen.baseline_params(2, 0.01, 1.0e-4), casegen.dam_case(2, (417, 373), (600, 420), 0.01, seed=10), 2)


def _long2_close():
    """With two particles whose viscous pair sets the phases' target, a new one every step."""
    dim, params, parts = _long2((61, 53), 1)
    params.shear_viscosity = (20.0, 20.0, 20.0, 20.0)
    a, b = 30 * 53 + 20, 30 * 53 + 21
    parts.pos[b] = parts.pos[a] + 0.06 * parts.spacing * np.array([0.6, 0.8, 0.0])
    parts.vel[b] = parts.vel[a] + np.array([3.0, 4.0, 0.0])
    return dim, params, parts


ITERATED = {"long2d": lambda: _long2((61, 53), 1), "close2d": _long2_close, "long3d": lambda: _long3((12, 13, 12), 11), "beyond2d": _beyond}


def _run(case, options, steps=2):
    dim, params, parts = case
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(1e-10, 1e-3, 50)
    g.set_option("extrapolate", 2)
    for k, v in options.items():
        g.set_option(k, v)
    stats, l0 = [], engine.launch_count()
    for _ in range(steps):
        g.step(1)
        s = g.solve_stats()
        assert s["status"] == 0
        stats.append((s["iter"], s["outer"], s["rr"], s["rr0"]))
    launches = engine.launch_count() - l0
    return g.fields(("id", "pos", "vel")), stats, s, launches


def _same(a, b):
    assert a[1] == b[1]
    for k in ("id", "pos", "vel"):
        assert np.array_equal(a[0][k], b[0][k]), k


@pytest.mark.parametrize("options", [{"graphs": 0}, {"chunk": 32}, {"chunk": 4}, {"device_loop": 1}, {"inner_local": 0}],
                         ids=["direct", "chunk32", "chunk4", "device", "gather"])
@pytest.mark.parametrize("name", list(ITERATED))
def test_iterated_kernels(engine_lib, name, options):
    case = ITERATED[name]()
    a, b = _run(case, {}), _run(case, options)
    print(name, options, a[1], a[3], b[3], a[2]["inner_local_blocks"], a[2]["inner_gather_blocks"])
    assert a[2]["inner_kernel"] == b[2]["inner_kernel"] == 1
    _same(a, b)
    if "device_loop" in options:   # the device stops at the iteration; the host's chunks run on to their end
        assert a[3] != b[3]


def test_iterated_kernels_over_a_batch(engine_lib):
    """Option batch_solve: groups of one dimension and block shape, cases that
    finish at different times, and resident cases that solve on their own."""
    made = [_long2((61, 53), 1), _long2((37, 29), 2), _long2((23, 40), 3), _long3((12, 13, 12), 11), _long3((14, 12, 13), 12)]
    made += [(dim, params, parts) for _, dim, params, parts in small_cases()]
    runs = {}
    for on in (0, 1):
        cases = []
        for dim, params, parts in made:
            g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
            g.set_solver(1e-10, 1e-3, 50)
            g.set_option("extrapolate", 2)
            g.set_option("batch_solve", on)
            cases.append(g)
        l0 = engine.launch_count()
        assert serving.batch_step(cases, 3) == 0
        runs[on] = [(g.fields(("id", "pos", "vel")), g.solve_stats()) for g in cases], engine.launch_count() - l0
        for g in cases:
            g.close()
    assert [s["inner_kernel"] for _, s in runs[1][0]] == [1] * 5 + [2] * 4
    assert runs[1][1] < runs[0][1]      # shared launches
    for (fa, sa), (fb, sb) in zip(runs[0][0], runs[1][0]):
        assert sa == sb
        for k in ("id", "pos", "vel"):
            assert np.array_equal(fa[k], fb[k]), k


FORMATS = {"fp16": {"pair_pack": 0}, "pack": {}, "recompute": {"pair_recompute": 1}}


def _pairs(name):
    """(dim, params, particles), options: a case on the pair-term operator."""
    dim, params, parts = next((d, p, q) for n, d, p, q in small_cases() if n == name.split("-")[0])
    if name.endswith("-close"):     # point Jacobi: two particles closer than MaxRadius / 256
        parts.pos[1] = parts.pos[0] + 5e-3 * parts.spacing * np.array([0.6, 0.8, 0.0])
        return (dim, params, parts), {}
    return (dim, params, parts), {"mg_depth": 0}


PAIRS = ["dam2d", "surface2d", "cube3d", "surface3d", "dam2d-close", "cube3d-close"]


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("name", PAIRS)
def test_pair_formats_staged_and_gathered(engine_lib, name, fmt):
    case, opts = _pairs(name)
    opts, steps = {**opts, **FORMATS[fmt]}, 1 if name.endswith("-close") else 2
    a, b = _run(case, opts, steps), _run(case, {**opts, "inner_local": 0}, steps)
    assert a[2]["inner_kernel"] == b[2]["inner_kernel"] == 0 and a[2]["inner_form"] == 2
    assert a[2]["inner_local_blocks"] > 0 and b[2]["inner_local_blocks"] == 0
    _same(a, b)


@pytest.mark.parametrize("options", [{"pair_pack": 0}, {"pair_recompute": 1}, {"pair_block": 128}, {"pair_block": 256, "ct_block": 128},
                                     {"split_apply": 1}, {"device_loop": 1}, {"chunk": 32}],
                         ids=["fp16", "recompute", "pb128", "pb256-ct128", "split", "device", "chunk32"])
@pytest.mark.parametrize("name", PAIRS)
def test_pair_options_reach_the_same_solution(engine_lib, name, options):
    case, opts = _pairs(name)
    a, b = _run(case, opts, 1), _run(case, {**opts, **options}, 1)
    assert a[2]["inner_kernel"] == b[2]["inner_kernel"] == 0
    if "device_loop" in options or "chunk" in options:
        _same(a, b)
    assert np.array_equal(a[0]["id"], b[0]["id"])
    assert np.linalg.norm(b[0]["vel"] - a[0]["vel"]) <= 1e-8 * np.linalg.norm(a[0]["vel"])
    assert abs(a[1][0][0] - b[1][0][0]) <= max(4, a[1][0][0] // 10)


@pytest.mark.parametrize("name", ["dam2d-close", "cube3d-close"])
def test_fused_slices(engine_lib, name):
    """Option pair_fuse: b bit for bit, D^-1 with its wall terms in another
    order (rel 1e-6)."""
    (dim, params, parts), _ = _pairs(name)
    out = {}
    for fuse in (0, 1):
        g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
        g.set_solver(1e-10, 1e-3, 50)
        g.set_option("pair_fuse", fuse)
        for st in ("step_begin", "cellsort", "neighbors", "explicit", "assemble"):
            g.stage(st)
        b, dinv = g.export("VectorB"), g.export("InvDiagA")
        g.stage("mg_build")
        g.stage("solve")
        s = g.solve_stats()
        assert s["status"] == 0 and s["inner_kernel"] == 0
        out[fuse] = (b, dinv, vec_proj(g.export("Velocity"), dim)[:g.fluid_count])
    (b0, d0, v0), (b1, d1, v1) = out[0], out[1]
    assert np.array_equal(b0, b1)
    assert rel(d1, d0) <= 1e-6
    assert np.linalg.norm(v1 - v0) <= 1e-8 * np.linalg.norm(v0)


@pytest.mark.parametrize("name,options,trials", [("resident", {}, 1), ("long2d", {}, 4), ("pairs", {"mg_depth": 0}, 7)])
def test_autotuner_times_what_acts(engine_lib, name, options, trials):
    case = ITERATED[name]() if name in ITERATED else _start(casegen.baseline_params(2, 0.01, 1.0e-4),
                                                            casegen.dam_case(2, (25, 20), (40, 30), 0.01, seed=2), 2)

    def make():
        g = engine.Case(case[1], case[2], case[0], precision=PRECISION_MIXED)
        g.set_solver(1e-10, 1e-3, 50)
        for k, v in options.items():
            g.set_option(k, v)
        return g
    out = autotune.tune(make, steps=1, warmup=1)
    assert len(out["ms_per_step"]) == trials
    for k, values in autotune.CANDIDATES:
        assert out["settings"][k] in values
