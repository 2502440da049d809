"""Branches of the stage kernels that a rule on sizes or options picks, at the
sizes where they can go wrong, bit for bit against the CPU oracle: the packed
last faces of x1 rows, fields too small for the branch-free quotients, electron
heating with and without the state, FixRecovery's one launch, and the CKS metric
tabulated or formed in the kernels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from parity_util import CASES, Case, field, to_device  # noqa: E402

from pangu_b200 import abi  # noqa: E402
from pangu_b200 import params as prm  # noqa: E402
from pangu_b200 import problems  # noqa: E402

pytestmark = pytest.mark.gpu


def _case(problem, extra, **kw):
    CASES["_branch"] = (problem, kw, extra)
    try:
        return Case("_branch")
    finally:
        del CASES["_branch"]


def _engine(case, hb):
    from pangu_b200.engine import Engine
    eng = Engine(case.params, case.mesh)
    base, one = eng.new_containers()
    to_device(hb, base)
    return eng, base, one


PPM4 = {("core", "limiter"): "ppm4", ("parthenon/mesh", "nghost"): 3}


# faces per row nx + 1 = 31 m + rest: rest 1, 2, 3 are packed (groups of 2, 4 and 4
# lanes), rest 0 and 4 are not; enough rows for the rule
@pytest.mark.parametrize("nx,blocks", [(31, 16), (32, 16), (33, 16), (34, 16), (61, 12), (64, 12)])
@pytest.mark.parametrize("limiter", ["mc", "ppm4"])
def test_last_faces_of_x1_rows(nx, blocks, limiter):
    over = {("core", "riemann_solver"): "hll"} if nx % 2 else {}
    case = _case("ot", {**(PPM4 if limiter == "ppm4" else {}), **over}, n=nx * blocks, nblock=nx)
    hb, _ = case.oracle_containers()
    eng, db, _ = _engine(case, hb)
    case.oracle.calculate_fluxes(hb)
    for march in (1, 8):
        if march == 8 and (nx + 2 * case.mesh.ng) % 2:
            continue  # the staged kernels need rows of whole 16-byte units
        eng.set_flux_config(x1_march=march)
        db.flux1.zero_()
        db.alfven.zero_()
        eng.calculate_fluxes(db)
        assert np.array_equal(field(db, "flux1"), hb.flux1), (nx, limiter, march)
        assert np.array_equal(field(db, "alfven"), hb.alfven)


def _packed_launches(eng, db):
    n = eng.launches()
    eng.calculate_fluxes(db)
    return eng.launches() - n


MHD3 = {("parthenon/mesh", "nx2"): 36, ("parthenon/mesh", "nx3"): 36,
        ("parthenon/meshblock", "nx2"): 12, ("parthenon/meshblock", "nx3"): 12}


@pytest.mark.parametrize("problem,kw,over", [
    ("torus", dict(nx1=64, nx2=32, nx3=32, bx=(32, 16, 8)), {}),
    ("torus", dict(nx1=66, nx2=32, nx3=32, bx=(33, 16, 8), limiter="mc", riemann="hll"), {}),
    ("torus", dict(nx1=62, nx2=32, nx3=32, bx=(31, 16, 8)), {}),
    ("cks", dict(n=64, nblock=32), MHD3), ("cks", dict(n=64, nblock=32), {**MHD3, **PPM4}),
    ("ot", dict(n=62 * 12, nblock=62), {}), ("ot", dict(n=62 * 12, nblock=62), PPM4)])
def test_last_faces_of_x1_rows_in_curved_metrics(problem, kw, over):
    """The packed last faces in blocks whose metric is not flat, in three dimensions,
    through pointer tables and beside the staged rows, one face a row (62) among them."""
    from pangu_b200.engine import TableContainer
    case = _case(problem, over, **kw)
    hb, _ = case.oracle_containers()
    eng, db, _ = _engine(case, hb)
    case.oracle.calculate_fluxes(hb)
    dims = 3 if case.mesh.nx3 > 1 else 2
    for march in (1, 8):
        if march == 8 and (case.mesh.nx1 + 2 * case.mesh.ng) % 2:
            continue
        eng.set_flux_config(x1_march=march)
        db.flux1.zero_()
        assert _packed_launches(eng, db) == dims + 1
        assert np.array_equal(field(db, "flux1"), hb.flux1), march
        assert np.array_equal(field(db, "alfven"), hb.alfven)
    tab = TableContainer(eng.nb, eng.nf, eng.shape, eng.device)
    db.flux1.zero_()
    tab.load(db)
    assert _packed_launches(eng, tab) == dims + 1
    assert np.array_equal(tab.gather("flux1").cpu().numpy(), hb.flux1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("limiter,riemann,nx", [("ppm4", "laxf", 32), ("mc", "hll", 33),
                                                ("ppm4", "hll", 62)])
def test_packed_faces_do_not_depend_on_the_other_jobs(precision, limiter, riemann, nx):
    """The first job's x1 fluxes with its last faces in the x1 kernel (alone in the pool)
    and packed with those of 23 more jobs."""
    from pangu_b200.engine import Pool
    pin = problems.fm_torus_input(nx, 128, 1, None, seed=4)
    for k, v in (("limiter", limiter), ("riemann_solver", riemann)):
        pin.set("core", k, v)
    pin.set("parthenon/mesh", "nghost", 3 if limiter == "ppm4" else 2)
    pin.set("b200", "precision", precision)
    pool = Pool(pin, 24, 24)
    job = pool.attach_problem(pin, "torus")
    slot = pool.jobs[job][0]
    assert _packed_launches(pool.engine, pool.base) == 2
    alone = pool.base.flux1[slot].clone()
    assert float(alone.abs().max()) > 0.0
    for _ in range(23):
        pool.attach_problem(pin, "torus")
    pool.base.flux1.zero_()
    assert _packed_launches(pool.engine, pool.base) == 3
    assert torch.equal(pool.base.flux1[slot], alone)


@pytest.mark.parametrize("problem,kw,over", [
    ("torus", dict(nx1=40, nx2=24), {}),
    ("torus", dict(nx1=40, nx2=24, limiter="mc", riemann="hll"), {}),
    ("ot", dict(n=32), {**PPM4, ("core", "riemann_solver"): "hll"})])
def test_fields_down_to_the_smallest_numbers(problem, kw, over):
    """The magnetic field of each cell scaled by 2^-e, e from 0 past the end of the
    subnormal numbers, zeros of both signs among them."""
    case = _case(problem, over, **kw)
    hb, ho = case.oracle_containers()
    rng = np.random.default_rng(5)
    shape = hb.prim.shape[:1] + hb.prim.shape[2:]
    scale = np.ldexp(rng.uniform(0.5, 1.0, shape), -rng.integers(0, 1100, shape))
    scale[rng.random(shape) < 0.1] = -0.0
    hb.prim[:, 5:8] = rng.uniform(-1.0, 1.0, hb.prim[:, 5:8].shape) * scale[:, None]
    eng, db, do = _engine(case, hb)
    to_device(ho, do)
    dt = torch.full((1,), 1e-3, dtype=torch.float64, device="cuda")
    for march, m2 in ((1, 1), (1, 0), (8, 8)):
        eng.set_flux_config(x1_march=march, x2_march=m2)
        case.oracle.calculate_fluxes(hb)
        eng.calculate_fluxes(db)
        for f in ("flux1", "flux2", "alfven"):
            assert np.array_equal(field(db, f), getattr(hb, f)), (march, f)
    case.oracle.stage(1, hb, ho, 0.5, 1e-3)
    eng.stage(1, db, do, 0.5, dt)
    for f in ("prim", "cons"):
        assert np.array_equal(field(do, f), getattr(ho, f), equal_nan=True), f


SHAPES = ((1, 1, 128), (8, 2, 128), (1, 4, 128), (1, 0, 128), (1, 0, 256), (8, 8, 128))


def _fluxes_of_every_shape(case, hb):
    """(shape, field, result, oracle's result) of calculate_fluxes for each tile shape."""
    eng, db, _ = _engine(case, hb)
    case.oracle.calculate_fluxes(hb)
    fields = ("flux1", "flux2", "alfven") + (("flux3",) if case.mesh.nx3 > 1 else ())
    for m1, m, t in SHAPES:
        eng.set_flux_config(x1_march=m1, x2_march=m, x2_threads=t, x3_march=m, x3_threads=t)
        for f in fields:
            getattr(db, f).zero_()
        eng.calculate_fluxes(db)
        for f in fields:
            yield (m1, m, t), f, field(db, f), getattr(hb, f)


def _some_not_finite(hb, seed):
    """NaN anywhere; infinities, alone and in pairs of one sign along each direction, in
    the scalars (where a component is structurally zero the oracle multiplies it out)."""
    rng = np.random.default_rng(seed)
    hb.prim[rng.random(hb.prim.shape) < 1e-3] = np.nan
    for v in {0, 1, hb.prim.shape[1] - 2, hb.prim.shape[1] - 1} - {7}:
        q = hb.prim[:, v]
        for ax in (None, -1, -2, -3):
            at = rng.random(q.shape) < 2e-3
            q[at if ax is None else at | np.roll(at, 1, ax)] = rng.choice([np.inf, -np.inf])


@pytest.mark.parametrize("problem,kw,over", [
    ("torus", dict(nx1=58, nx2=24), {}),
    ("torus", dict(nx1=26, nx2=16, nx3=8, bx=(26, 8, 8)), {}),
    ("ot", dict(n=58), PPM4)])
def test_ppm4_next_to_cells_that_are_not_finite(problem, kw, over):
    """Every shape of the flux kernels limits a cell beside a NaN or an infinity as the
    scalar limiter does, the staged tiles (march 8) among them."""
    case = _case(problem, over, **kw)
    hb, _ = case.oracle_containers()
    _some_not_finite(hb, 9)
    for shape, f, a, b in _fluxes_of_every_shape(case, hb):
        assert np.isfinite(b).mean() > 0.3
        assert np.array_equal(a, b, equal_nan=True), (shape, f)


@pytest.mark.parametrize("problem,kw,over", [
    ("torus", dict(nx1=60, nx2=24, limiter="mc", riemann="hll"), {}),
    ("ot", dict(n=60), {})])
def test_mc_next_to_cells_that_are_not_finite(problem, kw, over):
    case = _case(problem, over, **kw)
    hb, _ = case.oracle_containers()
    _some_not_finite(hb, 10)
    for shape, f, a, b in _fluxes_of_every_shape(case, hb):
        assert np.isfinite(b).mean() > 0.3
        assert np.array_equal(a, b, equal_nan=True), (shape, f)


@pytest.mark.parametrize("model", sorted(abi.HEATING_MODEL))
@pytest.mark.parametrize("suppress", [False, True])
def test_heating_with_and_without_the_state(model, suppress):
    case = _case("torus", {("electron", "model"): model,
                           ("electron", "suppress_highb_heat"): suppress}, nx1=40, nx2=24)
    hb, ho = case.oracle_containers()
    case.oracle.stage(1, hb, ho, 0.5, 1e-3)
    rng = np.random.default_rng(6)
    ho.cons[:, 8:10] *= rng.uniform(0.5, 2.0, ho.cons[:, 8:10].shape)
    eng, _, do = _engine(case, hb)
    to_device(ho, do)
    case.oracle.apply_electron_heating(ho)
    eng.apply_electron_heating(do)
    # the oracle's exp and log are the C library's: two ulp in the models that call them
    a, b = field(do, "prim"), ho.prim
    if model in ("howes", "kawazura", "rowan"):
        np.testing.assert_allclose(a, b, rtol=1e-14, atol=0.0)
    else:
        assert np.array_equal(a, b)


@pytest.mark.parametrize("share", [0.0, 1e-4, 0.02, 0.6, 1.0])
def test_fix_recovery_of_any_number_of_cells(share):
    case = Case("ot_mc_laxf") if share < 0.5 else _case("ot", {}, n=288)
    hb, _ = case.oracle_containers()
    rng = np.random.default_rng(7)
    hb.flag[...] = (rng.random(hb.flag.shape) >= share).astype(float)
    eng, db, _ = _engine(case, hb)
    for _ in range(2):  # the second call finds the ticket as the first left it
        to_device(hb, db)
        eng.fix_recovery(db)
    case.oracle.fix_recovery(hb)
    assert np.array_equal(field(db, "prim"), hb.prim)
    assert np.array_equal(field(db, "flag"), hb.flag)


def _repair(case, share, calls):
    hb, _ = case.oracle_containers()
    rng = np.random.default_rng(11)
    hb.flag[...] = (rng.random(hb.flag.shape) >= share).astype(float)
    eng, db, _ = _engine(case, hb)
    for _ in range(calls):  # each finds the counters as the one before left them
        to_device(hb, db)
        eng.fix_recovery(db)
    return hb, eng, db


# 9 components a cell: 8192 tasks (910 cells) are the longest list that one CTA writes
@pytest.mark.parametrize("n,share", [(96, 0.09), (96, 0.11), (96, 1.0), (512, 0.4), (512, 1.0)])
def test_fix_recovery_of_short_and_long_lists(n, share):
    case = _case("ot", {}, n=n)
    hb, _, db = _repair(case, share, 3)
    case.oracle.fix_recovery(hb)
    assert np.array_equal(field(db, "prim"), hb.prim)
    assert np.array_equal(field(db, "flag"), hb.flag)


def test_fix_recovery_of_every_cell_is_spread_over_the_gpu():
    """A list of 262,144 cells takes less time than two evaluations of the fluxes (it
    moves a fifth of their bytes): one CTA that wrote it alone took ten."""
    case = _case("ot", {}, n=512)
    hb, eng, db = _repair(case, 1.0, 1)
    one = torch.zeros_like(db.flag)

    def clock(f):
        best = np.inf
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            db.flag.copy_(one)
            e[0].record()
            f(db)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert clock(eng.fix_recovery) < 2.0 * clock(eng.calculate_fluxes)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cks_tables_or_not(precision):
    """One mesh keeps its metric in tables, a pool forms it in the kernels."""
    from pangu_b200.engine import Pool, Simulation
    pin = problems.cks_atmosphere_input(n=20, nblock=10)
    pin.set("b200", "precision", precision)
    geo = problems.Geometry(prm.mesh_struct(pin))
    prim = problems.cks_atmosphere(geo, prm.process_packages(pin))
    sim = Simulation(pin)
    sim.set_primitives(prim)
    pool = Pool(pin, 9, 1)
    job = pool.attach(pin, prim)
    for _ in range(3):
        sim.step()
        pool.step(graph=False)
    torch.cuda.synchronize()
    assert np.array_equal(sim.primitives(), pool.primitives(job), equal_nan=True)
    assert float(sim.dt) == float(pool.dt[job])


def test_forming_the_cks_metric_in_a_pool_costs_little_more_than_its_tables():
    """The fluxes of a pool, whose kernels form the metric, against those of a mesh that
    keeps it in tables: 1.1 times as long. Formed by a call out of the kernel, 1.3."""
    from pangu_b200.engine import Pool, Simulation
    pin = problems.cks_atmosphere_input(n=64, nblock=32)
    prim = problems.cks_atmosphere(problems.Geometry(prm.mesh_struct(pin)),
                                   prm.process_packages(pin))
    sim, pool = Simulation(pin), Pool(pin, 8, 1)
    sim.set_primitives(prim)
    pool.attach(pin, prim)
    times = []
    for x in (sim, pool):
        best = np.inf
        for _ in range(20):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            x.engine.calculate_fluxes(x.base)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        times.append(best)
    assert times[1] < 1.2 * times[0]


@pytest.mark.parametrize("cfl", [0.3, 0.0, -0.3])
@pytest.mark.parametrize("kind", ["plain", "zeros", "negative", "nan", "inf"])
def test_timestep_from_any_speeds(kind, cfl):
    """The reference's minimum (timestep_estimation.cc:56-92) takes a negative dt and
    skips a NaN."""
    case = _case("ot", {("core", "cfl_number"): cfl}, n=40, nblock=20)
    hb, _ = case.oracle_containers()
    rng = np.random.default_rng(8)
    a = rng.uniform(0.0, 2.0, hb.alfven.shape)
    pick = rng.random(a.shape)
    if kind == "zeros":
        a[pick < 0.5], a[pick > 0.8] = 0.0, -0.0
    elif kind == "negative":
        a[pick < 0.3] *= -1.0
    elif kind == "nan":
        a[pick < 0.9] = np.nan
    elif kind == "inf":
        a[pick < 0.1] = np.inf
    hb.alfven[...] = a
    eng, db, _ = _engine(case, hb)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    eng.estimate_dt(db, out)
    geo = case.geo
    big = np.finfo(np.float64).max
    est = big
    with np.errstate(all="ignore"):
        for b in range(geo.nb):
            inv = 0.0
            for d in range(3):
                m = np.float64(big)
                if geo.act[d]:
                    q = (cfl * geo.dx[d]) / hb.alfven[b, d][geo.interior()]
                    q = q[~np.isnan(q)]
                    m = np.float64(min(big, q.min())) if q.size else m
                inv = np.float64(1.0) / m if d == 0 else inv + np.float64(1.0) / m
            bdt = np.float64(1.0) / inv
            est = bdt if bdt < est else est
    # a minimum of zero may carry either sign, and so does its reciprocal
    got = float(out)
    if est == 0.0 or np.isinf(est):
        assert abs(got) == abs(float(est))
    else:
        assert got == float(est) or (np.isnan(got) and np.isnan(est))
