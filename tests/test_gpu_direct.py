"""The direct stencil kernels (a handle's own choice of form) against the
stream kernels, which share none of their code: at the remainders of their
16-byte cells and of a plane's threads, on both sides of the one-cell-per-thread
bound, with slabs that overlap, masked or missing, for every way alpha can
relate to beta, batch widths around a block's warps and the compact storages.
The roundings are spelled out, so the bits agree; where the two slabs of an axis
overlap, the direct kernels take all near faces before the far ones, another
order of the corrections, and agree to rounding."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 37  # odd, more than one 32-slot monitor block
TOL = {"double": 1e-12, "single": 1e-5}  # relative to the largest field


def _problem(n, layers, alpha, batch, seed=3):
    from magnelio_b200 import host
    from magnelio_b200.problem import FACES, CpmlFace, DftMonitor, FitProblem, LumpedPort

    rng = np.random.default_rng(seed)
    nx, ny, nz = n
    d = [1e-3 * rng.uniform(0.8, 1.2, v) for v in n]
    x, y, z = (np.concatenate([[0.0], np.cumsum(v)]) for v in d)
    mat = rng.integers(0, 3, n).astype(np.int32)
    M_eps = host.build_M_eps(x, y, z, [1.0, 2.5, 6.0], mat)
    M_mu = host.build_M_mu(x, y, z)
    dt = host.courant_dt(x, y, z)
    aE, bE, aH, bH = host.leapfrog_coefficients(M_eps, M_mu, dt)
    frozen = rng.choice(aE.size, aE.size // 50, replace=False)
    bE[frozen] = 0.0
    if alpha == "pec":  # frozen at zero: alpha = (beta != 0)
        aE[frozen] = 0.0
    elif alpha == "mixed":  # some frozen at zero, some kept: alpha is read
        aE[frozen[::2]] = 0.0
    elif alpha == "lossy":
        aE[bE != 0] *= rng.uniform(0.9, 1.0, int(np.sum(bE != 0)))
    prob = FitProblem(nx=nx, ny=ny, nz=nz, dt=dt, dx=d[0], dy=d[1], dz=d[2], alpha_E=aE, beta_E=bE, alpha_H=aH,
                      beta_H=bH, M_eps=M_eps, M_mu=M_mu, batch=batch)
    for face, k in zip(FACES, layers):
        if not k:
            continue
        axis = "xyz".index(face[0])
        b, c, ck = host.cpml_tables(d[axis], face, dt, thickness_cells=k)
        air = (None,) * 4
        if face == "ymin":  # PEC inside one slab
            shapes = [((nx, k, nz + 1)), (nx + 1, k, nz), (nx + 1, k, nz), (nx, k, nz + 1)]
            air = tuple((rng.random(s) > 0.2).astype(np.uint8) for s in shapes)
        prob.cpml.append(CpmlFace(face, b, c, ck, air))
    ey0 = nx * (ny + 1) * (nz + 1)
    for p in range(2):
        i, j, k = nx // 2 + p, ny // 2, (nz // 2 + p) % nz  # an edge of its own also for one cell in z
        flat = ey0 + (i * ny + j) * (nz + 1) + k
        prob.lumped.append(LumpedPort(np.array([flat]), np.ones(1), np.array([dt / M_eps[flat]]), R=50.0,
                                      v_src=[rng.standard_normal(STEPS) for _ in range(batch)]))
    prob.monitors.append(DftMonitor(((0, nx), (0, ny), (nz // 2, nz // 2 + 1)), ("Ex", "Hz"), np.array([1e9, 5e9]), 1))
    prob.e0 = [rng.standard_normal(aE.size) * (aE != 0) for _ in range(batch)]
    prob.h0 = [rng.standard_normal(aH.size) / 377.0 for _ in range(batch)]
    return prob


def _march(prob, precision, form, coef):
    with prob.build_engine(precision) as eng:
        if form:
            eng.configure_stencil(form)
        if coef != "native":
            eng.set_coefficient_storage(coef)
        eng.step(STEPS)
        return ([eng.read_fields(b) for b in range(prob.batch)], [eng.read_vi(b) for b in range(prob.batch)],
                [eng.read_dft(0, c) for c in ("Ex", "Hz")])


@pytest.mark.parametrize("n,layers,alpha,batch,precision,coef", [
    ((5, 4, 1), (0, 0, 0, 0, 0, 0), "pec", 1, "double", "native"),           # one cell in z, no slab
    ((9, 7, 12), (3, 3, 2, 2, 8, 7), "one", 1, "double", "native"),          # overlapping z slabs
    ((8, 9, 11), (8, 5, 9, 9, 0, 4), "pec", 2, "double", "native"),          # slabs as thick as the axis
    ((20, 19, 31), (4, 4, 4, 4, 4, 4), "mixed", 3, "single", "native"),      # batch without a stream form
    ((53, 52, 54), (6, 5, 4, 7, 5, 6), "pec", 1, "single", "native"),        # just below the 16-byte bound
    ((53, 53, 55), (6, 5, 4, 7, 5, 6), "one", 1, "single", "native"),        # just above it
    ((54, 53, 56), (0, 0, 6, 6, 1, 3), "lossy", 1, "single", "native"),      # z remainders 1 and 3
    ((62, 51, 49), (5, 0, 0, 5, 49, 0), "one", 1, "double", "native"),       # a z slab of the whole axis
    ((62, 51, 50), (5, 5, 0, 0, 30, 30), "pec", 1, "double", "native"),      # overlapping, 16-byte form
    ((300, 23, 25), (10, 10, 2, 2, 6, 6), "one", 5, "single", "native"),     # more field sets than warps
    ((53, 53, 55), (6, 6, 6, 6, 6, 6), "pec", 2, "single", "f16"),
    ((53, 53, 55), (6, 6, 6, 6, 6, 6), "one", 1, "single", "bf16"),
    ((53, 53, 55), (6, 6, 6, 6, 6, 6), "pec", 1, "double", "f16"),
])
def test_direct_kernels_match_the_stream_kernels(n, layers, alpha, batch, precision, coef):
    prob = _problem(n, layers, alpha, batch)
    got = _march(prob, precision, None, coef)
    if batch in (1, 2, 4, 8, 16):
        want = _march(prob, precision, "stream", coef)
    else:  # one field set per handle
        want = ([], [], None)
        for b in range(batch):
            one = _problem(n, layers, alpha, batch)
            one.batch, one.e0, one.h0 = 1, [one.e0[b]], [one.h0[b]]
            for lp in one.lumped:
                lp.v_src = [lp.v_src[b]]
            f, vi, dft = _march(one, precision, "stream", coef)
            want[0].append(f[0])
            want[1].append(vi[0])
            want = (want[0], want[1], want[2] or dft)
    tol = TOL[precision]
    overlap = any(layers[2 * q] + layers[2 * q + 1] > n[q] for q in range(3))

    def close(a, b, scale, t):
        assert np.all(np.isfinite(a)) and float(np.max(np.abs(a - b))) <= t * scale
        assert overlap or np.array_equal(a, b)

    for q in range(2):
        scale = max(float(np.max(np.abs(f[q]))) for f in want[0])
        for a, b in zip(got[0], want[0]):
            close(a[q], b[q], scale, tol)
        scale = max(float(np.max(np.abs(v[q]))) for v in want[1])
        for a, b in zip(got[1], want[1]):
            close(a[q], b[q], scale, 10 * tol)
    for a, b in zip(got[2], want[2]):
        close(a, b, float(np.max(np.abs(b))), 1e-5)  # float32 bins


@pytest.mark.parametrize("n", [(43, 41, 24), (44, 41, 24), (90, 67, 61), (131, 89, 113)])
def test_large_reads_return_every_entry(n):
    """Fields and monitor bins around the size of one piece of the threaded
    read, and over many pieces with a ragged last one: what was set comes
    back, and the complex read equals the split one."""
    import ctypes as C

    from magnelio_b200 import _lib
    from magnelio_b200._lib import f64p
    from magnelio_b200.engine import FitEngine

    rng = np.random.default_rng(4)
    d = [np.full(v, 1e-3) for v in n]
    with FitEngine(*n, 1e-13) as eng:
        one = [np.ones(s) for s in (eng.n_E, eng.n_E, eng.n_H, eng.n_H)]
        eng.set_coefficients(one[0], 0.1 * one[1], one[2], 0.1 * one[3])
        m = eng.add_dft_monitor(tuple((0, v) for v in n), ("Ey",), [1e9, 2e9, 3e9], *d)
        e, h = (rng.standard_normal(s).astype(np.float32) for s in (eng.n_E, eng.n_H))
        eng.set_fields(e, h)
        ge, gh = eng.read_fields()
        assert np.array_equal(ge, e) and np.array_equal(gh, h)
        eng.step(2)
        bins = eng.read_dft(m, "Ey")
        re, im = np.empty(bins.size), np.empty(bins.size)
        _lib.check(_lib.load().fitb_read_dft(eng._h, C.c_int32(m), 0, 1, f64p(re), f64p(im), bins.size))
        assert np.array_equal(bins.real.ravel(), re) and np.array_equal(bins.imag.ravel(), im)
        assert np.any(re != 0) and np.all(np.isfinite(re))


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("n,layers", [((26, 24, 45), 4), ((58, 55, 61), 6)])
def test_cpml_stays_fused_beside_clear_dispersion(n, layers, precision):
    """Dispersive entries outside the slabs: the direct kernels keep the CPML
    fused, the stream kernels run it as passes after the ADE update."""
    from magnelio_b200.workloads import dispersive_slab

    prob = dispersive_slab(*n, seed=6, cpml_cells=layers, n_freq=3)
    out = []
    for form in (None, "stream"):
        with prob.build_engine(precision) as eng:
            if form:
                eng.configure_stencil(form)
            eng.step(3 * max(n))
            out.append((*eng.read_fields(), *(eng.read_dft(m, "Ex") for m in range(2))))
    for a, b in zip(*out):
        assert float(np.max(np.abs(b))) > 0 and np.array_equal(a, b)


def _slab_case(name, precision):
    from conftest import load_golden

    from magnelio_b200.workloads import dispersive_slab

    if name == "box":
        return _problem((53, 53, 55), (6, 5, 4, 7, 5, 6), "pec", 1)
    if name == "small_batch":
        return _problem((20, 19, 31), (4, 4, 4, 4, 4, 4), "mixed", 2)
    if name == "two_edge_port":  # stepped between the E and the H update: buffer to buffer
        prob = _problem((53, 53, 55), (6, 6, 6, 6, 6, 6), "one", 1)
        lp = prob.lumped[0]
        lp.flat_idx = np.array([lp.flat_idx[0], lp.flat_idx[0] + 2 * (prob.nz + 1)])
        lp.signs, lp.betas = np.ones(2), np.repeat(lp.betas, 2)
        return prob
    if name == "dispersive":
        return dispersive_slab(26, 24, 45, seed=6, cpml_cells=4, n_freq=3)
    return load_golden(name)[0]


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("name", ["box", "small_batch", "two_edge_port", "dispersive", "wg_dtbc", "planewave_box"])
def test_slab_step_on_the_direct_kernels_matches_its_unit_lists(name, precision):
    """Without a march depth the slab step runs on the direct kernels, in
    place or from one buffer set to the other; with one it keeps its unit
    lists.  Odd and even step counts, so both buffer sets end up current."""
    out = []
    for depth in (0, 9):
        prob = _slab_case(name, precision)
        with prob.build_engine(precision) as eng:
            eng.configure_stencil("fused", 16, depth)
            assert (eng.stencil_config()["ichunk"] > 0) == (depth > 0)
            eng.step(20)
            eng.step(STEPS - 20)
            out.append([a for b in range(prob.batch) for a in (*eng.read_fields(b), *eng.read_vi(b))])
    for q, (a, b) in enumerate(zip(*out)):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b), q


@pytest.mark.parametrize("count", [1, 8, 9])
def test_monitor_slots_with_and_without_packed_descriptors(count):
    """Monitors of strides 1 .. count, up to and past the number whose
    descriptors travel as kernel arguments: the bins are the DFT sums of the
    fields read after every step, over whole and partial slot blocks."""
    from magnelio_b200.problem import DftMonitor

    prob = _problem((9, 8, 11), (0,) * 6, "one", 1)
    freqs = np.array([1e9, 7e9])
    prob.monitors = [DftMonitor(((1, 7), (2, 8), (3, 9)), ("Ez",), freqs, stride) for stride in range(1, count + 1)]
    want = [np.zeros((2, 6, 6, 6), complex) for _ in range(count)]
    steps = 70
    with prob.build_engine("double") as eng:
        shape = eng.shapes["Ez"]
        for n in range(steps):
            eng.step(1)
            ez = eng.read_fields()[0][-int(np.prod(shape)):].reshape(shape)
            a = ez[1:8, 2:9, 3:9]
            cell = 0.25 * (a[:-1, :-1] + a[1:, :-1] + a[:-1, 1:] + a[1:, 1:]) / prob.dz[None, None, 3:9]
            for m in range(count):
                if n % (m + 1) == 0:
                    w = np.exp(2j * np.pi * freqs * n * prob.dt) * (m + 1) * prob.dt
                    want[m] += w[:, None, None, None] * cell
        for m in range(count):
            got = eng.read_dft(m, "Ez")
            assert np.max(np.abs(got - want[m])) <= 1e-5 * np.max(np.abs(want[m]))  # float32 samples and bins


def _late_dispersion(prob, where):
    """A one-pole block on E entries inside the xmin slab, or on and beside
    the first port's edge (clear of every slab); coupling 5 % of a field step."""
    from magnelio_b200.problem import Dispersion, DispersionBlock

    if where == "slab":
        idx = np.flatnonzero(prob.beta_E[:2 * (prob.ny + 1) * (prob.nz + 1)])
    else:
        idx = prob.lumped[0].flat_idx[0] + np.arange(-2, 3)
        idx = idx[prob.beta_E[idx] != 0]
    block = DispersionBlock(idx.astype(np.int64), 0.05 / prob.beta_E[idx], np.zeros(1, np.int32), np.array([0.9]),
                            np.array([1.0]), np.ones(1))
    return [Dispersion("E", [block])]


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("form", [None, ("fused", 16), ("stream",)])
@pytest.mark.parametrize("where", ["slab", "port"])
def test_dispersion_added_to_a_prepared_handle(where, form, precision):
    """A block added after the handle prepared its step (a step of zero) is
    taken as if it had been there before: the CPML of a slab that it reaches
    into follows the pole update, a port on its edge follows it too, and the
    slab step recomputes H beside it (or refuses the block in a slab)."""
    from magnelio_b200._lib import FitbError

    prob = _problem((26, 24, 45), (4,) * 6, "one", 1)
    disp = _late_dispersion(prob, where)
    out = []
    for late in (True, False):
        prob.dispersion = [] if late else disp
        with prob.build_engine(precision) as eng:
            if form and late:
                eng.configure_stencil(*form)
            if late:
                eng.reserve_steps(STEPS)
                eng.step(0)
                for side in disp:
                    for block in side.blocks:
                        eng.add_dispersion_block(side.side, block)
            if form == ("fused", 16) and where == "slab":
                with pytest.raises(FitbError, match="outside the CPML slabs"):
                    eng.step(STEPS) if late else eng.configure_stencil(*form)
                continue
            if form and not late:
                eng.configure_stencil(*form)
            eng.step(STEPS)
            out.append((*eng.read_fields(), *eng.read_vi(), eng.read_dft(0, "Ex")))
    for a, b in zip(*out):  # the same operations in the same order
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.parametrize("form", [None, ("fused", 16, 0)])
def test_more_planes_than_one_grid_dimension(form):
    """A long thin box of 70 001 planes, more than the 65 535 blocks of a
    grid's y dimension: the direct kernels give the stream kernels' march."""
    out = []
    for f in (form, ("stream", 0, 0)):
        prob = _problem((70000, 2, 3), (10, 10, 0, 0, 0, 0), "pec", 1)
        with prob.build_engine("single") as eng:
            if f:
                eng.configure_stencil(*f)
            eng.step(STEPS)
            out.append((*eng.read_fields(), *eng.read_vi()))
            assert eng.steps_done == STEPS
    for q, (a, b) in enumerate(zip(*out)):
        scale = float(np.max(np.abs(b)))
        assert scale > 0 and float(np.max(np.abs(a - b))) <= (1 if q < 2 else 10) * TOL["single"] * scale, q


def test_a_form_that_cannot_launch_is_not_timed():
    """One plane per CTA asks the stream kernels for more blocks than a grid's
    z dimension has on a box of 70 001 planes: the stencil timer reports the
    refused launches, and the step does."""
    from magnelio_b200._lib import FitbError

    prob = _problem((70000, 2, 3), (0,) * 6, "one", 1)
    with prob.build_engine("single") as eng:
        eng.configure_stencil("stream", 0, 1)
        with pytest.raises(FitbError):
            eng.time_stencil(2)
        with pytest.raises(FitbError):
            eng.step(1)
        eng.configure_stencil("stream", 0, 0)
        assert sum(eng.time_stencil(2)) > 0


def test_a_step_that_cannot_launch_is_refused_every_time():
    """A monitor whose phasors exceed a block's shared memory: no step may
    count as done, on the first call or on any later one, timed or not, and
    the handle without it steps on."""
    from magnelio_b200._lib import FitbError
    from magnelio_b200.problem import DftMonitor

    prob = _problem((9, 8, 11), (0,) * 6, "one", 1)
    with prob.build_engine("single") as eng:
        eng.step(3)
        want = eng.read_fields()
    prob.monitors.append(DftMonitor(((0, 9), (0, 8), (5, 6)), ("Ez",), np.linspace(1e9, 9e9, 5000), 1))
    with prob.build_engine("single") as eng:
        for _ in range(2):
            with pytest.raises(FitbError):
                eng.step(3)
            with pytest.raises(FitbError):
                eng.step_timed(3)
            assert eng.steps_done == 0
    prob.monitors.pop()
    with prob.build_engine("single") as eng:
        eng.step(3)
        assert all(np.array_equal(a, b) for a, b in zip(want, eng.read_fields()))


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("depth", [1, 5, 54, 2**31 - 1])
def test_planes_per_thread_of_the_direct_kernels(depth, precision):
    """Any number of planes per thread, past the mesh too, gives the bits of
    one plane per thread, and the handle reports no more planes than it has."""
    out = []
    for d in (0, depth):
        prob = _problem((53, 53, 55), (6, 5, 4, 7, 5, 6), "pec", 1)
        with prob.build_engine(precision) as eng:
            eng.configure_stencil("simple", 0, d)
            assert eng.stencil_config()["ichunk"] <= prob.nx + 1
            eng.step(STEPS)
            out.append((*eng.read_fields(), *eng.read_vi(), eng.read_dft(0, "Hz")))
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("n,batch,n_freq", [
    ((9, 8, 11), 3, 5),        # a sample per thread, one launch
    ((20, 19, 31), 8, 130),    # blocks of fewer than 32 steps
    ((60, 62, 64), 1, 3),      # many samples: staging and flush as launches of their own
    ((60, 62, 64), 2, 100),    # the same with short blocks and two field sets
])
def test_monitored_batches_equal_their_field_sets(n, batch, n_freq, precision):
    """Volume monitors of a batch, over whole and partial slot blocks, on
    meshes on both sides of the samples that one launch takes: every field
    set's bins are those of a handle of its own, bit for bit, and the DFT sums
    of the fields read after every step."""
    from magnelio_b200.problem import DftMonitor

    steps = 70
    freqs = np.linspace(1e9, 9e9, n_freq)

    def problem(sets):
        prob = _problem(n, (0,) * 6, "one", batch)
        prob.lumped = []
        prob.e0, prob.h0 = [prob.e0[b] for b in sets], [prob.h0[b] for b in sets]
        prob.batch = len(sets)
        prob.monitors = [DftMonitor(tuple((0, v) for v in n), ("Ex", "Ey", "Hz"), freqs, 1)]
        return prob

    with problem(range(batch)).build_engine(precision) as eng:
        eng.step(steps)
        got = [[eng.read_dft(0, c, b) for c in ("Ex", "Ey", "Hz")] for b in range(batch)]
    for b in range(batch):
        prob = problem([b])
        with prob.build_engine(precision) as eng:
            shape, want = eng.shapes["Ex"], 0.0
            for s in range(steps):
                eng.step(1)
                if b == 0 and n_freq <= 5:
                    ex = eng.read_fields()[0][:int(np.prod(shape))].reshape(shape)
                    cell = 0.25 * (ex[:, :-1, :-1] + ex[:, 1:, :-1] + ex[:, :-1, 1:] + ex[:, 1:, 1:])
                    cell = cell / prob.dx[:, None, None]
                    want = want + np.exp(2j * np.pi * freqs * s * prob.dt)[:, None, None, None] * prob.dt * cell
            one = [eng.read_dft(0, c) for c in ("Ex", "Ey", "Hz")]
        assert all(np.array_equal(x, y) for x, y in zip(got[b], one))
        if b == 0 and n_freq <= 5:
            assert np.max(np.abs(one[0] - want)) <= 1e-5 * np.max(np.abs(want))  # float32 samples and bins


def test_the_form_reported_is_the_form_that_runs():
    """The slab step reports depth 0 and the direct kernels' grid where it runs
    on them, its march depth where it runs on its unit lists, and what it
    reports configures the same kernels again."""
    prob = _problem((53, 53, 55), (6, 5, 4, 7, 5, 6), "one", 1)
    with prob.build_engine("single") as eng:
        default = eng.stencil_config()
        assert default["kind"] == "simple" and default["ichunk"] == 1 and default["grid"][1] == prob.nx + 1
        for depth in (0, 9):
            eng.configure_stencil("fused", 18, depth)
            cfg = eng.stencil_config()
            assert (cfg["kind"], cfg["variant"], cfg["ichunk"]) == ("fused", 18, depth)
            assert (cfg["grid"] == default["grid"]) == (depth == 0)
            before = eng.launch_count
            eng.step(1)
            launches = eng.launch_count - before
            eng.configure_stencil(cfg["kind"], cfg["variant"], cfg["ichunk"])
            assert eng.stencil_config() == cfg
            before = eng.launch_count
            eng.step(1)
            assert eng.launch_count - before == launches


@pytest.mark.parametrize("n,batch,frozen,layers,lists", [
    ((97, 104, 89), 1, 0.0, 8, False),     # CPML all round
    ((97, 104, 89), 1, 0.45, 8, False),    # dead units, but few of them clear of the CPML
    ((60, 62, 64), 1, 0.7, 0, False),      # mostly dead, but too small for five launches
    ((160, 160, 160), 1, 0.5, 0, True),    # half dead
    ((128, 120, 128), 4, 0.25, 0, True),   # a quarter dead, in a batch
])
def test_slab_step_takes_the_cheaper_of_its_two_routes(n, batch, frozen, layers, lists):
    """Far from the line on both sides the unit lists run where dead units and
    batches pay for them, the direct kernels elsewhere; and the bits are those
    of the other route."""
    from magnelio_b200 import host
    from magnelio_b200.engine import FitEngine
    from magnelio_b200.problem import FACES

    rng = np.random.default_rng(1)
    out = []
    for depth in (0, 16):
        with FitEngine(*n, 1e-13, batch=batch) as eng:
            a, b = np.ones(eng.n_E), np.full(eng.n_E, 0.1)
            off = 0
            for c in ("Ex", "Ey", "Ez"):
                s = eng.shapes[c]
                m = int(np.prod(s))
                for v in (a, b):
                    v[off:off + m].reshape(s)[:, :int(frozen * s[1])] = 0.0
                off += m
            eng.set_coefficients(a, b, np.ones(eng.n_H), np.full(eng.n_H, 0.1))
            for face in FACES if layers else ():
                d = np.full(n["xyz".index(face[0])], 1e-3)
                eng.add_cpml(face, *host.cpml_tables(d, face, 1e-13, thickness_cells=layers), (None,) * 4)
            eng.configure_stencil("fused", 16, depth)
            assert (eng.stencil_config()["ichunk"] > 0) == (lists or depth > 0)
            if not out:
                e0, h0 = rng.standard_normal(eng.n_E) * (b != 0), rng.standard_normal(eng.n_H)
            eng.set_fields(e0.astype(np.float32), h0.astype(np.float32), batch - 1)
            eng.step(5)
            out.append(eng.read_fields(batch - 1))
    assert all(np.all(np.isfinite(x)) and np.array_equal(x, y) for x, y in zip(*out))
