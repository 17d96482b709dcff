"""The march kernel (plfbs_run on a mesh that fits one tile per SM) against the
same RK stages run one kernel at a time (plfbs_run_stages): the arithmetic and
the order of every sum are the same, so states, residual records, gradients and
fluxes agree bit for bit, over cell counts at the edges of the tiles, both
precisions and flavours, with and without the compact layout, and where the
context halts in the middle of a march."""

import threading

import numpy as np
import pytest

from plfbs import capi, cases

pytestmark = pytest.mark.gpu

STEPS = 5


def _mesh(kind, n):
    sides = ["inlet", "outlet", "side", "side", "side", "side"]
    if kind == "tets":
        pm = cases.jittered_tet_box(n[0], jitter=0.1, seed=3, patch_types=["side"] * 6)
    elif kind == "graded":
        grid = [np.concatenate([[0.0], np.cumsum(1.03 ** np.arange(k))]) for k in n]
        pm = cases.hex_box(*grid, patch_types=sides)
    else:
        pm = cases.uniform_box(*n, patch_types=sides)
    c = cases.Case(mesh_dir="", X=n[0], Y=n[1], Z=n[2], dt=0.05, mach=0.05, reynolds=50.0,
                   ref_length=4.0,
                   bcs=[cases.BC("inlet", 1, 1, 0, 0, "dirichlet", "neumann"),
                        cases.BC("outlet", 1, 0, 0, 0, "neumann", "dirichlet"),
                        cases.BC("side", 1, 0, 0, 0, "dirichlet", "neumann")])
    return cases.mesh_arrays(pm, c.visc, c.gamma, c.fneq_min), c


def _solver(ma, c, precision, flavour, renumber, tolerance=0.0):
    rt, vt, val = cases.bc_arrays(ma, c)
    cfg = dict(visc=c.visc, dt=c.dt, max_velocity=c.mach, channel_height=c.Y,
               lengths=(c.X, c.Y, c.Z), renumber=renumber, flavour=flavour, precision=precision,
               pressure_gradient=1e-5, tolerance=tolerance,
               gradient_mode=capi.GRAD_LS | capi.GRAD_EXACT_INVERSE)
    return capi.Solver(ma, rt, vt, val, cfg)


def _start(ma):
    rng = np.random.default_rng(2)
    q = np.zeros((ma.total_cells, 4))
    q[:, 0] = 0.04 + 0.002 * rng.standard_normal(ma.total_cells)
    q[:, 1:3] = 0.002 * rng.standard_normal((ma.total_cells, 2))
    q[:, 3] = 1.0 + 0.001 * rng.standard_normal(ma.total_cells)
    return q


def _same(ma, c, precision, flavour, renumber, compress=None):
    out = []
    for march in (True, False):
        s = _solver(ma, c, precision, flavour, renumber)
        if compress is not None:
            s.set_layout_compression(compress)
        s.set_state(_start(ma))
        if march:
            _, h = s.run(STEPS)
        else:
            s.run_stages(4 * STEPS)
            h = None
        grad, flux, state = s.gradients(), s.face_flux(), s.get_state()
        _, h2 = s.run(1)  # carries on from either
        out.append((grad, flux, state, h2, s.get_state()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert np.isfinite(out[0][2]).all()


# 1 cell; one tile of 32 and one cell more; one tile per SM of 32 and one cell
# more (148 SMs); several rounds of faces per block; a ragged last tile
@pytest.mark.parametrize("n", [(1, 1, 1), (8, 4, 1), (11, 3, 1), (37, 16, 8), (421, 9, 1),
                               (41, 29, 23), (40, 40, 41)])
@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32_DEVIATION])
def test_march_is_the_stages_boxes(plfbs_lib, n, precision):
    ma, c = _mesh("box", n)
    _same(ma, c, precision, capi.FLAVOUR_GPU, 0)


@pytest.mark.parametrize("kind,n", [("tets", (2, 2, 2)), ("tets", (11, 11, 11)),
                                    ("graded", (13, 11, 9)), ("box", (24, 20, 18))])
@pytest.mark.parametrize("precision,flavour", [(capi.FP64, capi.FLAVOUR_GPU),
                                               (capi.FP64, capi.FLAVOUR_CPU_SOLVER),
                                               (capi.FP32_DEVIATION, capi.FLAVOUR_GPU)])
@pytest.mark.parametrize("renumber", [0, 1])
def test_march_is_the_stages(plfbs_lib, kind, n, precision, flavour, renumber):
    ma, c = _mesh(kind, n)
    _same(ma, c, precision, flavour, renumber, 0 if kind == "box" else None)


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32_DEVIATION])
def test_march_halts_at_the_step(plfbs_lib, precision):
    """A tolerance that the residual passes after a few steps: the march stops
    with that step's state, and a march of one step at a time does the same."""
    ma, c = _mesh("box", (12, 10, 9))
    s = _solver(ma, c, precision, capi.FLAVOUR_GPU, 0)
    s.set_state(_start(ma))
    _, h = s.run(40)
    tol = float(h[17:20, 1].min())
    assert (h[:17, 1] > tol).all()
    first = int(np.argmax(h[:, 1] < np.nextafter(tol, 1)))
    s.close()
    out = []
    for chunk in (40, 1):
        s = _solver(ma, c, precision, capi.FLAVOUR_GPU, 0, tolerance=np.nextafter(tol, 1))
        s.set_state(_start(ma))
        for _ in range(40 // chunk):
            st, _ = s.run(chunk)
        assert st["converged"] and st["steps_done"] == first + 1
        out.append(s.get_state())
        s.close()
    np.testing.assert_array_equal(out[0], out[1])


def test_march_timed_out_leaves_no_old_gradients(plfbs_lib):
    """A march whose wait ran out has still replaced the state that the
    gradients and fluxes are read from."""
    ma, c = _mesh("box", (12, 10, 9))
    out = []
    for timed_out in (True, False):
        s = _solver(ma, c, capi.FP64, capi.FLAVOUR_GPU, 0)
        s.set_state(_start(ma))
        s.run_stages(4)
        if timed_out:
            s.set_timeout(1e-6)
            with pytest.raises(capi.PlfbsError) as e:
                s.run(300, history=False)
            assert e.value.code == capi.ERR_TIMEOUT
            assert s.wait(120.0)
        else:
            s.run(300, history=False)
        out.append((s.gradients(), s.face_flux(), s.get_state()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [(11, 3, 1), (37, 16, 8)])  # 2 tiles; one per SM
def test_march_beside_other_runs(plfbs_lib, n):
    """Runs on several threads take the march or the step graph batch by batch,
    by what else is in flight: the same bits as the run alone."""
    ma, c = _mesh("box", n)
    out = [None] * 4

    def solve(k, calls):
        s = _solver(ma, c, capi.FP64, capi.FLAVOUR_GPU, 0)
        s.set_state(_start(ma))
        h = [s.run(30)[1] for _ in range(calls)]
        out[k] = (np.concatenate(h), s.gradients(), s.face_flux(), s.get_state())
        s.close()

    solve(0, 10)
    threads = [threading.Thread(target=solve, args=(k, 10)) for k in (1, 2, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (1, 2, 3):
        for a, b in zip(out[0], out[k]):
            np.testing.assert_array_equal(a, b)


def test_march_tiles_of_different_sizes_on_three_threads(plfbs_lib):
    """The largest dynamic shared memory of a kernel is one value per device:
    meshes whose tiles take different amounts, one of them more than the 48 KB a
    kernel has without asking, and fit on the SMs together (144, 2 and 2 of 148)
    march on three threads in many short runs."""
    errs, out = [], {}

    def solve(n, runs, key):
        try:
            ma, c = _mesh("box", n)
            s = _solver(ma, c, capi.FP64, capi.FLAVOUR_GPU, 0)
            s.set_state(_start(ma))
            for _ in range(runs):
                s.run(1, history=False)
            out[key] = s.get_state()
            s.close()
        except capi.PlfbsError as e:
            errs.append((n, repr(e)))

    meshes = [(24, 24, 24), (11, 3, 1), (1, 33, 1)]
    for n in meshes:
        solve(n, 4000, n)
    threads = [threading.Thread(target=solve, args=(n, 4000, n + (0,))) for n in meshes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errs, errs
    for n in meshes:
        np.testing.assert_array_equal(out[n], out[n + (0,)])


def _same_run(ma, c, precision, flavour, want_compact, mode=None, compress=None, ibm=None,
              exact=True):
    """As _same, on given mesh arrays (want_compact: whether the face records and
    the weight sets of the layout repeat) and with an immersed body."""
    out = []
    for march in (True, False):
        rt, vt, val = cases.bc_arrays(ma, c)
        cfg = dict(visc=c.visc, dt=c.dt, max_velocity=c.mach, channel_height=c.Y,
                   lengths=(c.X, c.Y, c.Z), flavour=flavour, precision=precision,
                   pressure_gradient=1e-5, domain_dt=0.5,
                   gradient_mode=mode or (capi.GRAD_LS | capi.GRAD_EXACT_INVERSE))
        s = capi.Solver(ma, rt, vt, val, cfg, ibm=ibm)
        got = s.layout()["compact"]
        assert (got[0] > 0, got[1] > 0) == want_compact, got
        if all(want_compact):
            assert max(got) > 32  # not the form with the tables in shared memory
        if compress is not None:
            s.set_layout_compression(compress)
        s.set_state(_start(ma))
        if march:
            s.run(STEPS)
        else:
            s.run_stages(4 * STEPS)
        out.append((s.gradients(), s.face_flux(), s.get_state()) + (s.nodes() if ibm else ()))
        s.close()
    assert np.isfinite(out[0][2]).all()
    for a, b in zip(*out):
        if exact:
            np.testing.assert_array_equal(a, b)
        else:  # atomic sums of the body's forces in any order
            tol = 1e-12 if precision == capi.FP64 else 2e-5
            np.testing.assert_allclose(a, b, rtol=0, atol=tol * max(1.0, np.abs(b).max()))


FORMS = [(capi.FP64, capi.FLAVOUR_GPU), (capi.FP64, capi.FLAVOUR_CPU_SOLVER),
         (capi.FP32_DEVIATION, capi.FLAVOUR_GPU)]


# the compact layout with more records than the shared-memory tables take (along
# each axis), and with only the face records or only the weight sets repeating
@pytest.mark.parametrize("form", ["x", "y", "z", "faces", "weights"])
@pytest.mark.parametrize("precision,flavour", FORMS)
def test_march_is_the_stages_compact_forms(plfbs_lib, form, precision, flavour):
    n, mode = (21, 22, 23), None
    grid = [np.arange(k + 1.0) for k in n]
    if form in "xyz":
        k = "xyz".index(form)
        grid[k] = np.concatenate([[0.0], np.cumsum(1 + np.arange(n[k]) / 64)])  # exact sums
    sides = ["inlet", "outlet", "side", "side", "side", "side"]
    c = _mesh("box", (2, 2, 2))[1]
    ma = cases.mesh_arrays(cases.hex_box(*grid, patch_types=sides), c.visc, c.gamma, c.fneq_min)
    rng = np.random.default_rng(7)
    want = (True, True)
    if form == "weights":  # every face a streaming time of its own
        ma.streaming_dt = np.asarray(ma.streaming_dt) * rng.uniform(0.9, 1.0, len(ma.streaming_dt))
        want = (False, True)
    if form == "faces":  # every cell a hybrid weight of its own
        ma.cell_volume = np.array(ma.cell_volume) * rng.uniform(0.9, 0.99, len(ma.cell_volume))
        mode, want = capi.GRAD_HYBRID | capi.GRAD_EXACT_INVERSE, (True, False)
    _same_run(ma, c, precision, flavour, want, mode)


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32_DEVIATION])
@pytest.mark.parametrize("nodes", [1, 60])
def test_march_is_the_stages_with_a_body(plfbs_lib, precision, nodes):
    """The body's nodes inside a march: one node, whose eight cells get a force
    each, to the bit, and a sphere to the rounding of its atomic sums."""
    c = _mesh("box", (2, 2, 2))[1]
    n = (24, 16, 16)
    c.X, c.Y, c.Z = n
    grid = [np.arange(k + 1.0) for k in n]
    grid[2] = np.concatenate([[0.0], np.cumsum(1 + np.arange(n[2]) / 1024)])
    ma = cases.mesh_arrays(cases.hex_box(*grid, patch_types=["inlet", "outlet"] + ["side"] * 4),
                           c.visc, c.gamma, c.fneq_min)
    x = cases.fibonacci_sphere(nodes, 2.0, (8.0, 8.0, 8.0))
    ibm = dict(node_ref=x, stiffness=0.5, radius=2.0, depth=4.0, object_nodes=max(nodes, 2))
    _same_run(ma, c, precision, capi.FLAVOUR_GPU, (True, True), ibm=ibm, exact=nodes == 1)


def test_march_gives_way_to_a_network_pass(plfbs_lib):
    """A march holds its SMs for many steps: it has to stop for another call of the
    library (a pass waited for the march's launch, some 30 times its own time), and
    carry on to the same bits."""
    import time

    from plfbs import gnn

    ma, c = _mesh("box", (64, 32, 32))
    steps, out = 4000, {}

    def solve(key):
        s = _solver(ma, c, capi.FP64, capi.FLAVOUR_GPU, 0)
        s.set_state(_start(ma))
        _, h = s.run(steps)
        out[key] = (h, s.gradients(), s.face_flux(), s.get_state())
        s.close()

    g, _ = _mesh("box", (16, 16, 16))
    src, dst, ef = gnn.mesh_graph(g)
    net = gnn.GraphNet(src, dst, ef, g.n_cells, 9, 4, 4)
    net.set_params(gnn.init_params(9, ef.shape[1], 4, 4, seed=1))
    x = np.random.default_rng(1).standard_normal((g.n_cells, 9)).astype(np.float32)

    def passes(n):
        t = []
        for _ in range(n):
            t0 = time.perf_counter()
            y = net.forward(x)
            t.append(time.perf_counter() - t0)
        return float(np.median(t)), y

    solve("alone")
    passes(3)
    alone, y0 = passes(20)
    t = threading.Thread(target=solve, args=("beside",))
    t.start()
    time.sleep(0.1)
    beside, y1 = passes(20)
    t.join()
    net.close()
    np.testing.assert_array_equal(y0, y1)
    for a, b in zip(out["alone"], out["beside"]):
        np.testing.assert_array_equal(a, b)
    assert beside < 8 * alone, (alone, beside)


def test_timed_out_march_gives_way(plfbs_lib):
    """Steps of a timed-out run still hold their SMs: another context's run counts
    them, and they give way to it. Both carry on to the bits of a run alone."""
    import time

    ma, c = _mesh("box", (64, 32, 32))
    steps = 2048

    def fresh():
        s = _solver(ma, c, capi.FP64, capi.FLAVOUR_GPU, 0)
        s.set_state(_start(ma))
        s.run(3, history=False)
        return s

    s = fresh()
    t0 = time.perf_counter()
    s.run(steps, history=False)
    full = time.perf_counter() - t0  # some 140 ms
    want = s.get_state()
    s.close()
    a, b = fresh(), fresh()
    a.set_timeout(1e-6)
    with pytest.raises(capi.PlfbsError) as e:
        a.run(steps, history=False)
    assert e.value.code == capi.ERR_TIMEOUT
    t0 = time.perf_counter()
    b.run(30, history=False)
    beside = time.perf_counter() - t0
    assert a.wait(120.0)
    a.set_timeout(0.0)
    done = a.run(0, history=False)[0]["steps_done"]
    assert 3 < done <= steps + 3
    a.run(steps + 3 - done, history=False)
    b.run(steps - 30, history=False)
    np.testing.assert_array_equal(a.get_state(), want)
    np.testing.assert_array_equal(b.get_state(), want)
    a.close()
    b.close()
    assert beside < full / 3, (beside, full)


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32_DEVIATION])
def test_fluxes_of_a_march_leave_the_wall_forces_gradients(plfbs_lib, precision):
    """The fluxes of a march are recomputed when asked for, by way of gradients: those
    that a wall-force call has left since, and the state set after it (its ghosts
    among it), stay as they were."""
    ma, c = _mesh("box", (12, 10, 9))
    q = 0.5 * _start(ma)[::-1].copy()
    q[:, 3] += 0.5
    out = []
    for march in (True, False):
        s = _solver(ma, c, precision, capi.FLAVOUR_GPU, 0)
        s.set_state(_start(ma))
        if march:
            s.run(STEPS)
        else:
            s.run_stages(4 * STEPS)
        s.wall_forces([0, 1, 2])
        s.set_state(q)
        state = s.get_state()
        out.append((s.face_flux(), s.gradients(), s.get_state()))
        np.testing.assert_array_equal(out[-1][2], state)
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
