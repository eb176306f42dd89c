"""The default engine's choice between the frame kernel and the pass kernels,
and the stretch material's stress without an SVD.

A handle whose caller chose neither an engine nor a chunk shape runs the frame
kernel where every chunk has a resident CTA.  Its trajectories are the pass
kernels' (set_pass_engine("graph") on the same automatic chunks) bit for bit:
the residual stop is off and the regrouped energy sums do not flip a
line-search test on these meshes.
"""
import os

import numpy as np
import pytest

from oracle import restated as O
from phybs_gb300 import _lib as L
from phybs_gb300 import meshes as M
from phybs_gb300.solver import DescentSolver, make_params

pytestmark = pytest.mark.gpu

KEYS = ("passes", "iterations", "rejections", "converged", "status", "alpha", "rho", "omega", "graph_launches")


@pytest.fixture(scope="module", autouse=True)
def built():
    from phybs_gb300.build import build
    build()


def _box(nx, ny, nz):
    return M.box_mesh(nx, ny, nz, edge=0.25 / max(nx, ny), seed=nx, young=1e5)


# one tet; one cube (5); one chunk and a few more (120, 130, 180); around the 128 / 256 line
# (4,080, 4,160), 7,680, 8,320; one and two CTAs a SM of 256 tets (38,440, 60,000, 77,760); the
# pieces of 342 (78,000, 102,060); whole groups (104,780, 115,200, 119,000, 155,000); past
# the resident sizes (161,700: the pass kernels either way)
BOXES = [(1, 1, 1), (2, 3, 4), (2, 1, 13), (3, 3, 4), (8, 8, 24), (8, 8, 26), (31, 31, 8), (20, 20, 30),
         (24, 24, 40), (28, 25, 34), (31, 25, 40), (33, 28, 35), (8, 6, 17), (8, 8, 13), (24, 24, 27),
         (20, 20, 39), (27, 28, 27), (26, 26, 31)]


@pytest.mark.parametrize("dims", BOXES, ids=[f"{5 * a * b * c}" for a, b, c in BOXES])
@pytest.mark.parametrize("material,inc", [(0, 1), (0, 0), (1, 0)], ids=["incremental", "full", "stretch"])
def test_default_engine_equals_pass_kernels(dims, material, inc):
    m = _box(*dims)
    p = make_params("gpu_reference", h=1 / 30, max_iters=40, incremental_stress=inc)
    a = DescentSolver(m, params=p, material=material)
    b = DescentSolver(m, params=p, material=material)
    b.set_pass_engine("graph")
    for f in range(2):
        a.step()
        b.step()
        sa, sb = a.stats(), b.stats()
        assert [sa[k] for k in KEYS] == [sb[k] for k in KEYS], f
        assert np.array_equal(a.positions(), b.positions(), equal_nan=True), f
    a.close()
    b.close()


@pytest.mark.parametrize("cells", [820, 15560, 20790, 22000, 49000])
def test_meshes_with_many_nodes_a_tet(cells):
    """Strips one cell thick (0.8 nodes a tet): their chunks end at the node
    limits, so that there are more of them than of a box's at every line."""
    m = M.box_mesh(cells, 1, 1, edge=0.01, seed=2, young=1e5, pin="bottom")
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    alone, graph = DescentSolver(m, params=p), DescentSolver(m, params=p)
    graph.set_pass_engine("graph")
    packed = DescentSolver(_pack([_box(2, 1, 13), m, _box(8, 8, 12)]), params=p)
    n0 = 3 * 2 * 14
    for _ in range(2):
        for s in (alone, graph, packed):
            s.step(raise_on_error=False)
        assert np.array_equal(alone.positions(), graph.positions())
        assert np.array_equal(alone.positions(), packed.positions()[n0:n0 + m.n_nodes])
        assert alone.stats()["energy"] == graph.stats()["energy"] == packed.instance_stats(1)["energy"]
    for s in (alone, graph, packed):
        s.close()


def test_step_engine_is_the_one_that_ran():
    """What ran the passes, where the set engine (pass_engine) and the count of
    graph bodies do not tell."""
    for dims, want in (((8, 8, 24), "frame"), ((34, 34, 54), "graph")):
        s = DescentSolver(_box(*dims), params=make_params("gpu_reference", h=1 / 30, max_iters=8))
        assert s.step_engine() == s.pass_engine() == "graph"
        s.step()
        assert (s.step_engine(), s.pass_engine()) == (want, "graph") and s.stats()["graph_launches"] > 0
        s.set_pass_engine("graph")
        s.step()
        assert s.step_engine() == "graph"
        s.close()


@pytest.mark.parametrize("n", [1, 3])
def test_autotune_keeps_the_frame_kernel_where_it_is_faster(n):
    """A tuned handle of a size that the frame kernel steps in half the pass
    kernels' time goes on running it, with the bits of an untuned one; a chosen
    engine stays, and a body beyond residence gets a shape."""
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    m = _pack([_box(12, 12, 20)] * n)
    a, b = DescentSolver(m, params=p), DescentSolver(m, params=p)
    r = a.autotune(16)
    assert r["n_tried"] == 20 and 0 < r["pass_ms"] <= r["default_pass_ms"]
    for _ in range(2):
        a.step()
        b.step()
        assert a.step_engine() == "frame" and np.array_equal(a.positions(), b.positions())
    a.set_pass_engine("graph")
    a.autotune(4)
    a.step()
    assert a.step_engine() == "graph"
    a.close()
    b.close()
    s = DescentSolver(_box(34, 33, 46), params=p)
    s.autotune(4)
    s.step()
    assert s.step_engine() == "graph"
    s.close()


TEST_LARGE_STEPS = 2  # pbs_test_hook


def test_default_step_beside_others():
    """A step whose frame kernel takes more than half of the SMs runs the pass
    kernels when two such steps run already, with the same bits; smaller ones
    and a chosen engine stay."""
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    small, half, large = _box(8, 8, 12), _box(16, 14, 18), _box(20, 20, 30)  # 15, 79 and two CTAs a SM
    for m, others, want in ((small, 0, "frame"), (small, 7, "frame"), (half, 1, "frame"), (half, 2, "graph"),
                            (large, 1, "frame"), (large, 2, "graph")):
        a, b = DescentSolver(m, params=p), DescentSolver(m, params=p)
        b.set_pass_engine("graph")
        L.lib().pbs_test_hook(a._h, TEST_LARGE_STEPS, others)
        try:
            a.step()
        finally:
            L.lib().pbs_test_hook(a._h, TEST_LARGE_STEPS, -others)
        b.step()
        assert a.step_engine() == want
        assert np.array_equal(a.positions(), b.positions()) and a.stats()["energy"] == b.stats()["energy"]
        a.step()
        assert a.step_engine() == "frame"  # nothing is left counted
        a.close()
        b.close()


TEST_REFUSE_FRAME = 3  # pbs_test_hook


def test_refused_frame_kernel_leaves_the_pass_kernels():
    """A default step whose frame kernel cannot be resident after all runs the
    pass kernels; one that chose the frame engine reports the refusal."""
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    a, b = (DescentSolver(_box(8, 8, 12), params=p) for _ in range(2))
    for f in range(3):
        L.lib().pbs_test_hook(a._h, TEST_REFUSE_FRAME, int(f == 1))
        a.step()
        b.step()
        assert (a.step_engine(), b.step_engine()) == ("graph" if f == 1 else "frame", "frame")
        assert np.array_equal(a.positions(), b.positions()) and a.stats()["energy"] == b.stats()["energy"]
    a.set_pass_engine("frame")
    L.lib().pbs_test_hook(a._h, TEST_REFUSE_FRAME, 1)
    with pytest.raises(L.PhybsError):
        a.step()
    a.close()
    b.close()


IN_GREEN_CONTEXT = """
import ctypes as C, sys
cu = C.CDLL("libcuda.so.1")
def ok(rc):
    if rc:
        print("unavailable", rc)
        sys.exit(0)
dev, n = C.c_int(), C.c_uint(1)
full, part, rest = (C.create_string_buffer(144) for _ in range(3))  # CUdevResource
desc, green, ctx = C.c_void_p(), C.c_void_p(), C.c_void_p()
ok(cu.cuInit(0)); ok(cu.cuDeviceGet(C.byref(dev), 0))
ok(cu.cuDeviceGetDevResource(dev, full, 1))                                 # CU_DEV_RESOURCE_TYPE_SM
ok(cu.cuDevSmResourceSplitByCount(part, C.byref(n), full, rest, 0, 32))
ok(cu.cuDevResourceGenerateDesc(C.byref(desc), part, 1))
ok(cu.cuGreenCtxCreate(C.byref(green), desc, dev, 1))                       # CU_GREEN_CTX_DEFAULT_STREAM
ok(cu.cuCtxFromGreenCtx(C.byref(ctx), green)); ok(cu.cuCtxSetCurrent(ctx))
sms = int.from_bytes(part.raw[96:100], "little")
import numpy as np
from phybs_gb300 import meshes as M
from phybs_gb300.solver import DescentSolver, make_params
from phybs_gb300.warmstart import MLPTrainer
p = make_params("gpu_reference", h=1 / 30, max_iters=24)
out = {"sms": sms}
for name, n in (("small", (5, 4, 6)), ("large", (20, 20, 30))):
    m = M.box_mesh(*n, edge=0.25 / max(n[:2]), jitter=0.1, seed=2, young=1e5, pin="bottom")
    s = DescentSolver(m, params=p)
    s.step()
    out[name] = s.positions()
    out[name + "_engine"] = s.step_engine()
    s.backward_euler_step()
    out[name + "_be"] = s.positions()
    s.pd_step()
    out[name + "_pd"] = s.positions()
    s.close()
x = np.random.default_rng(0).standard_normal((9000, 24)).astype(np.float32)
t = MLPTrainer(seed=3)
t.set_data(x, np.tanh(x[:, :3]))
out["losses"] = t.train(4, batch=4096, seed=1)
t.close()
np.savez(sys.argv[1], **out)
print("done", sms)
"""


def test_in_a_context_with_fewer_sms(tmp_path):
    """Every default path in a green context of some of the SMs: grids fit it
    (the frame kernel where it does, else the pass kernels), and the results are
    those of the whole device: the descent's bit for bit, the solves' and the
    training's to the rounding of sums over another number of CTAs."""
    import subprocess
    import sys as _sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    f = str(tmp_path / "green.npz")
    r = subprocess.run([_sys.executable, "-c", IN_GREEN_CONTEXT, f], cwd=root, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    if r.stdout.startswith("unavailable"):
        pytest.skip("no green context here: " + r.stdout)
    g = np.load(f)
    assert 0 < g["sms"] < 152
    assert (str(g["small_engine"]), str(g["large_engine"])) == ("frame", "graph")
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    for name, n in (("small", (5, 4, 6)), ("large", (20, 20, 30))):
        m = M.box_mesh(*n, edge=0.25 / max(n[:2]), jitter=0.1, seed=2, young=1e5, pin="bottom")
        s = DescentSolver(m, params=p)
        s.step()
        assert np.array_equal(s.positions(), g[name])
        s.backward_euler_step()
        assert np.abs(s.positions() - g[name + "_be"]).max() <= 1e-5 * m.bbox_diagonal()
        s.pd_step()
        assert np.abs(s.positions() - g[name + "_pd"]).max() <= 1e-5 * m.bbox_diagonal()
        s.close()
    from phybs_gb300.warmstart import MLPTrainer
    x = np.random.default_rng(0).standard_normal((9000, 24)).astype(np.float32)
    t = MLPTrainer(seed=3)
    t.set_data(x, np.tanh(x[:, :3]))
    assert np.abs(t.train(4, batch=4096, seed=1) / g["losses"] - 1).max() <= 1e-5
    t.close()


@pytest.mark.parametrize("threads,tets", [(2, (9, 8, 13)), (8, (2, 1, 13)), (6, (12, 12, 20)), (4, (20, 20, 30)),
                                          (3, (28, 25, 34))])
def test_handles_stepped_from_threads(threads, tets):
    """Handles stepped from several threads at once, one each: every one's steps
    are those it takes by itself, whichever engine a step finds room for."""
    import threading
    p = make_params("gpu_reference", h=1 / 30, max_iters=40)
    meshes = [M.box_mesh(*tets, edge=0.25 / max(tets[:2]), jitter=0.1, seed=k, young=1e5) for k in range(threads)]
    want = []
    for m in meshes:
        s = DescentSolver(m, params=p)
        for _ in range(12):
            s.step()
        want.append((s.positions(), s.stats()["energy"]))
        s.close()
    got = [None] * threads
    start = threading.Barrier(threads)

    def run(k):
        s = DescentSolver(meshes[k], params=p)
        start.wait()
        for _ in range(12):
            s.step()
        got[k] = (s.positions(), s.stats()["energy"])
        s.close()

    ts = [threading.Thread(target=run, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g, w in zip(got, want):
        assert g is not None and np.array_equal(g[0], w[0]) and g[1] == w[1]


@pytest.mark.parametrize("n", [2, 5, 24])
def test_default_engine_packed(n):
    """Packed uneven boxes: resident (2, 5) and beyond (24); the iteration
    budget ends instances at different passes, some of them non-finite."""
    m = M.batch_of_boxes(n, seed=n, nxy=(4, 16), nz=(8, 32))
    p = make_params("gpu_reference", h=1 / 30, max_iters=64, alpha0=0.6, profile=((10, 0.9999),))
    a, b = DescentSolver(m, params=p), DescentSolver(m, params=p)
    b.set_pass_engine("graph")
    for f in range(2):
        a.step(raise_on_error=False)
        b.step(raise_on_error=False)
        for i in range(n):
            sa, sb = a.instance_stats(i), b.instance_stats(i)
            assert [sa[k] for k in KEYS[:8]] == [sb[k] for k in KEYS[:8]], (f, i)
        assert np.array_equal(a.positions(), b.positions(), equal_nan=True), f
    a.close()
    b.close()


def _pack(meshes):
    """Meshes as one packed handle's, in place (instances do not meet)."""
    nptr = np.cumsum([0] + [m.n_nodes for m in meshes]).astype(np.int32)
    tptr = np.cumsum([0] + [m.n_tets for m in meshes]).astype(np.int32)
    cat = lambda f: np.concatenate([f(m, int(o)) for m, o in zip(meshes, nptr)])
    return M.TetMeshData(cat(lambda m, o: m.rest), cat(lambda m, o: m.tets + o), cat(lambda m, o: m.pins + o),
                         cat(lambda m, o: np.broadcast_to(np.float32(m.young), m.n_tets)),
                         cat(lambda m, o: np.broadcast_to(np.float32(m.poisson), m.n_tets)),
                         instance_node_ptr=nptr, instance_tet_ptr=tptr, name="packed")


# bodies whose automatic chunks are of 128, 256 and 342 tets, whole groups
# (104,780; 260,100) and pieces of 342 beyond residence (161,700); what is said
# of a company is the pass kernels' CTA.  Copies keep a company from being resident
SMALL = [(2, 1, 13), (3, 5, 9), (8, 8, 12), (9, 8, 13), (12, 12, 20), (14, 13, 27)]
COMPANIES = {
    "resident": (SMALL, 1),
    "128 threads": (SMALL + [(24, 24, 27)], 12),
    "256 threads, pieces": (SMALL + [(24, 24, 28)], 8),
    "256 threads, groups": (SMALL + [(28, 25, 34), (26, 26, 31)], 3),
    "few groups": ([(26, 26, 31), (3, 5, 9)], 2),
    "largest": ([(34, 30, 51), (8, 8, 12), (33, 28, 35)], 1),
}


@pytest.mark.parametrize("company", COMPANIES)
@pytest.mark.parametrize("control", ["stop", "budget"])
@pytest.mark.parametrize("material,inc", [(0, 1), (0, 0), (1, 0)], ids=["incremental", "full", "stretch"])
def test_packed_instance_equals_the_body_alone(company, control, material, inc):
    """A body takes the same steps alone (the frame kernel, where its chunks are
    resident) and in any company (the pass kernels, at the company's CTA size):
    decisions, sums and positions bit for bit, with a stop on the residual and
    with the reference's line search at an iteration budget."""
    dims, copies = COMPANIES[company]
    meshes = [_box(*d) for d in dims]
    if control == "stop":
        p = make_params("gpu_reference", h=1 / 30, tol=3e-2, max_iters=2000, control=L.PBS_CONTROL_RESTART,
                        energy_slack=16.0, alpha0=0.45, alpha_grow=1.2, incremental_stress=inc,
                        profile=((5, 0.99), (25, 0.999), (100, 0.9999)))
    else:
        p = make_params("gpu_reference", h=1 / 30, max_iters=72, alpha0=0.6, profile=((10, 0.9999),),
                        incremental_stress=inc)
    packed = _pack(meshes * copies)
    s = DescentSolver(packed, params=p, material=material)
    keys = KEYS[:8] + ("energy", "residual_ratio")
    got = []
    for f in range(2):
        s.step(raise_on_error=False)
        x = s.positions()
        got.append([(s.instance_stats(i), x[packed.instance_node_ptr[i]:packed.instance_node_ptr[i + 1]])
                    for i in range(packed.n_instances)])
    s.close()
    for j, m in enumerate(meshes):
        a = DescentSolver(m, params=p, material=material)
        for f in range(2):
            a.step(raise_on_error=False)
            st, x = a.stats(), a.positions()
            for i in range(j, packed.n_instances, len(meshes)):
                sp, xp = got[f][i]
                assert repr([sp[k] for k in keys]) == repr([st[k] for k in keys]), (dims[j], f, i)
                assert np.array_equal(x, xp, equal_nan=True), (dims[j], f, i)
        a.close()


@pytest.mark.parametrize("engine", [None, "graph"])
@pytest.mark.parametrize("at", [0, 1, 2], ids=["first", "middle", "last"])
@pytest.mark.parametrize("inc", [0, 1], ids=["full", "incremental"])
def test_packed_instance_without_tets(engine, at, inc):
    """A packed instance of three nodes and no tets changes nothing for the
    others, wherever it lies (as the last one its chunk's records are past the
    table's end)."""
    m = M.batch_of_boxes(2, seed=4, nxy=(4, 6), nz=(8, 12))
    cut = m.instance_node_ptr[at]
    rest = np.insert(m.rest, [cut] * 3, [[9, 0, 0], [9, 1, 0], [9, 0, 1]], axis=0).astype(np.float32)
    up = lambda i: np.where(i >= cut, i + 3, i)
    nptr = np.insert(m.instance_node_ptr, at + 1, cut + 3)
    nptr[at + 2:] += 3
    tptr = np.insert(m.instance_tet_ptr, at + 1, m.instance_tet_ptr[at])
    e = M.TetMeshData(rest, up(m.tets), up(m.pins), m.young, m.poisson, instance_node_ptr=nptr.astype(np.int32),
                      instance_tet_ptr=tptr.astype(np.int32), name="with an empty instance")
    p = make_params("gpu_reference", h=1 / 30, max_iters=40, incremental_stress=inc)
    x = []
    for mesh in (m, e):
        s = DescentSolver(mesh, params=p)
        if engine:
            s.set_pass_engine(engine)
        s.step()
        s.step()
        x.append(s.positions())
        s.close()
    assert np.array_equal(x[0], np.delete(x[1], np.arange(cut, cut + 3), axis=0))


def test_single_tet_and_loose_nodes():
    """One tet, and nodes that no tet touches (more than a CTA has threads)."""
    x = np.random.default_rng(0).uniform(0, 1, (400, 3)).astype(np.float32)
    x[:4] = [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]
    m = M.TetMeshData(x, np.array([[0, 1, 2, 3]]), np.array([0]), 1e4, 0.3)
    p = make_params("gpu_reference", h=1 / 30, max_iters=24)
    a, b = DescentSolver(m, params=p), DescentSolver(m, params=p)
    b.set_pass_engine("graph")
    # a loose node has no mass: its update is 0 / 0, and the step ends non-finite
    ra, rb = a.step(raise_on_error=False), b.step(raise_on_error=False)
    assert (ra, a.last_status) == (rb, b.last_status)
    assert np.array_equal(a.positions(), b.positions(), equal_nan=True)
    a.close()
    b.close()


# principal stretches on both sides of the 2 det F >= 0.31 |F|^2 line, and of
# sigma_3 = 0.3 beyond it
STRETCHES = [(1.0, 1.0, 1.0), (2.2, 0.7, 0.7), (3.0, 0.6, 0.6), (0.95, 0.95, 0.32), (0.95, 0.95, 0.36), (1.5, 1.5, 0.25),
             (0.5, 0.5, 0.5), (2.0, 2.0, 2.0)]


@pytest.mark.parametrize("s", STRETCHES)
def test_stretch_stress_without_svd(s):
    """One iteration of the stretch material from a stretched, wobbling state
    against the FP64 restatement (the SVD of every tet).  The velocity after it
    is 0.99 alpha g / (H h): g within the 1e-5 bar of assembled forces, H's
    closed form within another 1e-5, so 3e-5 of the largest velocity."""
    m = M.box_mesh(5, 4, 6, edge=0.05, seed=3, young=1e5, pin="bottom")
    x = m.rest.astype(np.float64)
    x = x * np.array(s) + 0.002 * np.sin(40 * x[:, [1, 2, 0]])
    x[m.pins] = m.rest[m.pins] * np.array(s, np.float32)
    x = x.astype(np.float32)
    p = make_params("gpu_reference", h=1 / 30, max_iters=1, alpha0=0.05)
    a = DescentSolver(m, positions=x, material=L.PBS_MATERIAL_STRETCH, params=p)
    a.step()
    mu, lam = O.lame(m.young, m.poisson)
    pm = m.pin_mask()
    r64 = O.rest(m.rest, m.tets, pm, prec=64)
    st = O.StepState(x)
    O.step(st, O.make_params(h=1 / 30, max_iters=1, alpha0=0.05, body_force_scale=1.0, energy_clamp=1, material=1,
                             hessian_closed=1), m.tets, r64, mu, lam, pm, prec=64)
    v = a.velocities()[0]
    assert np.abs(v - st.v).max() <= 3e-5 * np.abs(st.v).max(), np.abs(v - st.v).max() / np.abs(st.v).max()
    a.close()


def test_stretch_stress_under_rotation():
    """One iteration of the stretch material (lambda = 100 mu) from 48 bodies
    turned about random axes and strained by up to 1.4% at constant volume,
    against the FP64 restatement; the velocities' error in units of the ln J
    that makes it (from a second restatement, of the body scaled by 1.001).
    Grid, deformation and G are exact in FP32.  What rounds at the size of the
    rotation are the nine terms of tr E, 2^-25 / sqrt(3) each and half of it in
    ln J: 2.6e-8 together, and the bound on the root mean square over the bodies
    is twice that.  A det F - 1 summed from G's invariants is off by 1.3e-7."""
    from scipy.spatial.transform import Rotation
    cube = M.box_mesh(4, 4, 5, edge=0.0625, jitter=0.0, seed=3, young=1e7, poisson=0.49, pin="bottom")
    x = []
    for k in range(48):
        s = 1 + (k % 7 + 1) / 512
        F = np.round(2**14 * Rotation.random(random_state=k).as_matrix() @ np.diag([s, 1 / s, 1])) / 2**14
        x.append((cube.rest.astype(np.float64) @ F.T).astype(np.float32))
        assert np.array_equal(x[-1], cube.rest.astype(np.float64) @ F.T)
    p = make_params("gpu_reference", h=1 / 30, max_iters=1, alpha0=0.05)
    a = DescentSolver(_pack([cube] * 48), positions=np.concatenate(x), material=L.PBS_MATERIAL_STRETCH, params=p)
    a.step()
    v = a.velocities()[0].reshape(48, -1, 3)
    a.close()
    pm = cube.pin_mask()
    r64 = O.rest(cube.rest, cube.tets, pm, prec=64)

    def exact(x0):
        st = O.StepState(x0)
        O.step(st, O.make_params(h=1 / 30, max_iters=1, alpha0=0.05, body_force_scale=1.0, energy_clamp=1, material=1,
                                 hessian_closed=1), cube.tets, r64, *O.lame(cube.young, cube.poisson), pm, prec=64)
        return st.v[pm == 0]

    err = []
    for k in range(48):
        e = exact(x[k])
        per_ln_j = np.abs(exact(np.float32(1.001) * x[k]) - e).max() / 3e-3
        err.append(np.abs(v[k][pm == 0] - e).max() / per_ln_j)
    assert np.sqrt(np.square(err).mean()) <= 2 * 2.6e-8, np.sqrt(np.square(err).mean())


PULLS = [(3, 3, 5), (8, 7, 12), (12, 9, 13), (20, 17, 31), (22, 21, 40), (25, 25, 40), (31, 23, 46), (34, 33, 46)]


@pytest.mark.parametrize("dims", PULLS, ids=[f"{5 * a * b * c}" for a, b, c in PULLS])
def test_pull_takes_one_path_at_every_chunk_size(dims):
    """Two frames of a pull to a residual of 1e-4 on the automatic chunks (one
    group and less, pieces of 128, 256, 342, whole groups, pieces of 342,
    whole groups) and on whole groups of 1,024:
    the tets' forces have the same bits, so that the passes and rejections are
    the same, and the positions to the sums' rounding."""
    m = M.box_mesh(*dims, edge=0.25 / max(dims[:2]), jitter=0.1, seed=7, young=1e5, pin="both")
    p = make_params("gpu_reference", h=1 / 30, tol=1e-4, max_iters=20000, control=L.PBS_CONTROL_RESTART,
                    energy_slack=16.0, alpha0=0.45, alpha_grow=1.2,
                    profile=((5, 0.99), (25, 0.999), (100, 0.9999)))
    z = m.rest[:, 2]
    bottom = np.nonzero(z <= z.min() + 1e-9)[0].astype(np.int32)
    down = np.float32([0, 0, 0.5 * float(z.max() - z.min()) / 30])
    out = []
    for shape in (None, (256, 1024, 448)):
        s = DescentSolver(m, params=p)
        if shape:
            s.set_chunk_shape(*shape)
        its = []
        for f in range(2):
            s.set_node_positions(bottom, m.rest[bottom] - (f + 1) * down)
            its.append((s.step(), s.stats()["rejections"]))
        out.append((its, s.positions()))
        s.close()
    assert out[0][0] == out[1][0]
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-6 * m.bbox_diagonal()


@pytest.mark.parametrize("staged,threads,tets,nodes", [(1, 256, 1388, 420), (2, 256, 866, 300), (0, 512, 2400, 1066)])
@pytest.mark.parametrize("inc", [0, 1])
def test_shapes_without_room_for_padding(staged, threads, tets, nodes, inc):
    """Shapes at the shared-memory limit, whose slot runs stay unpadded (or, not
    staged, just fit padded), against the same chunks at the limits' other side
    of the choice: bit for bit."""
    m = _box(20, 20, 30)
    p = make_params("gpu_reference", h=1 / 30, max_iters=24, incremental_stress=inc)
    x = []
    for st, th in ((staged, threads), (0, 256)):
        s = DescentSolver(m, params=p)
        s.set_chunk_shape(th, tets, nodes, st)
        s.step()
        x.append(s.positions())
        s.close()
    assert np.array_equal(x[0], x[1])


@pytest.mark.parametrize("inc", [0, 1])
def test_frame_engine_on_automatic_chunks_beyond_residence(inc):
    """A body whose automatic chunks run with 512 threads in the pass kernels
    takes the frame engine too, with the same bits; a caller's 512-thread shape
    stays refused."""
    m = _box(34, 33, 46)
    p = make_params("gpu_reference", h=1 / 30, max_iters=24, incremental_stress=inc)
    x = []
    for engine in ("graph", "frame"):
        s = DescentSolver(m, params=p)
        s.set_pass_engine(engine)
        s.step()
        x.append(s.positions())
        if engine == "frame":
            s.set_chunk_shape(512, 1024, 448)
            with pytest.raises(L.PhybsError):
                s.step()
        s.close()
    assert np.array_equal(x[0], x[1])
