"""GPU parity of the backward-Euler step (pbs_backward_euler_step) through the
C ABI against the FP64 restatement (oracle/implicit.py: the reference's
doBackEuler system, CUDAInterface.cu:784-884, with a direct sparse solve).

Bar: positions after a step within 1e-4 of the bounding-box diagonal of the
restatement's (the path's position bar), the CG residual below its tolerance,
bit-reproducible runs."""
import numpy as np
import pytest

from oracle import implicit as I
from oracle import restated as O
from phybs_gb300 import _lib as L
from phybs_gb300 import meshes as M
from phybs_gb300.solver import DescentSolver

pytestmark = pytest.mark.gpu

POS_TOL = 1e-4


@pytest.fixture(scope="module", autouse=True)
def built():
    from phybs_gb300.build import build
    build()


def twisted_bar():
    m = M.bar_mesh(10, 4, 4, edge=0.025, young=5e4, poisson=0.4)
    x0 = M.twist_positions(m.rest, 0.5, axis=0)
    x0[m.pins] = m.rest[m.pins]
    return m, x0


@pytest.mark.parametrize("material", [L.PBS_MATERIAL_NEOHOOKEAN, L.PBS_MATERIAL_STRETCH])
def test_steps_match_restatement(material):
    """Five steps from a twisted bar (x = 0 pinned, gravity), each compared with
    one restated FP64 step from the GPU's state."""
    m, x0 = twisted_bar()
    mu, lam = O.lame(m.young, m.poisson)
    s = DescentSolver(m, positions=x0, material=material, mu=mu, lam=lam)
    diag = m.bbox_diagonal()
    x, v = s.positions(), s.velocities()[0]
    for k in range(5):
        xo, vo, _, _ = I.backward_euler_step(x, v, m.rest, m.tets, m.pin_mask(), mu, lam, material=material)
        it, res = s.backward_euler_step(tol=1e-6)
        assert res <= 1e-6 and it > 0
        x, v = s.positions(), s.velocities()[0]
        err = np.abs(x - xo).max() / diag
        assert err < POS_TOL, (k, err, it, res)
        assert np.abs(x[m.pins] - m.rest[m.pins]).max() < 1e-6
    # the bar untwists and sags
    assert np.abs(x - x0).max() > 1e-3 * diag
    s.close()


def test_box_step_with_external_forces():
    """A 12 x 12 x 20 box (14,400 tets), top pinned, gravity plus a lateral pull
    on the bottom face, against the restatement."""
    m = M.box_mesh(12, 12, 20, edge=0.01, seed=3, young=2e5, poisson=0.4)
    mu, lam = O.lame(m.young, m.poisson)
    ext = np.zeros_like(m.rest)
    bottom = m.rest[:, 2] <= m.rest[:, 2].min() + 1e-6
    ext[bottom, 0] = 0.02
    s = DescentSolver(m, mu=mu, lam=lam)
    x, v = s.positions(), s.velocities()[0]
    xo, vo, _, _ = I.backward_euler_step(x, v, m.rest, m.tets, m.pin_mask(), mu, lam, ext=ext, h=1 / 30)
    it, res = s.backward_euler_step(dt=1 / 30, ext=ext, tol=1e-6)
    assert res <= 1e-6
    assert np.abs(s.positions() - xo).max() / m.bbox_diagonal() < POS_TOL
    assert np.abs(s.velocities()[0] - vo).max() <= 1e-3 * np.abs(vo).max()
    s.close()


def test_bitwise_reproducible_and_iteration_cap():
    m, x0 = twisted_bar()
    out = []
    for _ in range(2):
        s = DescentSolver(m, positions=x0)
        for _ in range(2):
            s.backward_euler_step()
        out.append(s.positions())
        s.close()
    assert np.array_equal(out[0], out[1])
    s = DescentSolver(m, positions=x0)
    it, res = s.backward_euler_step(max_iters=2, raise_on_cap=False)
    assert s.last_status == L.PBS_E_ITER_CAP and it == 2 and res > 1e-6
    assert not np.array_equal(s.positions(), x0)  # the last iterate was applied
    with pytest.raises(L.PhybsError):
        s.backward_euler_step(dt=-1.0)
    s.close()


# rows about the slice and CTA lines: 4 nodes; 12; 32 rows to a slice; 126,
# 128, 135 (a second CTA); 3,000 over two dozen CTAs; rows of 27 columns
# (6-tet split) and of 7 and 19 in turn (5-tet)
GRIDS = [(5, 1, 1, 1), (5, 1, 1, 2), (5, 1, 3, 3), (6, 2, 5, 6), (5, 3, 3, 7), (6, 2, 4, 8), (5, 9, 14, 19)]


def _moving(split, nx, ny, nz):
    """A twisted mesh held at its untwisted end, and its velocities: states
    whose matrix is positive definite (checked on the CPU for the small ones)."""
    if split == 6:
        m, axis = M.bar_mesh(nx, ny, nz, edge=0.03, young=5e4, poisson=0.4), 0
    else:
        m, axis = M.box_mesh(nx, ny, nz, edge=0.03, young=5e4, poisson=0.4, pin="bottom"), 2
    x0 = M.twist_positions(m.rest, 0.15, axis=axis)
    v0 = (0.1 * np.sin(20 * m.rest[:, [1, 2, 0]])).astype(np.float32)
    v0[m.pins] = 0.0
    return m, x0, v0


@pytest.mark.parametrize("split,nx,ny,nz", GRIDS)
def test_solve_sizes_match_restatement(split, nx, ny, nz):
    """One backward-Euler step of meshes of every row count near the solve's
    lines, twisted and moving, against the FP64 restatement."""
    m, x0, v0 = _moving(split, nx, ny, nz)
    mu, lam = O.lame(m.young, m.poisson)
    s = DescentSolver(m, positions=x0, mu=mu, lam=lam)
    s.write_velocities(v0, v0)
    xo, vo, _, _ = I.backward_euler_step(s.positions(), v0, m.rest, m.tets, m.pin_mask(), mu, lam)
    it, res = s.backward_euler_step(tol=1e-6)
    assert res <= 1e-6
    assert np.abs(s.positions() - xo).max() / m.bbox_diagonal() < POS_TOL
    assert np.abs(s.velocities()[0] - vo).max() <= 1e-3 * np.abs(vo).max()
    s.close()


@pytest.mark.parametrize("scale", [1e-4, 1e3])
def test_solve_scales(scale):
    """The same bar a ten-thousandth and a thousand times its size (masses and
    residuals by the cube): the sums' scaling keeps the solve's tolerance."""
    m = M.bar_mesh(6, 3, 3, edge=0.025 * scale, young=5e4, poisson=0.4)
    x0 = M.twist_positions(m.rest, 0.4, axis=0)
    x0[m.pins] = m.rest[m.pins]
    mu, lam = O.lame(m.young, m.poisson)
    s = DescentSolver(m, positions=x0, mu=mu, lam=lam)
    xo, vo, _, _ = I.backward_euler_step(s.positions(), np.zeros_like(x0), m.rest, m.tets, m.pin_mask(), mu, lam)
    it, res = s.backward_euler_step(tol=1e-6)
    assert res <= 1e-6 and it > 0
    assert np.abs(s.positions() - xo).max() / m.bbox_diagonal() < POS_TOL
    s.close()


@pytest.mark.parametrize("split,nx,ny,nz", [(6, 10, 4, 4), (5, 9, 9, 9), (6, 10, 10, 12)])
def test_solves_repeat_bitwise(split, nx, ny, nz):
    """The same two steps forty times over (3, 8 and 13 CTAs; the second solve
    of a handle finds the first one's words): one result, bit for bit."""
    m, x0, v0 = _moving(split, nx, ny, nz)
    mu, lam = O.lame(m.young, m.poisson)
    first = None
    for _ in range(40):
        s = DescentSolver(m, positions=x0, mu=mu, lam=lam)
        s.write_velocities(v0, v0)
        its = [s.backward_euler_step(tol=1e-6) for _ in range(2)]
        out = (its, s.positions().tobytes(), s.velocities()[0].tobytes())
        s.close()
        first = first or out
        assert out == first


def test_converted_inputs_outlive_the_call():
    """Arrays that have to be converted (other order, 64 bits) are copied for
    the call: what arrives is their values."""
    m, x0, _ = _moving(5, 3, 3, 7)
    s = DescentSolver(m, positions=x0)
    rng = np.random.default_rng(3)
    for k in range(50):
        v = rng.standard_normal((m.n_nodes, 3))
        s.write_velocities(np.asfortranarray(v), (2 * v)[:, ::1])
        got, old = s.velocities()
        assert np.array_equal(got, v.astype(np.float32)) and np.array_equal(old, (2 * v).astype(np.float32)), k
        s.update_positions(np.asfortranarray(x0.astype(np.float64)))
        assert np.array_equal(s.positions(), x0)
    s.close()


TEST_WAIT_ERROR = 0  # pbs_test_hook


@pytest.mark.parametrize("integrator", ["be", "pd"])
def test_wait_that_gave_up_is_an_error(integrator):
    """A set flag (a CTA whose wait ran out, whether or not the solve's first
    CTA noticed) ends the step with PBS_E_DEVICE_TIMEOUT, the state as it was;
    the next step is the one of a handle without it."""
    m, x0, v0 = _moving(5, 9, 9, 9)
    mu, lam = O.lame(m.young, m.poisson)
    a, b = DescentSolver(m, positions=x0, mu=mu, lam=lam), DescentSolver(m, positions=x0, mu=mu, lam=lam)
    step = lambda s: s.backward_euler_step(tol=1e-6) if integrator == "be" else s.pd_step()
    a.write_velocities(v0, v0)
    b.write_velocities(v0, v0)
    assert L.lib().pbs_test_hook(a._h, TEST_WAIT_ERROR, 1) == 0
    with pytest.raises(L.PhybsError) as e:
        step(a)
    assert e.value.code == L.PBS_E_DEVICE_TIMEOUT
    assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities()[0], b.velocities()[0])
    for _ in range(2):
        step(a)
        step(b)
        assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities()[0], b.velocities()[0])
    a.close()
    b.close()


def _fan(n):
    """n tets around one edge, its two nodes in all of them."""
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    rest = np.concatenate([[[0, 0, 0], [0, 0, 1]], np.stack([np.cos(a), np.sin(a), 0.5 + 0.1 * np.cos(3 * a)], 1)])
    i = np.arange(n)
    tets = np.stack([np.zeros(n), np.ones(n), 2 + i, 2 + (i + 1) % n], 1).astype(np.int64)
    tets = M.orient_positive(rest, tets)
    return M.TetMeshData(rest.astype(np.float32), tets, np.array([0, 1]), 1e5, 0.3)


# rows on both sides of the line between the device's columns and the host's (256 incident tets)
@pytest.mark.parametrize("n", [40, 255, 256, 257, 600])
def test_rows_of_nodes_with_many_tets(n):
    m = _fan(n)
    mu, lam = O.lame(m.young, m.poisson)
    v0 = (0.1 * np.sin(7 * m.rest[:, [1, 2, 0]])).astype(np.float32)
    v0[m.pins] = 0.0
    s = DescentSolver(m, mu=mu, lam=lam)
    s.write_velocities(v0, v0)
    xo, vo, _, _ = I.backward_euler_step(s.positions(), v0, m.rest, m.tets, m.pin_mask(), mu, lam)
    it, res = s.backward_euler_step(tol=1e-6)
    assert res <= 1e-6
    assert np.abs(s.positions() - xo).max() / m.bbox_diagonal() < POS_TOL
    assert np.abs(s.velocities()[0] - vo).max() <= 1e-3 * np.abs(vo).max()
    s.close()


def test_pattern_time_at_a_node_of_many_tets():
    """The pattern of a node with 6,000 tets: sorted, not selected (36 million
    tets read one after the other, a second and more, against milliseconds)."""
    import time
    s = DescentSolver(_fan(6000))
    t = time.perf_counter()
    s.backward_euler_step(max_iters=1, raise_on_cap=False)
    assert time.perf_counter() - t < 0.5
    s.close()


TEST_SOLVE_SMEM, TEST_SOLVE_COL32 = 4, 5  # pbs_test_hook


@pytest.mark.parametrize("integrator", ["be", "pd"])
@pytest.mark.parametrize("split,nx,ny,nz", [(5, 1, 1, 2), (5, 3, 3, 7), (6, 10, 6, 6), (5, 9, 14, 19)])
def test_solve_with_vectors_in_global_memory(integrator, split, nx, ny, nz):
    """What does not fit a CTA's shared memory on large meshes (the solution from
    0.3 million nodes, then the residual, q, the direction) stays in global
    memory, and columns beyond 65,535 take 32 bits: here under a smaller budget,
    bit for bit as with everything in shared memory."""
    m, x0, v0 = _moving(split, nx, ny, nz)
    mu, lam = O.lame(m.young, m.poisson)

    def solve(smem, wide):
        s = DescentSolver(m, positions=x0, mu=mu, lam=lam)
        s.write_velocities(v0, v0)
        L.lib().pbs_test_hook(s._h, TEST_SOLVE_SMEM, smem)
        L.lib().pbs_test_hook(s._h, TEST_SOLVE_COL32, wide)
        its = [s.backward_euler_step(tol=1e-6) if integrator == "be" else s.pd_step() for _ in range(2)]
        out = its, s.positions(), s.velocities()[0]
        s.close()
        return out

    want = solve(-1, 0)
    # nothing; the rows' records; the direction; q; r; all but the matrix; all but the inverses and x
    for smem in (0, 1536, 6144, 8192, 10240, 12288, 16384, 65536):
        for wide in (0, 1):
            got = solve(smem, wide)
            assert got[0] == want[0] and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2]), (smem, wide)


TEST_LARGE_STEPS = 2


@pytest.mark.parametrize("integrator", ["be", "pd"])
@pytest.mark.parametrize("nx,ny,nz", [(20, 20, 24), (24, 26, 40)])
def test_solve_beside_others(integrator, nx, ny, nz):
    """The solve of a part of a SM, which a step takes when two large ones run
    already (84 CTAs; one on every SM): bit for bit the one of a whole SM."""
    m, x0, v0 = _moving(5, nx, ny, nz)
    out = []
    for others in (0, 2):
        s = DescentSolver(m, positions=x0)
        s.write_velocities(v0, v0)
        L.lib().pbs_test_hook(s._h, TEST_LARGE_STEPS, others)
        try:
            its = [s.backward_euler_step(tol=1e-6) if integrator == "be" else s.pd_step() for _ in range(2)]
        finally:
            L.lib().pbs_test_hook(s._h, TEST_LARGE_STEPS, -others)
        out.append((its, s.positions(), s.velocities()[0]))
        s.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("integrator", ["be", "pd", "pbd"])
def test_solves_of_several_threads(integrator):
    """Handles of different sizes stepped from threads of their own: every one's
    steps are those it takes by itself, and none is refused (the shared memory
    that a launch may have is set per kernel, not per handle)."""
    import threading
    sizes = [(9, 14, 19), (3, 3, 7), (12, 12, 24), (6, 9, 9), (14, 14, 20), (9, 9, 9)]
    ms = [_moving(5, *n) for n in sizes]

    def steps(k, n):
        m, x0, v0 = ms[k]
        s = DescentSolver(m, positions=x0)
        s.write_velocities(v0, v0)
        out = []
        for _ in range(n):
            s.update_positions(x0)
            s.write_velocities(v0, v0)
            if integrator == "be":
                s.backward_euler_step(tol=1e-6)
            elif integrator == "pd":
                s.pd_step()
            else:
                s.pbd_step()
            out.append(s.positions())
        s.close()
        return out

    want = [steps(k, 1)[0] for k in range(len(sizes))]
    got, bad = [None] * len(sizes), []
    start = threading.Barrier(len(sizes))

    def run(k):
        try:
            start.wait()
            got[k] = steps(k, 60)
        except Exception as e:  # noqa: BLE001
            bad.append((k, repr(e)))

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(sizes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
    for g, w in zip(got, want):
        assert all(np.array_equal(x, w) for x in g)
