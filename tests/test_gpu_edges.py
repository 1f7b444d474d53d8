"""Edge cases of the CUDA path against the FP64 oracle (B200).

Empty inputs (no targets, sheets without rings), ragged strip shapes (column
counts that leave a short last chunk, row counts that leave a short last row
group), the smallest wing the reference accepts (1 x 2 rings) and a batch of
one case.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheet(rng, num, rows, cols):
    i = np.arange(rows + 1)[:, None]
    j = np.arange(cols + 1)[None, :]
    pos = np.zeros((num, rows + 1, cols + 1, 3))
    for n in range(num):
        pos[n, ..., 0] = 0.25 * i + 0.01 * rng.standard_normal((rows + 1, cols + 1))
        pos[n, ..., 1] = 0.0625 * j + 0.01 * rng.standard_normal((rows + 1, cols + 1))
        pos[n, ..., 2] = 0.3 * n + 0.05 * np.sin(0.7 * i + 0.3 * j)
    return pos, rng.standard_normal((num, rows, cols))


def test_no_targets_and_no_rings():
    import uvlm_b200 as U

    rng = np.random.default_rng(0)
    pos, gamma = _sheet(rng, 1, 3, 4)
    for prec in ("fp64", "mixed"):
        out = U.InducedVelocity(np.zeros((0, 3)), pos, gamma, prec)
        assert out.shape == (0, 3)
        # a sheet with one node row has no rings: zero velocity everywhere
        v = U.InducedVelocity(rng.standard_normal((5, 3)), pos[:, :1], np.zeros((1, 0, 4)), prec)
        assert np.all(v == 0.0)


@pytest.mark.parametrize("shape", [(1, 7, 66), (2, 5, 129), (1, 130, 3), (1, 9, 64), (1, 9, 65)])
def test_ragged_strips_both_precisions(shape):
    import pyoracle as o

    import uvlm_b200 as U

    rng = np.random.default_rng(sum(shape))
    pos, gamma = _sheet(rng, *shape)
    targets = np.concatenate([rng.uniform(-0.5, 4.5, size=(300, 3)), pos.reshape(-1, 3)[::7]])
    ref = o.sheet_induced_velocity(pos, gamma, targets)
    scale = np.max(np.abs(ref))
    got64 = U.InducedVelocity(targets, pos, gamma, "fp64")
    assert np.max(np.abs(got64 - ref)) <= 1e-12 * scale
    got32 = U.InducedVelocity(targets, pos, gamma, "mixed")
    assert np.all(np.isfinite(got32))
    assert np.max(np.abs(got32 - ref)) <= 1e-5 * scale


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_smallest_wing_matches_oracle(precision):
    import pyoracle as o

    import uvlm_b200 as U

    dt, steps = 0.1, 12
    kin = dict(alpha=math.radians(4), plug_amp=0.1, plug_omega=1.3)
    sim = U.SimpleSimulator(precision=precision)
    m = U.Morphing().set_alpha(kin["alpha"]).set_plug(kin["plug_amp"], kin["plug_omega"])
    sim.AddWing(U.RectGenerator(), m, 1.0, 2.0, 1, 2)
    sim.set_forward_flight([-1.0, 0.0, 0.0])
    sim.set_advection("RK2")
    rows = sim.Run(steps, dt)
    sim.close()
    ref = o.Simulator()
    ref.add_wing(1.0, 2.0, 1, 2, kin=o.kinematics(**kin))
    ref.set_forward_flight((-1.0, 0.0, 0.0))
    ref.set_advection("RK2")
    want = ref.run(steps, dt)
    tol = 1e-8 if precision == "fp64" else 1e-5
    assert np.max(np.abs(np.asarray(rows)[:, 1:] - want[:, 1:])) <= tol * np.max(np.abs(want[:, 1:]))


def test_batch_of_one_smallest_case():
    import pyoracle as o

    import uvlm_b200 as U
    from uvlm_b200.batch import BatchSimulator

    dt, steps = 0.1, 10
    sim = BatchSimulator(precision="fp64", max_steps=steps)
    sim.add_case(U.Morphing().set_alpha(math.radians(4)).set_plug(0.1, 1.3), 1.0, 2.0, 1, 2, dt)
    sim.run(steps)
    L = sim.loads()
    sim.close()
    ref = o.Simulator()
    ref.add_wing(1.0, 2.0, 1, 2, kin=o.kinematics(alpha=math.radians(4), plug_amp=0.1, plug_omega=1.3))
    ref.set_forward_flight((-1.0, 0.0, 0.0))
    ref.set_advection("euler")
    want = ref.run(steps - 1, dt)
    assert np.max(np.abs(L[:, 0, 1:] - want[:, 1:])) <= 1e-9 * np.max(np.abs(want[:, 1:]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_velocity_at_points_of_the_current_state(precision):
    """SimpleSimulator::Velocity on a grid of points (the velocity-field
    tools' use) equals -ff + the oracle's induced velocity of the state."""
    import pyoracle as o

    import uvlm_b200 as U

    sim = U.SimpleSimulator(precision=precision)
    sim.AddWing(U.RectGenerator(), U.Morphing().set_alpha(0.08).set_plug(0.1, 1.0), 1.0, 4.0, 4, 8)
    sim.set_forward_flight([-1.0, 0.0, 0.0])
    sim.set_advection("RK2")
    sim.Run(15, 0.15)
    st = sim.state()
    g = np.stack(np.meshgrid(np.linspace(-0.5, 3.5, 9), np.linspace(-2.5, 2.5, 7), [-0.3, 0.21], indexing="ij"),
                 -1).reshape(-1, 3)
    got = sim.Velocity(g)
    sim.close()
    ref = (o.sheet_induced_velocity(st["wing_pos"], st["wing_gamma"], g)
           + o.sheet_induced_velocity(st["wake_pos"], st["wake_gamma"], g) + np.array([1.0, 0.0, 0.0]))
    tol = 1e-12 if precision == "fp64" else 1e-6
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 192, 257, 321, 1088, 2305, 4161])
def test_lu_of_a_general_matrix_at_its_block_edges(n):
    """Factors and solves of matrices whose pivots lie anywhere, at the edges of the 64-wide panels, of the 64-row and
    64-column CTAs behind a panel and of the panel's clusters (n = 4161 starts with panels of more than one cluster).
    Bounds: n rounding errors per entry, times a growth of n^(2/3) (random matrices with partial pivoting)."""
    import uvlm_b200 as M

    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    b = rng.standard_normal(n)
    x, _ = M.dense_solve(A, b, "fp64")
    res = np.max(np.abs(A @ x - b)) / (np.linalg.norm(A, np.inf) * np.max(np.abs(x)))
    assert res <= n ** (5 / 3) * np.finfo(np.float64).eps
    A32 = A.astype(np.float32)
    LU, ipiv = M.lu_factor_f32(A32, "simt")
    assert np.all(ipiv >= np.arange(n)) and np.all(ipiv < n)
    PA = A32.astype(np.float64)
    for k, p in enumerate(ipiv):
        if p != k:
            PA[[k, p]] = PA[[p, k]]
    L = np.tril(LU, -1).astype(np.float64) + np.eye(n)
    err = np.max(np.abs(PA - L @ np.triu(LU).astype(np.float64))) / np.max(np.abs(A32))
    assert err <= n ** (5 / 3) * np.finfo(np.float32).eps


@pytest.mark.parametrize("n,nt", [(0, 5), (1, 1), (31, 127), (32, 128), (33, 129), (1025, 300), (70, 160000)])
@pytest.mark.parametrize("chordwise", [False, True])
def test_ring_velocities_at_tile_and_split_edges(n, nt, chordwise):
    """AoS rings against the reference's segment formula (src/vortex.cpp:24-38) in NumPy, a few targets on nodes.  The
    points are in general position at distances above 1e-3 of the segments, where the formula loses at most 1e-9."""
    from uvlm_b200 import rings as R

    rng = np.random.default_rng(1000 * n + nt)
    r = rng.uniform(-1, 1, (n, 1, 3)) + np.array([[0, 0, 0], [0.3, 0, 0], [0.3, 0.4, 0.1], [0, 0.4, 0]])
    g = rng.standard_normal(n)
    x = rng.uniform(-1.5, 1.5, (nt, 3))
    if n:
        x[:: max(nt // 7, 1)] = r[rng.integers(0, n, len(x[:: max(nt // 7, 1)])), 2]
    got = R.InducedVelocity(x, r, g, chordwise=chordwise)
    check = np.unique(np.linspace(0, nt - 1, 257).astype(int))
    ref = np.zeros((len(check), 3))
    for i, t in enumerate(x[check]):
        for k in (0, 2) if chordwise else range(4):  # nodes[k + 1] -> nodes[k]
            r1, r2 = t - r[:, (k + 1) % 4], t - r[:, k]
            d = np.cross(r1, r2)
            d2, n1, n2 = (d * d).sum(1), np.linalg.norm(r1, axis=1), np.linalg.norm(r2, axis=1)
            ok = (d2 >= 1e-10) & (n1 >= 1e-10) & (n2 >= 1e-10)
            f = ((r1 - r2)[ok] * (r1[ok] / n1[ok, None] - r2[ok] / n2[ok, None])).sum(1) / d2[ok]
            ref[i] += ((g[ok] * f / (4 * np.pi))[:, None] * d[ok]).sum(0)
    assert np.max(np.abs(got[check] - ref), initial=0) <= 1e-9 * max(np.max(np.abs(ref)), 1)


def test_ring_velocities_round_once_per_ring():
    """A running sum over rings rounds once per ring: 1000 rings whose velocities add up, more targets than one split
    of the rings needs.  Bound: one rounding of the sum per ring, uniform over a unit in the last place (variance a
    twelfth of its square), against an 80-bit evaluation; the segments' own roundings are a tenth of that.  1.5 times
    the root of the sum."""
    from uvlm_b200 import rings as R

    rng = np.random.default_rng(8)
    n, nt, L = 1000, 256, np.longdouble
    base = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], float)
    r = base + 0.05 * rng.standard_normal((n, 4, 3))
    g = rng.uniform(0.5, 1.5, n)
    x = np.array([0.5, 0.5, 0.0]) + rng.uniform(-0.8, 0.8, (nt, 3)) + np.array([0, 0, 2.5]) * rng.choice([-1, 1], (nt, 1))
    got = R.InducedVelocity(np.tile(x, (600, 1)), r, g).reshape(600, nt, 3)
    assert np.all(got == got[0])
    run, var = np.zeros((nt, 3), L), np.zeros((nt, 3))
    pi = L("3.14159265358979323846264338327950288")
    for k in range(n):
        p = r[k].astype(L)
        for s in range(4):  # nodes[s + 1] -> nodes[s]
            r1, r2 = x.astype(L) - p[(s + 1) % 4], x.astype(L) - p[s]
            n1, n2 = np.sqrt((r1 * r1).sum(1)), np.sqrt((r2 * r2).sum(1))
            f = (n1 + n2) / (n1 * n2 * (n1 * n2 + (r1 * r2).sum(1)))
            run += (g[k] * f / (4 * pi))[:, None] * np.cross(r1, r2)
        var += np.spacing(np.abs(run).astype(float)) ** 2 / 12
    rms = float(np.sqrt(np.mean((got[0] - run) ** 2)))
    assert rms <= 1.5 * np.sqrt(np.mean(var))


def test_simulators_do_not_see_a_busy_default_stream():
    """Batches and simulators run on streams of their own; their first arrays are there before the first step although
    another thread keeps the default stream, which fills them, busy."""
    import threading

    import torch

    import uvlm_b200 as U
    from uvlm_b200.batch import BatchSimulator

    def batch(precision, graph):
        sim = BatchSimulator(precision=precision, max_steps=4, use_graph=graph,
                             nbody_tile=0 if precision == "mixed" else -1)
        for _ in range(3):
            sim.add_case(U.Morphing().set_alpha(0.05).set_plug(0.1, 1.0), 1.0, 4.0, 4, 8, 0.15)
        sim.run(4)
        out = sim.loads()
        sim.close()
        return out

    def simulator(precision):
        sim = U.SimpleSimulator(precision=precision)
        sim.AddWing(U.RectGenerator(), U.Morphing().set_alpha(0.05).set_plug(0.1, 1.0), 1.0, 4.0, 4, 8)
        sim.set_forward_flight([-1.0, 0.0, 0.0])
        sim.set_advection("euler")
        out = sim.Run(3, 0.15)
        gamma = sim.state()["wing_gamma"]
        sim.close()
        return np.concatenate([out.ravel(), gamma.ravel()])

    calls = [lambda p=p, g=g: batch(p, g) for p in ("fp64", "mixed") for g in (True, False)]
    calls += [lambda p=p: simulator(p) for p in ("fp64", "mixed")]
    want = [call() for call in calls]
    stop = threading.Event()

    def busy():
        done = [torch.cuda.Event() for _ in range(4)]
        k = 0
        while not stop.is_set():
            done[k % 4].synchronize()  # four sleeps of about 20 ms queued at a time
            torch.cuda._sleep(40_000_000)
            done[k % 4].record()
            k += 1

    th = threading.Thread(target=busy)
    th.start()
    try:
        got = [call() for _ in range(2) for call in calls]
    finally:
        stop.set()
        th.join()
    for a, b in zip(got, want + want):
        np.testing.assert_array_equal(a, b)


def test_small_mixed_evaluations_take_the_near_tiles():
    """FP32 stages below 2^25 pairs run a near tile (2 or 3 rows), unless one is pinned or their near pairs are FP64; the
    loads are those of the pinned part walker to the mixed tolerance."""
    import uvlm_b200 as U

    names = [U.lib().uvlm_nbody_variant_name(v).decode() for v in range(64)]
    near, far = ("fp32_h2_t2_b128_x2", "fp32_h3_t2_b128_x2"), "fp32_h2_t2_b128_x2f"

    def run(**kw):
        sim = U.SimpleSimulator(precision="mixed", **kw)
        sim.AddWing(U.RectGenerator(), U.Morphing().set_alpha(0.08).set_plug(0.1, 1.0), 1.0, 4.0, 6, 12)
        sim.set_forward_flight([-1.0, 0.0, 0.0])
        sim.set_advection("RK2")
        loads = sim.Run(20, 0.12)
        tiles = [names[v] for v in sim.stats().stage_variant[:3]]
        sim.close()
        return loads[:, 1:], tiles

    loads, tiles = run()
    assert tiles[0].endswith("x2f") and tiles[1] in near and tiles[2] in near, tiles
    pinned, tiles = run(nbody_variant=names.index(far))
    assert tiles == [far] * 3
    _, tiles = run(near_fp64=True)
    assert all(t.endswith("x2f") for t in tiles), tiles
    assert np.max(np.abs(loads - pinned)) <= 1e-6 * np.max(np.abs(pinned))


@pytest.mark.parametrize("chordwise", [False, True])
def test_shared_segments_of_equal_rings_cancel(chordwise):
    """A lattice of rings of one circulation carries nothing on the segments inside it, and points 1e-4 away from
    those see the boundary alone: both rings evaluate the segment alike.  Bound: the sum of each ring's terms, up to
    v = g / (2 pi distance), rounds by at most half a unit each, eight terms; an evaluation from the other end would be
    off by the length over the distance, 1e4 units."""
    from uvlm_b200 import rings as R

    rng = np.random.default_rng(4)
    rows, cols, L = 5, 6, np.longdouble
    i, j = np.meshgrid(np.arange(rows + 1), np.arange(cols + 1), indexing="ij")
    p = np.stack([1.0 * i, 1.0 * j, 0 * i], -1) + 0.05 * rng.standard_normal((rows + 1, cols + 1, 3))
    rings = np.stack([p[:-1, :-1], p[:-1, 1:], p[1:, 1:], p[1:, :-1]], 2).reshape(-1, 4, 3)
    # inner segments along j (every ring's first and third) and, for whole rings, along i
    a, b = [p[1:-1, :-1].reshape(-1, 3)], [p[1:-1, 1:].reshape(-1, 3)]
    if not chordwise:
        a, b = a + [p[:-1, 1:-1].reshape(-1, 3)], b + [p[1:, 1:-1].reshape(-1, 3)]
    a, b = np.concatenate(a), np.concatenate(b)
    side = np.cross(b - a, rng.standard_normal(a.shape))
    x = a + (b - a) * rng.uniform(0.2, 0.8, (len(a), 1)) + side / np.linalg.norm(side, axis=1)[:, None] * 1e-4
    got = R.InducedVelocity(x, rings, np.ones(len(rings)), chordwise=chordwise)
    # the boundary, nodes[k + 1] -> nodes[k] of the rings on it
    edges = [(p[0, k + 1], p[0, k]) for k in range(cols)] + [(p[rows, k], p[rows, k + 1]) for k in range(cols)]
    if not chordwise:
        edges += [(p[k, 0], p[k + 1, 0]) for k in range(rows)] + [(p[k + 1, cols], p[k, cols]) for k in range(rows)]
    ref = np.zeros(x.shape, L)
    for s, e in edges:
        r1, r2 = x.astype(L) - s, x.astype(L) - e
        n1, n2 = np.sqrt((r1 * r1).sum(1)), np.sqrt((r2 * r2).sum(1))
        dot, d = (r1 * r2).sum(1), np.cross(r1, r2)
        f = np.where(dot >= 0, (n1 + n2) / (n1 * n2 * (n1 * n2 + dot)), (n1 + n2) * (n1 * n2 - dot) / (n1 * n2 * (d * d).sum(1)))
        ref += f[:, None] * d
    ref /= 4 * L("3.14159265358979323846264338327950288")
    assert float(np.max(np.abs(got - ref))) <= 8 * 2.0 ** -53 / (2 * np.pi * 1e-4)
