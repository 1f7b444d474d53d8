"""Batched independent cases (uvlm_batch_*) against the FP64 oracle and the
single-case library path, on a B200.

Cases come from the seeded flapping-wing sweep (rows 4-16, even cols 8-64,
aspect ratio 2-10, k 0.1-1, heave 0.05-0.3, pitch 0-20 deg), cut to sizes the
oracle finishes in seconds.  Each case of the batch must reproduce its own
SimpleSimulator run: FP64 batch within 1e-9 of the oracle on the loads and
circulation; the mixed batch (FP32 N-body, FP32 LU + FP64 refinement) within
1e-6 relative.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 20


def _small_cases(n, seed=3):
    from uvlm_b200.batch import draw_cases

    cs = draw_cases(n, seed)
    for d in cs:  # cut to oracle-sized lattices, keep the drawn kinematics
        d["rows"] = 2 + d["rows"] // 4
        d["cols"] = 2 * (2 + d["cols"] // 16)
        d["span"] = min(d["span"], 6.0)
    return cs


def _oracle(d, steps, advection="euler"):
    import pyoracle as o

    sim = o.Simulator()
    kin = o.kinematics(plug_amp=d["heave"], plug_omega=d["omega"], twist_amp=math.radians(d["pitch_deg"]),
                       twist_omega=d["omega"], twist_phase=math.pi / 2)
    sim.add_wing(d["chord"], d["span"], d["rows"], d["cols"], kin=kin)
    sim.set_forward_flight((-1.0, 0.0, 0.0))
    sim.set_advection(advection)
    loads = sim.run(steps - 1, d["dt"])
    return np.asarray(loads), sim.state()


@pytest.mark.parametrize("advection", ["euler", "RK2"])
def test_batch_fp64_matches_oracle(advection):
    from uvlm_b200.batch import make_batch

    cases = _small_cases(5)
    sim = make_batch(cases, precision="fp64", advection=advection, max_steps=STEPS)
    sim.run(STEPS)
    L = sim.loads()
    assert L.shape == (STEPS, len(cases), 3)
    for c, d in enumerate(cases):
        ref, st = _oracle(d, STEPS, advection)
        np.testing.assert_allclose(L[:, c, 0], ref[:, 0], rtol=0, atol=1e-12)
        scale = np.max(np.abs(ref[:, 1:])) + 1e-30
        np.testing.assert_allclose(L[:, c, 1:], ref[:, 1:], rtol=0, atol=1e-9 * scale)
        got = sim.case_state(c)
        np.testing.assert_allclose(got["wing_gamma"], st["wing_gamma"][0], rtol=0,
                                   atol=1e-9 * np.max(np.abs(st["wing_gamma"])))
        np.testing.assert_allclose(got["wake_pos"], st["wake_pos"][0], rtol=0, atol=1e-9)
        np.testing.assert_allclose(got["wake_gamma"], st["wake_gamma"][0], rtol=0,
                                   atol=1e-9 * np.max(np.abs(st["wing_gamma"])))
    sim.close()


def test_batch_mixed_refinement_matches_oracle():
    from uvlm_b200.batch import make_batch

    cases = _small_cases(6, seed=11)
    sim = make_batch(cases, precision="mixed", max_steps=STEPS)
    sim.run(STEPS)
    L = sim.loads()
    sweeps, res = sim.solve_stats()
    assert np.all(res <= 1e-12)
    for c, d in enumerate(cases):
        ref, st = _oracle(d, STEPS)
        scale = np.max(np.abs(ref[:, 1:]))
        assert np.max(np.abs(L[:, c, 1:] - ref[:, 1:])) <= 1e-6 * scale
    sim.close()


def test_batch_graph_replay_equals_direct_launches():
    from uvlm_b200.batch import make_batch

    cases = _small_cases(7, seed=5)
    out = []
    for g in (True, False):
        # one pinned tile for both (each batch's autotuner could pick another)
        sim = make_batch(cases, precision="mixed", max_steps=12, use_graph=g, nbody_tile=0)
        sim.run(5)
        sim.run(7)
        out.append((sim.loads(), [sim.case_state(c)["wake_pos"] for c in range(len(cases))]))
        if g:
            assert sim.launches_per_step() > 10
        sim.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)


def test_batch_case_equals_single_case_library_path():
    """A case inside a ragged batch gives the single-case FP64 path's answer."""
    import uvlm_b200 as U
    from uvlm_b200.batch import case_morphing, make_batch

    cases = _small_cases(4, seed=9)
    sim = make_batch(cases, precision="fp64", max_steps=10)
    sim.run(10)
    L = sim.loads()
    for c, d in enumerate(cases):
        one = U.SimpleSimulator(precision="fp64")
        one.AddWing(U.RectGenerator(), case_morphing(d), d["chord"], d["span"], d["rows"], d["cols"])
        one.set_forward_flight([-1.0, 0.0, 0.0])
        one.set_advection("euler")
        one.begin()
        rows = np.array([one.step(s, d["dt"]) for s in range(10)])
        np.testing.assert_allclose(L[:, c, 1:], rows[:, 1:], rtol=0, atol=1e-10 * np.max(np.abs(rows[:, 1:])))
        one.close()
    sim.close()


def test_batch_full_sweep_shapes_run():
    """The 256-case sweep at its drawn sizes: a few steps, finite loads,
    refinement converged in every case."""
    from uvlm_b200.batch import draw_cases, make_batch

    cases = draw_cases(256, seed=0)
    sim = make_batch(cases, precision="mixed", max_steps=8)
    sim.run(8)
    L = sim.loads()
    assert np.all(np.isfinite(L))
    sweeps, res = sim.solve_stats()
    assert np.all(res <= 1e-12)
    sim.close()


def test_batch_rejects_bad_cases():
    import uvlm_b200 as U
    from uvlm_b200.batch import BatchError, BatchSimulator

    sim = BatchSimulator()
    sim.add_case(U.Morphing(), 1.0, 4.0, 4, 7, 0.1)  # odd cols
    with pytest.raises(BatchError):
        sim.begin()
    sim2 = BatchSimulator(max_steps=3)
    sim2.add_case(U.Morphing(), 1.0, 4.0, 4, 8, 0.1)
    sim2.run(3)
    with pytest.raises(BatchError):
        sim2.run(1)
    sim2.close()


def test_batch_wide_and_narrow_cases_mixed_vs_oracle():
    """Cases wide enough for the padded packed walker (cols >= 48) and narrow
    ones in one mixed batch, each against its own oracle run."""
    from uvlm_b200.batch import make_batch

    rng = np.random.default_rng(21)
    cases = []
    for cols in (64, 8, 50, 12, 48):
        k = float(rng.uniform(0.3, 0.8))
        cases.append(dict(rows=3, cols=cols, chord=1.0, span=float(rng.uniform(3, 8)), k=k, omega=2 * k,
                          heave=float(rng.uniform(0.05, 0.2)), pitch_deg=float(rng.uniform(2, 15)),
                          dt=2 * math.pi / (2 * k) / 40))
    steps = 12
    sim = make_batch(cases, precision="mixed", max_steps=steps)
    sim.run(steps)
    L = sim.loads()
    sim.close()
    for c, d in enumerate(cases):
        ref, _ = _oracle(d, steps)
        scale = np.max(np.abs(ref[:, 1:]))
        assert np.max(np.abs(L[:, c, 1:] - ref[:, 1:])) <= 1e-6 * scale, d["cols"]


def test_batch_stale_factors_same_answer_fewer_factorizations():
    """Refining from the previous circulation with an earlier step's FP32
    factors converges to the same 1e-12 residual as a fresh factorisation
    every step, with fewer factorisations."""
    from uvlm_b200.batch import make_batch

    cases = _small_cases(6, seed=17)
    steps = 20
    out = {}
    for stale in (False, True):
        # one pinned tile for both: each batch's autotuner could pick another, and
        # another tile's FP32 rounding, grown by the wake over 20 steps, exceeds 1e-9
        sim = make_batch(cases, precision="mixed", max_steps=steps, stale_factors=stale, nbody_tile=0)
        sim.run(steps)
        out[stale] = (sim.loads(), sim.factorizations(), sim.solve_stats()[1])
        sim.close()
    assert out[False][1] == len(cases) * steps
    assert out[True][1] < out[False][1]
    assert np.all(out[True][2] <= 1e-12)
    scale = np.max(np.abs(out[False][0][:, :, 1:]))
    assert np.max(np.abs(out[True][0][:, :, 1:] - out[False][0][:, :, 1:])) <= 1e-9 * scale


def test_batch_tile_autotuner_is_fixed_under_graph_replay():
    """The tile autotuner picks one compiled FP32 tile at creation; every
    graph-replayed step runs it: the autotuned batch equals, bit for bit, a
    batch pinned to the tile it chose, with and without graph replay."""
    from uvlm_b200.batch import draw_cases, make_batch

    cases = draw_cases(12, seed=4)
    auto = make_batch(cases, precision="mixed", max_steps=30)
    name = auto.nbody_tile()
    assert name.startswith("fp32_") and name.endswith("_x2f"), name
    auto.run(20)
    tiles = ["fp32_h3_t2_b128_x2f", "fp32_h2_t2_b128_x2f", "fp32_h4_t2_b128_x2f"]
    outs = []
    for graph in (True, False):
        from uvlm_b200.batch import BatchSimulator, case_morphing

        sim = BatchSimulator(precision="mixed", max_steps=30, use_graph=graph, nbody_tile=tiles.index(name))
        for d in cases:
            sim.add_case(case_morphing(d), d["chord"], d["span"], d["rows"], d["cols"], d["dt"])
        assert sim.nbody_tile() == name
        sim.run(20)
        outs.append(sim.loads())
        sim.close()
    np.testing.assert_array_equal(auto.loads(), outs[0])
    np.testing.assert_array_equal(outs[0], outs[1])
    auto.close()


def test_every_batch_tile_agrees_with_the_fp64_batch():
    from uvlm_b200.batch import BatchSimulator, case_morphing, draw_cases

    cases = draw_cases(6, seed=9)

    def run(precision, tile=-1):
        sim = BatchSimulator(precision=precision, max_steps=16, nbody_tile=tile)
        for d in cases:
            sim.add_case(case_morphing(d), d["chord"], d["span"], d["rows"], d["cols"], d["dt"])
        sim.run(15)
        out = sim.loads()
        sim.close()
        return out

    ref = run("fp64")
    scale = np.max(np.abs(ref[:, :, 1:]))
    for t in range(3):
        got = run("mixed", t)
        assert np.max(np.abs(got[:, :, 1:] - ref[:, :, 1:])) <= 1e-6 * scale, t


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_per_case_solve_at_its_block_edges(precision):
    """Cases whose N = rows x cols sits at and between the edges of the per-case solver (panels of 32 or 16 columns,
    32-row diagonal blocks, 64 x 256 and 64 x 128 update tiles, the largest N = 1024) against single-case FP64
    simulators: loads within the batch tolerances."""
    import uvlm_b200 as U
    from uvlm_b200.batch import BatchSimulator

    shapes = [(1, 2), (1, 16), (1, 18), (2, 16), (3, 10), (3, 22), (4, 16), (5, 26), (8, 32), (9, 30), (16, 64)]
    steps, dt = 4, 0.15
    sim = BatchSimulator(precision=precision, max_steps=steps, nbody_tile=0 if precision == "mixed" else -1)
    for k, (r, c) in enumerate(shapes):
        m = U.Morphing().set_alpha(0.05).set_plug(0.1 + 0.01 * k, 1.0).set_twist(0.1, 1.0, math.pi / 2)
        sim.add_case(m, 1.0, 3.0 + 0.2 * k, r, c, dt)
    sim.run(steps)
    rows = sim.loads()
    sim.close()
    tol = 1e-9 if precision == "fp64" else 1e-6
    for k, (r, c) in enumerate(shapes):
        one = U.SimpleSimulator()
        m = U.Morphing().set_alpha(0.05).set_plug(0.1 + 0.01 * k, 1.0).set_twist(0.1, 1.0, math.pi / 2)
        one.AddWing(U.RectGenerator(), m, 1.0, 3.0 + 0.2 * k, r, c)
        one.set_forward_flight([-1.0, 0.0, 0.0])
        one.set_advection("euler")
        ref = one.Run(steps - 1, dt)
        one.close()
        assert np.max(np.abs(rows[:, k, 1:] - ref[:, 1:])) <= tol * np.max(np.abs(ref[:, 1:])), (r, c)


@pytest.mark.parametrize("n", [2, 37, 38, 49, 50, 74, 75, 149])
def test_solve_clusters_of_every_size_give_the_same_loads(n):
    """Batches whose cases are solved by clusters of 4, 3, 2 and 1 CTAs (as many as run all cases at once): copies of one
    case, N = 90 (rows that leave remainders in every CTA's share), against a batch of one, to the mixed tolerance."""
    import uvlm_b200 as U
    from uvlm_b200.batch import BatchSimulator

    def loads(copies):
        sim = BatchSimulator(precision="mixed", max_steps=5, nbody_tile=0)
        m = U.Morphing().set_alpha(0.05).set_plug(0.1, 1.0).set_twist(0.1, 1.0, math.pi / 2)
        for _ in range(copies):
            sim.add_case(m, 1.0, 4.0, 9, 10, 0.15)
        sim.run(5)
        rows = sim.loads()
        sim.close()
        return rows[:, :, 1:]

    one, many = loads(1), loads(n)
    assert np.max(np.abs(many - one)) <= 1e-6 * np.max(np.abs(one))


def _small_batch(rows, cols, n, precision="mixed", use_graph=True, steps=3, tile=0):
    import uvlm_b200 as U
    from uvlm_b200.batch import BatchSimulator

    sim = BatchSimulator(precision=precision, max_steps=steps, use_graph=use_graph,
                         nbody_tile=tile if precision == "mixed" else -1)
    m = U.Morphing().set_alpha(0.05).set_plug(0.1, 1.0).set_twist(0.1, 1.0, math.pi / 2)
    for _ in range(n):
        sim.add_case(m, 1.0, 4.0, rows, cols, 0.15)
    return sim


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batches_of_different_sizes_live_at_once(precision, use_graph):
    """A batch of large cases runs after one of small cases was created: its loads are those it has alone."""
    alone = _small_batch(16, 64, 2, precision, use_graph)
    alone.run(3)
    want = alone.loads()
    alone.close()
    large, small = _small_batch(16, 64, 2, precision, use_graph), _small_batch(4, 8, 2, precision, use_graph)
    large.begin()
    small.begin()
    small.run(1)
    large.run(3)
    got = large.loads()
    large.close()
    small.close()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cols", [2, 36, 64])
def test_memory_of_a_long_batch(precision, cols):
    """The partial sums of a batch take 1 GiB, or one set per 16 wake rows and 64 columns (at least 8 sets per case):
    what a batch of 24 cases and 1000 steps takes on the device beside its other arrays."""
    import torch

    _small_batch(4, cols, 1, precision, steps=4).close()
    sim = _small_batch(4, cols, 24, precision, steps=1000)
    before = torch.cuda.mem_get_info(0)[0]
    sim.begin()
    used = before - torch.cuda.mem_get_info(0)[0]
    sim.run(2)
    sim.close()
    nodes = 24 * 1002 * (cols + 1)
    sets = max(8, math.ceil(1002 / 16) + 1)
    # per node: positions, circulation, record, targets and velocities, one set of partial sums each
    other = nodes * (24 + 8 + 96 + 24 + 24)
    assert used <= max(1 << 30, nodes * 24 * sets) + other + (16 << 20)


@pytest.mark.parametrize("precision,cols,steps,longest", [("fp64", 64, 56, 1000), ("fp64", 34, 80, 1000),
                                                          ("mixed", 64, 105, 1300)])
def test_long_batches_whose_items_take_more_than_three_strips(precision, cols, steps, longest):
    """Batches made for wakes so long that their partial sums are bounded, once their wakes pass 24 strips, against a
    single-case FP64 simulator, to the batch tolerances."""
    import uvlm_b200 as U

    sim = _small_batch(1, cols, 40, precision, steps=longest, tile=1)
    sim.run(steps)
    rows = sim.loads()
    sim.close()
    one = U.SimpleSimulator()
    m = U.Morphing().set_alpha(0.05).set_plug(0.1, 1.0).set_twist(0.1, 1.0, math.pi / 2)
    one.AddWing(U.RectGenerator(), m, 1.0, 4.0, 1, cols)
    one.set_forward_flight([-1.0, 0.0, 0.0])
    one.set_advection("euler")
    ref = one.Run(steps - 1, 0.15)
    one.close()
    tol = 1e-9 if precision == "fp64" else 1e-6
    for k in (0, 39):
        assert np.max(np.abs(rows[:, k, 1:] - ref[:, 1:])) <= tol * np.max(np.abs(ref[:, 1:]))


@pytest.mark.parametrize("n", [2, 37, 38, 49, 50, 74, 75, 149])
def test_solve_clusters_of_every_size_give_the_same_bits(n):
    """A residual row is the same sum whichever CTA of a cluster forms it: copies of one case, solved by clusters of 4,
    3, 2 and 1 CTAs, against a batch of one: equal loads, sweeps and residuals, bit by bit."""
    def run(copies):
        sim = _small_batch(9, 10, copies, steps=5)
        sim.run(5)
        out = sim.loads()[:, :, 1:], *sim.solve_stats()
        sim.close()
        return out

    (one, sweeps1, res1), (many, sweeps, res) = run(1), run(n)
    np.testing.assert_array_equal(many, np.repeat(one, n, axis=1))
    np.testing.assert_array_equal(sweeps, np.repeat(sweeps1, n))
    np.testing.assert_array_equal(res, np.repeat(res1, n))
