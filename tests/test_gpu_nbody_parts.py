"""The far-field N-body walkers over sheet parts against the FP64 oracle (B200).

Sheets whose rows and columns leave remainders in every direction of a part
(2, 4 or 6 node rows x 32 segment columns, up to 8 narrow parts per strip), at
targets that are near, between near and far, and far, on nodes and along the
extension of segments, where the reference's cut-off |r1 x r2|^2 < 1e-10
decides.  Tolerances are those of the other N-body tests: FP64 1e-12 of
max |v|; FP32 2e-5 of the local velocity + 1e-6 of max |v|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 33), (2, 3, 32), (1, 4, 65), (1, 7, 8), (5, 2, 3), (40, 1, 1), (1, 26, 31), (1, 13, 130)]


def _sheet(num, rows, cols, seed, wobble):
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(0.15 * np.arange(rows + 1), 0.06 * np.arange(cols + 1), indexing="ij")
    pos = np.stack([np.stack([x, y + 0.3 * n, 0.2 * n + 0 * x], -1) for n in range(num)])
    return pos + wobble * rng.standard_normal(pos.shape), rng.standard_normal((num, rows, cols))


def _targets(pos, seed):
    """Nodes, points at every distance, and points along the extension of both kinds of segments at offsets on
    both sides of the cut-off (|r1 x r2| = |r0| offset against 1e-5)."""
    rng = np.random.default_rng(seed)
    flat = pos.reshape(-1, 3)
    d = rng.standard_normal((300, 3))
    d *= (10.0 ** rng.uniform(-3, 1.5, 300) / np.linalg.norm(d, axis=1))[:, None]
    out = [flat[rng.integers(0, len(flat), 64)], flat[rng.integers(0, len(flat), 300)] + d]
    for a, b in ((pos[:, :-1], pos[:, 1:]), (pos[:, :, :-1], pos[:, :, 1:])):
        a, b = a.reshape(-1, 3), b.reshape(-1, 3)
        k = rng.integers(0, len(a), 120)
        r0 = b[k] - a[k]
        length = np.linalg.norm(r0, axis=1)
        side = np.cross(r0, rng.standard_normal(r0.shape))
        side /= np.linalg.norm(side, axis=1)[:, None]
        away = rng.choice([-1.0, 1.0], 120) * 10.0 ** rng.uniform(-0.5, 1.3, 120)
        factor = rng.choice([0.0, 0.5, 0.8, 1.25, 2.0, 100.0], 120)  # of the cut-off
        out.append(b[k] + r0 / length[:, None] * away[:, None] + side * (factor * 1e-5 / length)[:, None])
    return np.concatenate(out)


@pytest.mark.parametrize("wobble", [0.0, 0.004])
@pytest.mark.parametrize("shape", SHAPES)
def test_parts_match_oracle(shape, wobble):
    import pyoracle as o

    import uvlm_b200 as U

    pos, gamma = _sheet(*shape, seed=sum(shape), wobble=wobble)
    targets = _targets(pos, seed=7 + shape[1])
    ref = o.sheet_induced_velocity(pos, gamma, targets)
    scale, mag = np.max(np.abs(ref)), np.linalg.norm(ref, axis=1)
    got = U.InducedVelocity(targets, pos, gamma)
    assert np.max(np.abs(got - ref)) <= 1e-12 * scale
    got = U.InducedVelocity(targets, pos, gamma, precision="mixed")
    assert np.all(np.abs(got - ref).max(axis=1) <= 2e-5 * mag + 1e-6 * scale)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_strengths_scale_exactly(precision):
    """Powers of two of the circulations scale the velocities exactly, and zero circulations give zeros."""
    import uvlm_b200 as U

    pos, gamma = _sheet(1, 9, 40, seed=3, wobble=0.003)
    t = _targets(pos, seed=4)
    v = U.InducedVelocity(t, pos, gamma, precision)
    for e in (-20, 10):
        np.testing.assert_array_equal(U.InducedVelocity(t, pos, gamma * 2.0 ** e, precision), v * 2.0 ** e)
    np.testing.assert_array_equal(U.InducedVelocity(t, pos, gamma * 0, precision), 0)
    # circulations so small that their squares leave the FP32 range
    small = U.InducedVelocity(t, pos, gamma * 2.0 ** -60, precision) * 2.0 ** 60
    np.testing.assert_allclose(small, v, rtol=0, atol=(1e-12 if precision == "fp64" else 2e-5) * np.max(np.abs(v)))


@pytest.mark.parametrize("n", [2048, 8191, 8193, 20011, 33000])
@pytest.mark.parametrize("kind", ["box", "line", "one", "odd"])
def test_point_sets_that_are_ordered_first(n, kind):
    """Point sets large enough to be put in the order of a space-filling curve against the same points in pieces that are
    evaluated as given: spread in a box, along a line, all in one place, with a few that are not finite.  Tolerances of
    the other N-body tests between two evaluations (FP64 1e-12 of max |v|; FP32 4e-5 of the local velocity + 2e-6 of
    max |v|, twice a single one's)."""
    import uvlm_b200 as U

    pos, gamma = _sheet(1, 70, 64, seed=n, wobble=0.0)  # 9104 segments
    rng = np.random.default_rng(n)
    x = rng.uniform([-1, -1, -1], [12, 5, 1], (n, 3))
    if kind == "line":
        x = np.outer(rng.uniform(0.1, 30, n), [1.0, 0.0, 0.0]) + [0.0, 0.333, 0.77]
    if kind == "one":
        x[:] = x[0]
    odd = np.zeros(n, bool)
    if kind == "odd":
        odd[rng.integers(0, n, 9)] = True
        x[odd] = rng.choice([np.nan, np.inf, -np.inf, 1e300], (odd.sum(), 3))
    for precision, piece in (("fp64", 1000), ("mixed", 1000)):
        got = U.InducedVelocity(x, pos, gamma, precision=precision)
        ref = np.concatenate([U.InducedVelocity(x[i:i + piece], pos, gamma, precision=precision)
                              for i in range(0, n, piece)])
        got, ref = got[~odd], ref[~odd]
        assert np.all(np.isfinite(got))
        scale, mag = np.max(np.abs(ref)), np.linalg.norm(ref, axis=1)
        bound = 1e-12 * scale if precision == "fp64" else 4e-5 * mag + 2e-6 * scale
        assert np.all(np.abs(got - ref).max(axis=1) <= bound)
    np.testing.assert_array_equal(U.InducedVelocity(x, pos, gamma), U.InducedVelocity(x, pos, gamma))


# ---------------------------------------------------------------- ends of the range
def _lattice():
    pos, gamma = _sheet(1, 9, 40, seed=11, wobble=0.003)
    return pos, gamma, _targets(pos, seed=12)


DISTANCES = [1e9, 1e20, 1e78, 1e100, 1e153, 1e154, 1e155, 1e250]


def _far_points(distance, n=64):
    d = np.random.default_rng(1).standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1)[:, None] * distance


def _far_limit(gamma, distance):
    """Bound of the velocity at a distance: every segment is shorter than 1."""
    return np.abs(gamma).sum() / distance * min(1e3 / distance, 1.0)


@pytest.mark.parametrize("distance", DISTANCES)
def test_near_walkers_and_rings_give_no_velocity_far_away(distance):
    """Points so far away that products of distances leave the FP64 range: rings, and a sheet of circulations below
    1e-13, which the near walkers take."""
    import uvlm_b200 as U
    from uvlm_b200 import rings as R

    pos, gamma, _ = _lattice()
    gamma = gamma * 1e-14
    far = _far_points(distance)
    n = pos[0]
    ring = np.stack([n[:-1, :-1], n[:-1, 1:], n[1:, 1:], n[1:, :-1]], 2).reshape(-1, 4, 3)
    for got in (U.InducedVelocity(far, pos, gamma), R.InducedVelocity(far, ring, gamma.reshape(-1))):
        assert np.all(np.isfinite(got)) and np.max(np.abs(got)) <= _far_limit(gamma, distance)


# ---------------------------------------------------------------- pinned tiles
def _velocity(pos, gamma, wing, wing_gamma, targets, variant, near_fp64=(), precision="mixed", max_wake_rows=64):
    """Velocities of a wing and a wake sheet set (the same column count, even) by one pinned tile."""
    import uvlm_b200 as U

    num, rows, cols = gamma.shape
    sim = U.SimpleSimulator(precision=precision, nbody_variant=variant, near_fp64=near_fp64 if precision == "mixed"
                            else None, max_wake_rows=max(max_wake_rows, rows + 2))
    for _ in range(num):
        sim.AddWing(U.RectGenerator(), U.Morphing(), 1.0, 4.0, wing_gamma.shape[1], cols)
    sim.set_forward_flight([-1.0, 0.0, 0.0])
    sim.set_advection("euler")
    sim.begin()
    sim.set_state(rows, wing, pos, wing_gamma, wing_gamma, gamma)
    out = sim.Velocity(targets, include_freestream=False)
    sim.close()
    return out


def _variants():
    import uvlm_b200 as U

    names = [U.lib().uvlm_nbody_variant_name(i).decode() for i in range(64)]
    return {name: i for i, name in enumerate(names) if name != "?"}


PART_TILES = ["fp32_h2_t2_b128_x2f", "fp32_h3_t2_b128_x2f", "fp32_h4_t2_b128_x2f"]


@pytest.mark.parametrize("distance", DISTANCES)
def test_part_walkers_give_no_fp64_velocity_far_away(distance):
    """The same by the part walkers, alone and beside points that are near and keep their velocities."""
    import uvlm_b200 as U

    pos, gamma, near = _lattice()
    far, limit = _far_points(distance), _far_limit(gamma, distance)
    got = U.InducedVelocity(far, pos, gamma)
    assert np.all(np.isfinite(got)) and np.max(np.abs(got)) <= limit
    mixed = np.empty((128, 3))
    mixed[0::2], mixed[1::2] = far, near[:64]
    got = U.InducedVelocity(mixed, pos, gamma)
    assert np.all(np.isfinite(got)) and np.max(np.abs(got[0::2])) <= limit
    ref = U.InducedVelocity(near, pos, gamma)[:64]
    assert np.max(np.abs(got[1::2] - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("tile", PART_TILES)
@pytest.mark.parametrize("distance", [1e6, 1e12, 1e18, 1e21, 1e30])
def test_part_walkers_give_no_fp32_velocity_far_away(tile, distance):
    """The same in FP32, whose squares of distances leave the range from 1e19 on."""
    pos, gamma, near = _lattice()
    wing, wing_gamma = pos[:, :2] - [0.31, 0.0, 0.0], np.ones((1, 1, 40))
    x = np.empty((128, 3))
    x[0::2], x[1::2] = _far_points(distance), near[:64]
    got = _velocity(pos, gamma, wing, wing_gamma, x, _variants()[tile])
    assert np.all(np.isfinite(got)) and np.max(np.abs(got[0::2])) <= _far_limit(gamma, distance)


@pytest.mark.parametrize("exponent", [40, 66, 100, 160])
def test_fp64_sheets_of_any_size(exponent):
    """A lattice and its points scaled by a power of two (on nodes, near and far; not along the extension of segments,
    where the oracle itself cancels once its absolute cut-off is out of reach): the oracle's velocities, to 1e-12 of
    max |v|, where coordinates, their squares and the bounds of a part leave the FP32 range."""
    import pyoracle as o

    import uvlm_b200 as U

    pos, gamma, t = _lattice()
    t, s = t[:364], 2.0 ** exponent
    ref = o.sheet_induced_velocity(pos * s, gamma, t * s)
    got = U.InducedVelocity(t * s, pos * s, gamma)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("exponent", [-400, 60, 130, 520])
def test_fp64_strengths_of_any_size(exponent):
    """Circulations scaled by a power of two: the velocities scaled by it, to 1e-12 of max |v|."""
    import uvlm_b200 as U

    pos, gamma, t = _lattice()
    ref = U.InducedVelocity(t, pos, gamma)
    got = U.InducedVelocity(t, pos, gamma * 2.0 ** exponent) * 2.0 ** -exponent
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("tile", PART_TILES)
def test_part_walkers_scale_with_the_strengths(tile):
    """As test_strengths_scale_exactly, by the FP32 part walkers: powers of two scale exactly, and circulations whose
    squares leave the FP32 range on either side give the same velocities to the rounding of another walker (2e-5 of
    max |v|)."""
    pos, gamma, t = _lattice()
    wing, wing_gamma = _sheet(1, 2, 40, seed=8, wobble=0.0)
    wing = wing - [0.31, 0.0, 0.0]
    v = {e: _velocity(pos, gamma * 2.0 ** e, wing, wing_gamma * 2.0 ** e, t, _variants()[tile]) * 2.0 ** -e
         for e in (0, -20, 10, -60, 75)}
    for e in (-20, 10):
        np.testing.assert_array_equal(v[e], v[0])
    for e in (-60, 75):
        np.testing.assert_allclose(v[e], v[0], rtol=0, atol=2e-5 * np.max(np.abs(v[0])))


@pytest.mark.parametrize("tile,h", [("fp32_h2_t2_b128_x2f", 2), ("fp32_h3_t2_b128_x2f", 3), ("fp32_h4_t2_b128_x2f", 4)])
def test_fp32_sums_are_short_on_narrow_sheets(tile, h):
    """FP32 sums go to FP64 after h node rows of one sheet.  A wake of 8 columns whose spanwise segments all add up the
    same way over 210 rows at a time, seen from far away, so that the rounding of the sums outweighs that of the terms;
    all coordinates are multiples of 2^-18 below 32, so that positions relative to any node are exact in FP32.

    Bound: adding the k-th of n = 8 h terms of size t to a sum rounds by at most u k t, uniformly distributed (variance
    a third of the square), so a sum gathers (u t)^2 n^3 / 9 and all N terms N n^2 / 9; the terms themselves are taken
    to be off by 4 u each at random.  Twice the root of the sum of both."""
    import pyoracle as o

    rows, cols, n_t = 2100, 8, 256
    rng = np.random.default_rng(h)
    i, j = np.meshgrid(np.arange(rows + 1), np.arange(cols + 1), indexing="ij")
    pos = np.stack([2.0 ** -17 * i, 0.125 * j, 0.0 * i], -1)[None]
    up = np.where((np.arange(rows) // 210) % 2 == 0, 1.0, -1.0) * rng.uniform(0.5, 1.5, rows)
    gamma = np.repeat(np.cumsum(up)[:, None], cols, 1)[None]
    wing, wing_gamma = pos[:, :2] - [1.0, 0.0, 0.0], np.zeros((1, 1, cols))
    d = rng.standard_normal((n_t, 3)) * [1.0, 0.3, 1.0]
    targets = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(20, 25, (n_t, 1))
    targets = np.round(targets * 2.0 ** 18) * 2.0 ** -18
    ref = o.sheet_induced_velocity(pos, gamma, targets)
    copies = 141
    got = _velocity(pos, gamma, wing, wing_gamma, np.tile(targets, (copies, 1)), _variants()[tile],
                    max_wake_rows=copies * n_t // (cols + 1) + 1)
    got = got.reshape(copies, n_t, 3)
    assert np.all(got == got[0])
    t = 0.125 / (4 * np.pi * np.linalg.norm(targets, axis=1)[:, None] ** 2)
    rms = np.sqrt(np.mean(np.sum(((got[0] - ref) / t) ** 2, axis=1)))  # in mean terms of one segment
    u, terms = 2.0 ** -24, rows * cols
    bound = 2 * u * np.sqrt(terms * ((cols * h) ** 2 / 9 + 16))
    print(f"{tile}: rms error {rms / u:.0f} u terms, bound {bound / u:.0f}")
    assert rms <= bound


@pytest.mark.parametrize("shape,n", [((1, 1, 3), 220000), ((1, 2, 4), 95325), ((1, 2, 4), 95326), ((1, 8, 36), 3382),
                                     ((1, 8, 36), 3383), ((1, 6, 64), 30001), ((3, 5, 9), 12345), ((1, 21, 22), 17000),
                                     ((1, 21, 23), 17000), ((1, 15, 70), 9000)])
def test_unordered_points_at_the_edges_of_the_tile_rule(shape, n):
    """Point sets on both sides of 2^21 pairs and of 1000 segments, and sheets whose node rows fill strips of 2, 3 or 4
    rows differently, against the oracle; tolerances as above."""
    import pyoracle as o

    import uvlm_b200 as U

    pos, gamma = _sheet(*shape, seed=n, wobble=0.003)
    t = _targets(pos, seed=n)
    x = np.tile(t, (n // len(t) + 1, 1))[:n]
    ref = o.sheet_induced_velocity(pos, gamma, t)
    ref = np.tile(ref, (n // len(t) + 1, 1))[:n]
    scale, mag = np.max(np.abs(ref)), np.linalg.norm(ref, axis=1)
    assert np.max(np.abs(U.InducedVelocity(x, pos, gamma) - ref)) <= 1e-12 * scale
    got = U.InducedVelocity(x, pos, gamma, precision="mixed")
    assert np.all(np.abs(got - ref).max(axis=1) <= 2e-5 * mag + 1e-6 * scale)


PINNED = [("fp32_h2_t2_b128_x2f", ()), ("fp32_h3_t2_b128_x2f", ()), ("fp32_h4_t2_b128_x2f", ()),
          ("fp32_h3_t2_b128_x2f", ("advect",)), ("fp64_h2_t1_b128_m3f", None), ("fp64_h3_t1_b128_m2f", None),
          ("fp64_h2_t2_b128_f", None)]
# (sheets, wake rows, columns, copies of the targets): remainders of 2, 4, 6 and 8 node rows and of 32 columns,
# uneven parts, and enough targets that narrow parts share a strip (4 CTAs' worth of tiles times strips per slot)
PINNED_SHAPES = [(1, 1, 2, 1), (5, 2, 6, 1), (2, 7, 8, 500), (1, 26, 16, 300), (1, 13, 34, 1), (2, 9, 66, 1),
                 (1, 5, 130, 1), (1, 45, 2, 800)]


@pytest.mark.parametrize("shape", PINNED_SHAPES)
@pytest.mark.parametrize("tile,near", PINNED)
def test_pinned_part_walkers_match_oracle(tile, near, shape):
    """Every part walker at every target of _targets (nodes, all distances, both sides of the cut-off) against the
    oracle, in both precisions, and in FP32 not the near tile's bits (the part walker has run)."""
    import pyoracle as o

    num, rows, cols, copies = shape
    pos, gamma = _sheet(num, rows, cols, seed=rows + cols, wobble=0.004)
    wing, wing_gamma = _sheet(num, 2, cols, seed=rows, wobble=0.002)
    wing = wing - [0.31, 0.0, 0.0]
    targets = _targets(pos, seed=5 + rows)
    ref = o.sheet_induced_velocity(pos, gamma, targets) + o.sheet_induced_velocity(wing, wing_gamma, targets)
    scale, mag = np.max(np.abs(ref)), np.linalg.norm(ref, axis=1)
    many = np.tile(targets, (copies, 1))
    fp64 = near is None
    got = _velocity(pos, gamma, wing, wing_gamma, many, _variants()[tile], near or (), "fp64" if fp64 else "mixed",
                    max_wake_rows=max(64, len(many) // (num * (cols + 1)) + 1))
    bound = np.full(len(ref), 1e-12 * scale) if fp64 else 2e-5 * mag + 1e-6 * scale
    err = np.abs(got.reshape(copies, -1, 3) - ref).max(axis=(0, 2))
    assert np.all(err <= bound)
    if not fp64:
        plain = _velocity(pos, gamma, wing, wing_gamma, targets, _variants()["fp32_h3_t2_b128_x2"])
        assert np.any(got[: len(ref)] != plain)
