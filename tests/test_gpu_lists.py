"""GPU: the neighbour-list builder at the edges of its work split (particles per warp, candidate rounds, list and staging
capacities), against the oracle and against the plain walk of the buckets (kernel variant 1)."""
import numpy as np
import pytest

from gpu_util import RTOL, assert_close, fluid_like

pytestmark = pytest.mark.gpu

D = 0.02  # lattice spacing: h = 2 D, 8 particles a cell at rest


def _cloud(n, per_cell, seed):
    """n particles at uniform random places of a cube that holds per_cell of them per cell of size h."""
    side = 2 * D * (n / per_cell) ** (1 / 3)
    return (np.random.default_rng(seed).random((n, 3)) * side).astype(np.float32)


# sizes around the particles of a warp and of a block for each of the three splits (2, 4 and 8 particles a warp: up to
# 8,192, up to 16,384, beyond) and around the sweeps' own (8,192, 49,152), and dense clouds: more candidates than the 320 of one pass, more neighbours than the
# near list (64), the skin list (96) and the staging area hold
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n,per_cell", [(1, 8), (2, 8), (7, 8), (9, 8), (33, 20), (1000, 40), (700, 300), (2000, 600),
                                        (8191, 8), (8192, 8), (8193, 8), (49152, 8), (49153, 10), (60001, 8)])
def test_lists_hold_the_walks_neighbours(oracle, n, per_cell, order):
    pos = _cloud(n, per_cell, seed=n)
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    got = {}
    for variant in (2, 1):
        f = fluid_like(p, kernel_variant=variant, spatial_order=order)
        f.set_fluid_state(pos)
        f.run_stage("sort")
        f.run_stage("density")
        f.run_stage("normal")
        f.run_stage("force")
        f.set_field("predicted_position", f.get_field("sorted_position"))
        f.run_stage("pressure")
        f.run_stage("pressure_force", 0)
        got[variant] = {k: f.get_field(k) for k in ("density", "normal", "other_force", "density_variation",
                                                    "pressure_force", "sorted_position", "cell_offsets")}
        f.close()
    a, w = got[2], got[1]
    off = a["cell_offsets"].astype(np.int64).reshape(-1, 2)
    rho = oracle.update_density(p, None, None, a["cell_offsets"], a["sorted_position"])
    # sums of up to K terms in FP32, each side rounded on its own: 2 K ulp of the sum of the terms' magnitudes
    k = min(n, 27 * int((off[:, 1] - off[:, 0]).max()))
    tol = max(RTOL, 2 * k * 2.0 ** -24)
    assert_close("density", a["density"], rho, rtol=tol)
    assert_close("density_variation", a["density_variation"], np.maximum(rho - 1000.0, 0), scale=float(rho.max()), rtol=tol)
    for name in ("density", "normal", "other_force", "pressure_force"):
        assert_close(name, a[name], w[name], rtol=tol)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [64, 9000])
def test_nonfinite_particles_reach_the_same_sums(oracle, n, value):
    pos = _cloud(n, 8, seed=3)
    pos[n // 3, 1] = value
    pos[n // 2] = value
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    rho = []
    for variant in (2, 1):
        f = fluid_like(p, kernel_variant=variant, spatial_order=0)
        f.set_fluid_state(pos)
        f.run_stage("sort")
        f.run_stage("density")
        rho.append(f.get_field("density"))
        f.close()
    np.testing.assert_array_equal(np.isnan(rho[0]), np.isnan(rho[1]))
    ok = ~np.isnan(rho[1])
    assert_close("density", rho[0][ok], rho[1][ok])


# one particle more takes the next split of the sweeps (eight lanes per particle up to 8,192, two chunks in flight up to
# 49,152, then one); its own place is far away, and the bucket count is the same
@pytest.mark.parametrize("boundary", [False, True])
@pytest.mark.parametrize("n", [8192, 49152])
def test_splits_of_the_sweeps_give_the_same_bits(oracle, n, boundary):
    rng = np.random.default_rng(n)
    pos = _cloud(n, 8, seed=n + 1) + np.float32(0.1)
    pos[:90] = pos[0] + rng.random((90, 3)).astype(np.float32) * 0.5 * D  # a clump that overflows its lists
    vel = (0.3 * rng.standard_normal((n, 3))).astype(np.float32)
    vel[rng.choice(n, 30, replace=False)] *= 20.0  # predictions that outrun the lists
    far = np.float32([[40.0, 40.0, 40.0]])
    floor = np.stack(np.meshgrid(np.arange(20), [0.0], np.arange(20), indexing="ij"), -1).reshape(-1, 3) * D + 0.1
    out = []
    for extra in (False, True):
        x = np.concatenate([pos, far]) if extra else pos
        v = np.concatenate([vel, 0 * far]) if extra else vel
        p = oracle.derive_params(0.5 * D, 1000.0, len(x), len(floor) if boundary else 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
        f = fluid_like(p, min_iters=3, max_iters=3, spatial_order=0)
        f.set_fluid_state(x, v)
        if boundary:
            f.set_boundary_state(floor.astype(np.float32))
        f.update()
        keep = f.get_field("src") < n
        out.append({k: f.get_field(k)[keep] for k in ("src", "density", "normal", "other_force", "predicted_position",
                                                      "pressure", "pressure_force", "position", "velocity")})
        assert f.stats().fast_particles > 0
        f.close()
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)


@pytest.mark.parametrize("loop_mode,order", [(0, 0), (0, 1), (1, 1), (2, 0)])
@pytest.mark.parametrize("motion", ["fall", "shear", "random", "half"])
def test_moving_lists_change_no_bits(oracle, motion, loop_mode, order):
    """A scene of which many particles move faster than the skin allows builds its skin lists around y = x + v dt. The
    same steps without that (per-particle skins build every list around x) give the same bits and the same counts."""
    n = 12000
    rng = np.random.default_rng(7)
    pos = _cloud(n, 8, seed=11) + np.float32(0.2)
    vel = np.zeros_like(pos)
    if motion == "fall":
        vel[:, 1] = -9.0  # 0.23 h per step, the whole body
    elif motion == "shear":
        vel[:, 0] = 20.0 * (pos[:, 1] - 0.2)
    elif motion == "random":
        vel = (6.0 * rng.standard_normal(pos.shape)).astype(np.float32)
    else:
        vel[pos[:, 0] < np.median(pos[:, 0]), 2] = 15.0  # one half slides past the other
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    out = []
    for skins in (0, 1):
        f = fluid_like(p, min_iters=4, max_iters=4, loop_mode=loop_mode, spatial_order=order, walls=True,
                       box_hi=(3.0, 3.0, 3.0))
        f.set_options(particle_skin=skins)
        f.set_fluid_state(pos, vel)
        f.step(2)
        st = f.stats()
        out.append(({k: f.get_field(k) for k in ("src", "density", "normal", "pressure", "pressure_force", "position",
                                                 "velocity", "predicted_position")},
                    (st.fast_particles, st.list_fallbacks, st.status_all)))
        f.close()
    assert out[0][1] == out[1][1] and out[0][1][0] > n // 8
    for k in out[0][0]:
        np.testing.assert_array_equal(out[0][0][k], out[1][0][k], err_msg=k)


def test_moving_lists_keep_nonfinite_velocities(oracle):
    n = 9000
    pos = _cloud(n, 8, seed=12)
    vel = np.full_like(pos, 8.0)
    vel[5, 0], vel[77] = np.nan, np.inf
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    out = []
    for skins in (0, 1):
        f = fluid_like(p, min_iters=3, max_iters=3, spatial_order=0)
        f.set_options(particle_skin=skins)
        f.set_fluid_state(pos, vel)
        f.update()
        assert f.stats().status & 2
        out.append([f.get_field(k) for k in ("density", "pressure", "density_variation")])
        f.close()
    for a, w in zip(*out):
        np.testing.assert_array_equal(a, w)


# The pressure sweeps from the third iteration on read lists rebuilt at the second one's predictions. Sizes at the edges of
# their launches (8,192; 155,648 and 194,560 where the building sweep changes its form; past 2M); loops that end before
# a list is built, before it is used and long after it was left behind; a block that overflows them; predictions that
# outrun every list at once or keep leaving the rebuilt ones; boundary particles; skins of other sizes; NaN
@pytest.mark.parametrize("n,gap,jitter,speed,iters,options", [
    (1, 1.0, 0.1, 0.0, (5, 5), {}), (4097, 1.0, 0.3, 1.0, (25, 25), {}), (8192, 0.75, 0.4, 8.0, (12, 12), {}),
    (5000, 1.0, 0.2, 0.0, (20, 20), {"boundary": 1}), (5001, 1.0, 0.1, 4.0, (8, 8), {"list_skin": 0.0}),
    (7777, 1.0, 0.2, 3.0, (9, 9), {"nan": 1}),
    (8193, 1.0, 0.1, 0.0, (3, 3), {}), (9001, 1.0, 0.1, 0.0, (1, 1), {}), (9001, 1.0, 0.1, 0.0, (2, 2), {}),
    (9001, 1.0, 0.2, 0.0, (1, 9), {}), (20000, 1.0, 0.3, 0.0, (40, 40), {}), (30000, 0.8, 0.1, 0.0, (12, 12), {}),
    (30000, 0.75, 0.4, 8.0, (30, 30), {}), (12000, 1.0, 0.1, 4.0, (8, 8), {"list_skin": 0.0}),
    (12000, 1.0, 0.3, 1.0, (25, 25), {"list_skin": 0.5}), (16000, 1.0, 0.2, 0.0, (20, 20), {"particle_skin": 0, "boundary": 1}),
    (16000, 1.0, 0.2, 0.0, (20, 20), {"boundary": 1}), (16000, 1.0, 0.3, 1.0, (9, 9), {"particle_skin": 1}),
    (16000, 1.0, 0.2, 3.0, (20, 20), {"nan": 1}), (155648, 1.0, 0.2, 0.0, (12, 12), {}),
    (155649, 1.0, 0.15, 0.0, (8, 8), {"sweep_block": 512}), (194561, 1.0, 0.2, 0.5, (9, 9), {"sweep_block": 128}),
    (2097153, 1.0, 0.2, 0.0, (9, 9), {})])
def test_rebuilt_lists_change_no_bits(oracle, n, gap, jitter, speed, iters, options):
    """The persistent loop builds no such lists: the same bits and the same counts."""
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    at = np.stack(np.unravel_index(np.arange(n), (side, side, side)), -1) + 0.5
    pos = ((at + jitter * (2 * rng.random((n, 3)) - 1)) * gap * D).astype(np.float32)
    vel = (speed * rng.standard_normal((n, 3))).astype(np.float32)
    if options.get("nan"):
        vel[n // 2] = np.nan
    floor = np.stack(np.meshgrid(np.arange(side), [-0.5], np.arange(side), indexing="ij"), -1).reshape(-1, 3) * D
    walls = len(floor) if options.get("boundary") else 0
    p = oracle.derive_params(0.5 * D, 1000.0, n, walls, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    out = []
    for loop_mode in (0, 1, 2):
        f = fluid_like(p, min_iters=iters[0], max_iters=iters[1], loop_mode=loop_mode, spatial_order=2)
        f.set_options(**{k: v for k, v in options.items() if k not in ("nan", "boundary")})
        f.set_fluid_state(pos, vel)
        if walls:
            f.set_boundary_state(floor.astype(np.float32))
        f.step(2)
        st = f.stats()
        out.append(({k: f.get_field(k) for k in ("src", "density", "density_variation", "pressure", "pressure_force",
                                                 "position", "velocity", "predicted_position")},
                    (st.fast_particles, st.list_fallbacks, st.status_all, st.total_iterations)))
        f.close()
    for got in out[:2]:
        assert got[1] == out[2][1]
        for k in got[0]:
            np.testing.assert_array_equal(got[0][k], out[2][0][k], err_msg=k)


# Predictions that a caller sets between the stages lie where the caller puts them, here at x: lists around y = x + v dt, which
# a step of fast particles builds, do not hold their pairs (neighbours of opposite velocities are 2 h apart there)
@pytest.mark.parametrize("after", ["sort", "step", "step, density"])
@pytest.mark.parametrize("n,order", [(4000, 0), (12000, 0), (12000, 1)])
def test_set_predictions_find_every_pair(oracle, n, order, after):
    rng = np.random.default_rng(n)
    pos = _cloud(n, 8, seed=n) + np.float32(1.0)
    vel = np.zeros_like(pos)
    vel[:, 2] = rng.choice([-40.0, 40.0], n)
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, 0.0, 0.0, 0.0)
    f = fluid_like(p, min_iters=1, max_iters=1, spatial_order=order)
    f.set_fluid_state(pos, vel)
    if after == "sort":
        f.run_stage("sort")
    else:
        f.update()
    if after != "step":
        f.run_stage("density")
    x, cells = f.get_field("sorted_position"), f.get_field("cell_offsets")
    f.set_field("predicted_position", x)
    f.run_stage("pressure")
    got = f.get_field("density_variation")
    f.close()
    rho = oracle.update_density(p, None, None, cells, x)
    off = cells.astype(np.int64).reshape(-1, 2)
    tol = max(RTOL, 2 * min(n, 27 * int((off[:, 1] - off[:, 0]).max())) * 2.0 ** -24)
    assert rho.max() > 1000.0
    assert_close("density_variation", got, np.maximum(rho - 1000.0, 0), scale=float(rho.max()), rtol=tol)


# Predictions that outrun the skin lists before, at and after the building of the tight ones: few in a thousand, at speeds around
# half the skin per step (they cross it within a step), a whole corner, or most, whose lists are then not built for some
# sweeps or steps; skins narrower than the tight lists' margin; sizes on either side of the forms that mark by themselves, with
# and without bucket order, boundary particles (and their skins), several steps
@pytest.mark.parametrize("n,motion,speed,options", [
    (1000, "few", 2.0, {}), (4096, "few", 4.0, {}), (8192, "few", 2.7, {}), (8193, "few", 2.7, {}), (20000, "few", 2.0, {}),
    (20000, "few", 3.5, {"boundary": 1}), (20000, "few", 3.5, {"boundary": 1, "particle_skin": 0}), (6000, "few", 2.7, {"boundary": 1}),
    (4096, "corner", 8.0, {}), (20000, "corner", 8.0, {}), (140000, "corner", 3.0, {}), (20000, "all", 1.2, {}), (5000, "all", 1.2, {}),
    (20000, "all", 8.0, {}), (5000, "few", 2.0, {"list_skin": 0.03}), (9000, "few", 2.0, {"list_skin": 0.03}),
    (9000, "few", 2.0, {"list_skin": 0.07}), (9000, "all", 0.6, {"list_skin": 0.1}), (9000, "few", 2.0, {"list_skin": 0.08, "boundary": 1}),
    (200000, "few", 2.7, {}), (2100000, "few", 2.7, {}), (1000, "few", 4.6, {}), (4096, "few", 5.0, {}), (8192, "few", 4.8, {}),
    (8193, "few", 4.8, {}), (20000, "few", 5.2, {}), (20000, "few", 4.8, {"boundary": 1}), (6000, "few", 5.0, {"boundary": 1}),
    (140000, "corner", 5.0, {}), (20000, "all", 3.6, {}), (5000, "all", 3.6, {}), (200000, "few", 5.0, {}), (2100000, "few", 5.0, {})])
def test_outrun_lists_change_no_bits(oracle, n, motion, speed, options):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    at = np.stack(np.unravel_index(np.arange(n), (side, side, side)), -1) + 0.5
    pos = ((at + 0.15 * (2 * rng.random((n, 3)) - 1)) * D).astype(np.float32)
    vel = (0.3 * rng.standard_normal((n, 3))).astype(np.float32)
    who = {"few": rng.random(n) < 0.004, "corner": (at < 0.5 * side).all(1), "all": np.ones(n, bool)}[motion]
    way = rng.standard_normal((n, 3))
    vel[who] = (speed * way / np.linalg.norm(way, axis=1)[:, None] * (0.8 + 0.4 * rng.random((n, 1)))).astype(np.float32)[who]
    floor = np.stack(np.meshgrid(np.arange(side), [-0.5], np.arange(side), indexing="ij"), -1).reshape(-1, 3) * D
    walls = len(floor) if options.get("boundary") else 0
    steps, iters = (2, 9) if n > 100000 else (5, 12)
    p = oracle.derive_params(0.5 * D, 1000.0, n, walls, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    out = []
    for loop_mode in (0, 1, 2):
        f = fluid_like(p, min_iters=iters, max_iters=iters, loop_mode=loop_mode, spatial_order=2)
        f.set_options(**{k: v for k, v in options.items() if k != "boundary"})
        f.set_fluid_state(pos, vel)
        if walls:
            f.set_boundary_state(floor.astype(np.float32))
        f.step(steps)
        st = f.stats()
        out.append(({k: f.get_field(k) for k in ("src", "density_variation", "pressure", "position", "velocity", "predicted_position")},
                    (st.fast_particles, st.list_fallbacks, st.status_all)))
        f.close()
    for got in out[:2]:
        assert got[1] == out[2][1]
        for k in got[0]:
            np.testing.assert_array_equal(got[0][k], out[2][0][k], err_msg=k)


@pytest.mark.parametrize("n,block", [(8000, 256), (8000, 512), (2100000, 256), (2100000, 128)])
def test_autotune_chooses_among_different_launches(oracle, n, block):
    """The block stays what it was where another's launches are the same: scenes of at most 8,192 particles have their own,
    and above 2,097,152 256 stands for 128."""
    p = oracle.derive_params(0.5 * D, 1000.0, n, 0, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    for _ in range(3 if n < 10000 else 1):
        f = fluid_like(p, spatial_order=1)
        f.set_options(sweep_block=block)
        f.set_fluid_state(_cloud(n, 8, seed=n))
        r = f.autotune(steps=1)
        assert r["candidates"] == 26
        assert r["sweep_block"] in ((block,) if n < 10000 else (block, 512))
        f.close()


# the builder's second split (4 particles a warp up to 16,384, 8 beyond)
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n", [16384, 16385])
def test_lists_at_the_builders_second_split(oracle, n, order):
    test_lists_hold_the_walks_neighbours(oracle, n, 8, order)


# Long loops in which particles keep crossing half the skin: after some sweeps the rebuilt lists are built once more, with
# predictions flagged before they reach it
@pytest.mark.parametrize("n,motion,speed,options", [
    (6000, "few", 4.7, {}), (8193, "few", 4.7, {}), (30000, "few", 4.7, {}), (30000, "corner", 4.4, {}), (30000, "all", 2.2, {}),
    (20000, "few", 4.7, {"boundary": 1}), (20000, "corner", 4.4, {"list_skin": 0.2}), (160000, "corner", 4.4, {})])
def test_early_flags_change_no_bits(oracle, n, motion, speed, options):
    rng = np.random.default_rng(n + 1)
    side = int(np.ceil(n ** (1 / 3)))
    at = np.stack(np.unravel_index(np.arange(n), (side, side, side)), -1) + 0.5
    pos = ((at + 0.2 * (2 * rng.random((n, 3)) - 1)) * 0.95 * D).astype(np.float32)
    vel = np.zeros((n, 3), np.float32)
    who = {"few": rng.random(n) < 0.02, "corner": (at < 0.5 * side).all(1), "all": np.ones(n, bool)}[motion]
    vel[who, 1] = (-speed * (0.95 + 0.1 * rng.random(n))).astype(np.float32)[who]
    floor = np.stack(np.meshgrid(np.arange(side), [-0.5], np.arange(side), indexing="ij"), -1).reshape(-1, 3) * D
    walls = len(floor) if options.get("boundary") else 0
    p = oracle.derive_params(0.5 * D, 1000.0, n, walls, 1e-3, -9.81, 0.2 * D ** 3, 0.5)
    out = []
    for loop_mode in (0, 1, 2):
        f = fluid_like(p, min_iters=40, max_iters=40, loop_mode=loop_mode, spatial_order=2)
        f.set_options(**{k: v for k, v in options.items() if k != "boundary"})
        f.set_fluid_state(pos, vel)
        if walls:
            f.set_boundary_state(floor.astype(np.float32))
        f.step(3)
        st = f.stats()
        out.append(({k: f.get_field(k) for k in ("src", "density_variation", "pressure", "position", "velocity", "predicted_position")},
                    (st.fast_particles, st.list_fallbacks, st.status_all)))
        f.close()
    for got in out[:2]:
        assert got[1] == out[2][1]
        for k in got[0]:
            np.testing.assert_array_equal(got[0][k], out[2][0][k], err_msg=k)
