"""The forms of the plain step and of the force pass (four warps for 32 beads in
small batches, one thread a bead in large ones) give the same bits, and the
bending sine holds for angles of any size."""
import numpy as np
import pytest

from mt_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [dict(), dict(barrier=1, is_wall=1, rep_r=20.0)], ids=str)
@pytest.mark.parametrize("keep", [False, True])
def test_small_batches_equal_a_large_one(over, keep):
    """80 trajectories of 1018 and one of 33 beads: above the size of the small form
    together, below it in three parts."""
    from mt_gb300 import engine
    p = synth.default_params(seed=71, **over)
    a = synth.make_trajectory(18, 784, seed=71, radius=8.12, psi_mode="make_mt", cube=90.0, thermal=0.05)
    c = synth.make_trajectory(1, 20, seed=72, radius=8.12, psi_mode="make_mt", cube=40.0, thermal=0.05)
    trajs = [a] * 40 + [c] + [a] * 40
    b = synth.batch_from_trajectories(p, trajs)
    b.extra[5:6000:97] = 1
    assert b.nbeads > 80000
    with engine.Engine(b) as e, engine.ShardedEngine(b, [0, 0, 0]) as s:
        e.upload_state(b.coords)
        s.upload_state(b.coords)
        for k in [e] + s.engines:
            k.set_keep_forces(keep)
            k.rebuild_pairs()
        f = e.compute_forces()
        assert np.array_equal(f, np.concatenate([k.compute_forces() for k in s.engines]))
        assert np.abs(f[b.extra == 1]).max() == 0 and np.isfinite(f).all()
        e.step(0, 13)
        s.step(0, 13)
        assert np.array_equal(e.download_state(), s.download_state())
        assert np.array_equal(e.download_rng(), s.download_rng())
        if keep:
            assert np.array_equal(e.download_state(forces=True)[1],
                                  np.concatenate([k.download_state(forces=True)[1] for k in s.engines]))


@pytest.mark.parametrize("keep", [False, True])
def test_very_large_batch_equals_its_halves(keep):
    """500 trajectories of 1018 beads and an odd one, above the size from which the step asks ahead."""
    from mt_gb300 import engine
    p = synth.default_params(seed=74)
    a = synth.make_trajectory(18, 784, seed=74, radius=8.12, psi_mode="make_mt", cube=90.0, thermal=0.05)
    c = synth.make_trajectory(1, 20, seed=75, radius=8.12, psi_mode="make_mt", cube=40.0, thermal=0.05)
    b = synth.batch_from_trajectories(p, [a] * 250 + [c] + [a] * 250)
    assert b.nbeads > 500000
    with engine.Engine(b) as e, engine.ShardedEngine(b, [0, 0]) as s:
        for k in [e, s]:
            k.upload_state(b.coords)
        for k in [e] + s.engines:
            k.set_keep_forces(keep)
        e.step(0, 12)
        s.step(0, 12)
        assert np.array_equal(e.download_state(), s.download_state())
        assert np.array_equal(e.download_rng(), s.download_rng())


@pytest.mark.parametrize("turns", [3, 150, 170, 4000])
def test_bending_of_large_angles(turns):
    """Angle differences of many turns, on both sides of the 1000 rad where the sine
    goes to the library: the psi force of the dimers' harmonic bonds (no lists are
    built) in FP64 from the same FP32 angles.  Allowed: the FP32 rounding of the
    site vectors (2 nm, at most 8 units each, on the 2 nm arm of the bond C) and of
    the sine's argument and value (4 units)."""
    from mt_gb300 import engine
    b = synth.uniform_batch(synth.default_params(seed=73, lj_on=0), 1, 8, 0, seed=73, radius=8.12,
                            psi_mode="make_mt", thermal=0.05)
    rng = np.random.default_rng(turns)
    b.coords[:, 3:6] += (2 * np.pi * rng.integers(-turns, turns + 1, (b.nbeads, 3))).astype(np.float32)
    p = b.params
    with engine.Engine(b) as e:
        e.upload_state(b.coords)
        f = e.compute_forces().astype(np.float64)
    c, j = b.coords.astype(np.float64), np.abs(b.harmonic)
    sg = np.where(b.harmonic < 0, 1.0, -1.0)
    cs, sn = np.cos(c[:, 3:6]), np.sin(c[:, 3:6])
    uz = np.stack([cs[:, 2] * sn[:, 1] * cs[:, 0] + sn[:, 2] * sn[:, 0],
                   sn[:, 2] * sn[:, 1] * cs[:, 0] - cs[:, 2] * sn[:, 0], cs[:, 1] * cs[:, 0]], 1)
    w = 2.0 * sg[:, None] * uz
    d = c[j, :3] - 2.0 * sg[:, None] * uz[j] - c[:, :3] - w
    dpsi = c[j, 5] - c[:, 5]
    near = np.linalg.norm(d, axis=1) < 0.99
    assert near.sum() > 20
    want = p.B_psi * sg * np.sin(sg * dpsi - p.psi_0) + p.C * np.cross(w, d)[:, 2]
    ulp = np.spacing(np.abs(dpsi).astype(np.float32)).astype(np.float64)
    tol = p.C * 2.0 * 8 * 2.0 ** -22 + p.B_psi * (ulp + 4 * 2.0 ** -24)
    assert (np.abs(f[:, 5] - want)[near] <= tol[near]).all()


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("sizes", [(2, 0), (12, 0), (1, 8), (14, 10), (2, 38), (14, 12)], ids=str)
def test_persistent_seed_equals_per_step_kernels(sizes, keep):
    """The persistent kernel of small trajectories (four threads a bead, lists rebuilt
    inside) against the per-step kernels, bit for bit: 13 x sizes[0] lattice and
    sizes[1] free beads, fixed and extra beads, barriers and walls, period ends inside a run."""
    from mt_gb300 import engine
    p = synth.default_params(seed=81, barrier=1, is_wall=1, rep_r=15.0)
    trajs = [synth.make_trajectory(*sizes, seed=81 + k, radius=8.12, psi_mode="make_mt", cube=40.0, thermal=0.05)
             for k in range(3)]
    b = synth.batch_from_trajectories(p, trajs)
    b.extra[7:b.nbeads:31] = 1
    runs = []
    for persistent in (0, 1):
        with engine.Engine(b) as e:
            e.upload_state(b.coords)
            e.set_keep_forces(keep)
            t = e.tuning()
            t["plain_persistent"] = persistent
            e.set_tuning(**t)
            for first, n in ((0, 20), (20, 7), (27, 1), (28, 14)):
                e.step(first, n)
            runs.append((e.download_state(forces=True), e.download_rng(), e.lists()))
    (x0, f0), r0, l0 = runs[0]
    (x1, f1), r1, l1 = runs[1]
    assert np.array_equal(x0, x1) and np.array_equal(r0, r1)
    if keep:
        assert np.array_equal(f0, f1)
    for k in ("lj", "long", "lat"):
        assert np.array_equal(l0[k][0], l1[k][0]) and np.array_equal(l0[k][1], l1[k][1])
    assert l0["lj"][0].max() > 1


@pytest.mark.parametrize("over", [dict(), dict(barrier=1)], ids=str)
def test_bonds_past_the_largest_square(over):
    """A listed partner so far away that the squared distance overflows exerts no force, as one does
    whose exponential is 0: the other beads' forces are those with the partner at 1e9 nm."""
    from mt_gb300 import engine
    b = synth.uniform_batch(synth.default_params(seed=76, **over), 1, 6, 0, seed=76, radius=8.12, psi_mode="make_mt",
                            thermal=0.05)
    far, partner = 40, abs(int(b.harmonic[40]))
    f = []
    with engine.Engine(b) as e:
        e.upload_state(b.coords)
        e.rebuild_pairs()
        L = e.lists()
        assert L["lat"][0][far] >= 2
        for x in (1.0e9, 2.5e19):
            c = b.coords.copy()
            c[far, 0] = x
            e.upload_state(c)
            f.append(np.delete(e.compute_forces(), (far, partner), 0))
    assert np.isfinite(f[0]).all() and np.array_equal(f[0], f[1])


@pytest.mark.parametrize("mode", ["plain", "tea", "learned"])
def test_chained_launches_equal_unchained(mode):
    """Small batches launch their kernels chained, except while kernels are timed: 300 steps
    with 30 rebuilds of lists that change, from graphs and step by step, bit for bit."""
    from mt_gb300 import engine
    p = synth.default_params(seed=83, hdi_on=int(mode != "plain"), tea_epsilon_freq=5, viscosity=8.0e3)
    b = synth.batch_from_trajectories(p, [synth.make_trajectory(*s, seed=83, radius=8.12, psi_mode="make_mt", cube=45.0,
                                                                thermal=0.05) for s in ((20, 400), (12, 100))])
    runs = []
    for timed in (False, True):
        with engine.Surrogate(seed=5) as net, engine.Engine(b) as e:
            e.upload_state(b.coords)
            e.set_kernel_timing(timed)
            if mode == "learned":
                e.set_surrogate(net, recheck_every=20, max_err=1.0e9)
                e.set_tea_farfield(True, 0.85, refresh_every=100)
            e.rebuild_pairs()
            before = e.lists()["lj"][0]
            for first in range(0, 300, 60):
                e.step(first, 47)
                e.step(first + 47, 13)
            runs.append((e.download_state(), e.download_rng(), e.lists()))
    (x0, r0, l0), (x1, r1, l1) = runs
    assert np.isfinite(x0).all() and np.array_equal(x0, x1) and np.array_equal(r0, r1)
    for k in ("lj", "long", "lat"):
        assert np.array_equal(l0[k][0], l1[k][0]) and np.array_equal(l0[k][1], l1[k][1])
    assert (before != l0["lj"][0]).any()


@pytest.mark.parametrize("block", [64, 256])
def test_autotune_keeps_a_block_without_effect(block):
    """step_block has no effect on batches of the four-warp form: its value is kept, not drawn by timing noise."""
    from mt_gb300 import engine
    b = synth.uniform_batch(synth.default_params(seed=77), 2, 12, 200, seed=77, radius=8.12, psi_mode="make_mt", cube=60.0)
    with engine.Engine(b) as e:
        e.upload_state(b.coords)
        t = e.tuning()
        e.set_tuning(**dict(t, step_block=block))
        res = e.autotune(0, 10)
        assert res["tuning"]["step_block"] == block and e.tuning()["step_block"] == block
