"""The descriptors from the one-launch ordered binning against the FP64 oracle
(odd sizes, extra beads, clusters far out) and against the general binning at the
largest size it takes, and the surrogate's kept scratch."""
import concurrent.futures as cf

import numpy as np
import pytest

from mt_gb300 import synth
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu
COLUMN_RTOL = 2e-5     # per feature column, as the suite's other descriptor checks


def cloud(sizes, seed, spread=1.0):
    rng = np.random.default_rng(seed)
    n = int(sum(sizes))
    off = np.zeros(len(sizes) + 1, np.int32)
    off[1:] = np.cumsum(sizes)
    c = np.zeros((n, 7), np.float32)
    side = np.concatenate([np.full(k, spread * 6.0 * k ** (1.0 / 3.0)) for k in sizes])
    c[:, :3] = rng.uniform(-0.5, 0.5, (n, 3)) * side[:, None]
    c[:, 3:6] = rng.uniform(-3, 3, (n, 3))
    p = synth.default_params(seed=seed, hdi_on=1, lj_on=0, is_assembly=1, tea_capricious=0)
    return synth.Batch(params=p, offsets=off, coords=c, mon_type=np.zeros(n, np.int32), fixed=np.zeros(n, np.uint8),
                       extra=np.zeros(n, np.uint8), gtp=np.ones(n, np.int32), on_tubule=np.zeros(n, np.int32),
                       harmonic_count=np.zeros(n, np.int32), harmonic=np.full(n, -1, np.int32),
                       zs=np.full(len(sizes), 160.0, np.float32))


def clear_of_shells(b):
    """No pair within FP32's error of a shell boundary (3e-7 of r, twice)."""
    for t in range(b.ntraj):
        x = b.coords[b.offsets[t]:b.offsets[t + 1], :3].astype(np.float64)
        r = np.linalg.norm(x[:, None] - x[None], axis=2)
        if any((np.abs(r - s) < 6e-7 * s).any() for s in (5.0, 10.0, 20.0)):
            return False
    return True


def columns(X, ref):
    for k in range(M.IN):
        assert np.linalg.norm(X[:, k] - ref[:, k]) <= COLUMN_RTOL * np.linalg.norm(ref[:, k]) + 1e-12, k


def descriptors(b):
    from mt_gb300 import engine
    with engine.Engine(b, force_ragged=True) as e:
        e.upload_state(b.coords)
        X = e.tea_training_data(targets=False)[0]
        assert np.array_equal(X, e.tea_training_data(targets=False)[0])     # the same bits every time
        return X


@pytest.mark.parametrize("sizes,spread", [((1, 2, 31, 33, 64), 1.0), ((511, 512, 513), 1.0), ((300, 200), 0.35),
                                          ((400, 150), 6.0)], ids=str)
def test_against_fp64(sizes, spread):
    seed = 1
    while not clear_of_shells(cloud(sizes, seed, spread)):
        seed += 1
    b = cloud(sizes, seed, spread)
    b.extra[len(b.extra) // 2::7] = 1
    b.coords[-20:, 0] += np.float32(2560.0)      # a cluster of its own, its cells 256 away
    X = descriptors(b)
    assert (X[b.extra != 0] == 0).all()
    columns(X, M.descriptors(b.coords, b.offsets, b.extra))


def test_largest_trajectory_equals_the_general_kernels():
    b = cloud((16384,), 3, 3.0)
    X = descriptors(b)
    g = cloud((16385,), 3)       # one bead more than the shared memory takes, an extra one
    g.coords[:16384] = b.coords
    g.extra[16384] = 1
    columns(X, descriptors(g)[:16384])


def test_large_batch_against_fp64():
    """400 copies of one trajectory: one thread a bead (the smaller batches have four)."""
    seed = 1
    while not clear_of_shells(cloud((151,), seed)):
        seed += 1
    one = cloud((151,), seed)
    b = cloud((151,) * 400, seed)
    b.coords[:] = np.tile(one.coords, (400, 1))
    X = descriptors(b)
    columns(X[:151], M.descriptors(one.coords, one.offsets, one.extra))
    assert np.array_equal(X, np.tile(X[:151], (400, 1)))


@pytest.mark.parametrize("n", [33, 129, 19_500])
def test_gradient_of_uneven_batches(n):
    """Batches that end inside a tile, and one with a second tile for some CTAs: the
    suite's bars for the gradient (see test_gpu_surrogate)."""
    from mt_gb300 import engine
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, M.IN)).astype(np.float32)
    T = rng.normal(0.9, 0.3, size=(n, M.OUT)).astype(np.float32)
    with engine.Surrogate(seed=7) as s:
        p, nrm = s.params()
        loss, g = s.loss_grad(X, T)
    Xn, Tn = M.normalise(X, T, nrm)
    want, gw = M.loss_grad(p, Xn, Tn, emulate_bf16=True)
    assert abs(loss - want) / want < 2e-3
    for a, b in zip((M.OFF_W1, M.OFF_W2, M.OFF_W3, M.OFF_W4, M.OFF_B), (M.OFF_W2, M.OFF_W3, M.OFF_W4, M.OFF_B, M.NPARAMS)):
        assert np.linalg.norm(g[a:b] - gw[a:b]) <= 2e-2 * np.linalg.norm(gw[a:b])


def test_surrogate_scratch():
    """Calls of any order of sizes, past the scratch that is kept, and from two threads
    at once give what a fresh surrogate gives."""
    from mt_gb300 import engine
    rng = np.random.default_rng(5)
    X = rng.normal(size=(50_000, M.IN)).astype(np.float32)
    T = rng.normal(size=(50_000, M.OUT)).astype(np.float32)
    sizes = (4096, 1, 50_000, 33, 129, 4096)

    def fresh(n):
        with engine.Surrogate(seed=9) as s:
            return s.predict(X[:n]), s.loss_grad(X[:n], T[:n])

    want = {n: fresh(n) for n in set(sizes)}

    def check(got, n):
        assert np.array_equal(got[0], want[n][0]) and got[1][0] == want[n][1][0]
        assert np.array_equal(got[1][1], want[n][1][1])

    with engine.Surrogate(seed=9) as s:
        for n in sizes:
            check((s.predict(X[:n]), s.loss_grad(X[:n], T[:n])), n)
        with cf.ThreadPoolExecutor(2) as pool:
            jobs = [(n, pool.submit(lambda n=n: (s.predict(X[:n]), s.loss_grad(X[:n], T[:n])))) for n in sizes * 3]
            for n, j in jobs:
                check(j.result(), n)


def test_a_trajectory_gets_the_same_bits_in_every_batch():
    """Descriptors of a batch with one thread a bead and a trajectory past the one-launch ordering, and of
    its parts with four threads a bead and in one launch."""
    from mt_gb300 import engine
    p = synth.default_params(seed=61, hdi_on=1)
    trajs = [synth.make_trajectory(pf, free, seed=61 + pf, radius=8.12, psi_mode="make_mt", cube=cube, thermal=0.05)
             for pf, free, cube in ((200, 2600, 120.0), (60, 700, 60.0), (31, 90, 50.0), (120, 1500, 90.0),
                                    (300, 12600, 260.0))]
    b = synth.batch_from_trajectories(p, [trajs[k % 4] for k in range(20)] + [trajs[4]])
    assert b.nbeads > 60000 and np.diff(b.offsets).max() > 16384
    with engine.Engine(b) as e, engine.ShardedEngine(b, [0] * 3) as s:
        e.upload_state(b.coords)
        s.upload_state(b.coords)
        whole, _ = e.tea_training_data(targets=False)
        assert np.array_equal(whole, np.concatenate([k.tea_training_data(targets=False)[0] for k in s.engines]))
