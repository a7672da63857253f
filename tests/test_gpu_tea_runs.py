"""The all-pairs TEA passes cut their work into equal runs of (128 beads) x
(32-bead block) units: sizes around both, items held by one run and by many,
extra beads, and results that do not depend on which CTA finishes an item."""
import numpy as np
import pytest

from mt_gb300 import synth

pytestmark = pytest.mark.gpu
RTOL = 1e-5     # the suite's bar for FP32 sums against FP64, norm of the difference over norm


def batch(sizes, seed, extra=True):
    rng = np.random.default_rng(seed)
    n = int(sum(sizes))
    off = np.zeros(len(sizes) + 1, np.int32)
    off[1:] = np.cumsum(sizes)
    side = np.concatenate([np.full(k, 6.0 * k ** (1.0 / 3.0)) for k in sizes])
    c = np.zeros((n, 7), np.float32)
    c[:, :3] = rng.uniform(-0.5, 0.5, (n, 3)) * side[:, None]
    c[:, 3:6] = rng.uniform(-3, 3, (n, 3))
    ex = np.zeros(n, np.uint8)
    if extra:
        ex[off[-2] + 3:off[-1]:5] = 1
    p = synth.default_params(seed=seed, hdi_on=1, tea_a=2.0, tea_epsilon_freq=2, tea_capricious=0)
    return synth.Batch(params=p, offsets=off, coords=c, mon_type=(np.arange(n) % 2).astype(np.int32),
                       fixed=np.zeros(n, np.uint8), extra=ex, gtp=np.ones(n, np.int32),
                       on_tubule=np.zeros(n, np.int32), harmonic_count=np.zeros(n, np.int32),
                       harmonic=np.full(n, -1, np.int32), zs=np.full(len(sizes), 160.0, np.float32))


def tensors(x, a):
    """T_ij blocks [n, n, 3, 3] of one trajectory in FP64 (zero where i is j)."""
    d = x[None, :, :] - x[:, None, :]
    r = np.linalg.norm(d, axis=2)
    np.fill_diagonal(r, 1.0)
    u, ra = d / r[:, :, None], r / a
    far = ra > 2.0
    cii = np.where(far, 0.75 / ra * (1 + 2 / (3 * ra * ra)), 1 - 9 * ra / 32)
    crr = np.where(far, 0.75 / ra * (1 - 2 / (ra * ra)), 3 * ra / 32)
    T = cii[:, :, None, None] * np.eye(3) + crr[:, :, None, None] * u[:, :, :, None] * u[:, :, None, :]
    T[np.arange(len(x)), np.arange(len(x))] = 0.0
    return T


# the first three take a warp a bead, the last one the equal runs
@pytest.mark.parametrize("sizes", [(2, 31, 32, 33), (127, 128, 129), (300, 5, 417), (300, 5, 417) + (151,) * 40],
                         ids=lambda v: f"{len(v)}x{max(v)}")
def test_row_sums_against_fp64(sizes):
    from mt_gb300 import engine
    b = batch(sizes, 91)
    with engine.Engine(b) as e:
        e.upload_state(b.coords)
        _, _, ci, rc = e.tea_update()
        assert rc in (0, -5)
    for t in range(b.ntraj):
        s = slice(int(b.offsets[t]), int(b.offsets[t + 1]))
        act = b.extra[s] == 0
        x = b.coords[s, :3].astype(np.float64)
        T = tensors(x, b.params.tea_a)[:, act]
        want = (T ** 2).sum((1, 3))[act]
        got = ci[s, :3].astype(np.float64)[act]
        assert np.linalg.norm(got - want) <= RTOL * np.linalg.norm(want)
        assert (ci[s][~act] == 0).all()


@pytest.mark.parametrize("sizes", [(40, 130, 2000, 77), (3000,), (150,) * 300], ids=lambda v: f"{len(v)}x{max(v)}")
def test_same_bits_every_time(sizes):
    from mt_gb300 import engine
    b = batch(sizes, 92, extra=False)
    out = []
    for _ in range(3):
        with engine.Engine(b) as e:
            e.upload_state(b.coords)
            e.step(0, 4)
            out.append((e.download_state(), e.tea_update()[2]))
    assert np.isfinite(out[0][0]).all()
    for x, c in out[1:]:
        assert np.array_equal(x, out[0][0]) and np.array_equal(c, out[0][1])


# (sizes, extra): a CTA a few beads; items held by one run and by several, runs that end one item and begin
# the next; cuts at fine segments in batches of one and of several waves; cuts at coarse segments
PRODUCTS = [((299,), False), ((2, 31, 33, 129, 300), True), ((3100,), True), ((1500, 40, 1700, 3000), True),
            ((130,) * 70 + (2400,), True), ((900, 77) * 45, False), ((1600, 1590) * 60, False)]


@pytest.mark.parametrize("sizes,extra", PRODUCTS, ids=lambda v: f"{len(v)}x{max(v)}" if isinstance(v, tuple) else str(v))
def test_mobility_product_against_fp64(sizes, extra):
    """Effective forces of the exact product in FP64 from the engine's own F, R, C_i and beta,
    on both sides of the small form's limits, with overlapping pairs.  Bar: a term carries about a dozen FP32
    roundings (6e-8 each) and three approximations (1.3e-7), 1.1e-6 of |T||g|, and the sums of
    at most 64 blocks' terms in one accumulator and 48 segments' sums as much again at most: 4e-6."""
    from mt_gb300 import engine
    b = batch(sizes, 93, extra)
    with engine.Engine(b) as e:
        e.upload_state(b.coords)
        e.rebuild_pairs()
        F = e.compute_forces()[:, :3].astype(np.float64)
        _, beta, ci, rc = e.tea_update()
        assert rc in (0, -5)
        fe, _, R = e.tea_effective_forces(exact=True, farfield=False)
    check = range(b.ntraj) if b.ntraj < 10 else [0, 1, b.ntraj // 2, b.ntraj - 2, b.ntraj - 1]
    for t in check:
        s = slice(int(b.offsets[t]), int(b.offsets[t + 1]))
        act = b.extra[s] == 0
        x, f = b.coords[s, :3].astype(np.float64)[act], F[s][act]
        c = 1.0 / np.sqrt(1.0 + float(beta[t]) ** 2 * ci[s, :3].astype(np.float64)[act])
        r = R[s, :3].astype(np.float64)[act]
        got = fe[s, :3].astype(np.float64)[act]
        for i in range(0, len(x), 500):
            k = slice(i, min(len(x), i + 500))
            d = x[None, :, :] - x[k][:, None, :]
            rr = np.linalg.norm(d, axis=2)
            rr[np.arange(k.stop - k.start), np.arange(k.start, k.stop)] = 1.0
            u, ra = d / rr[:, :, None], rr / b.params.tea_a
            far = ra > 2.0
            cii = np.where(far, 0.75 / ra * (1 + 2 / (3 * ra * ra)), 1 - 9 * ra / 32)
            crr = np.where(far, 0.75 / ra * (1 - 2 / (ra * ra)), 3 * ra / 32)
            for w in (cii, crr):
                w[np.arange(k.stop - k.start), np.arange(k.start, k.stop)] = 0.0
            g = f[None, :, :] + float(beta[t]) * c[k][:, None, :] * r[None, :, :]
            ug = np.einsum("ija,ija->ij", u, g)
            want = f[k] + c[k] * r[k] + np.einsum("ij,ija->ia", cii, g) + np.einsum("ij,ija->ia", crr * ug, u)
            size = (np.einsum("ij,ija->ia", np.abs(cii), np.abs(g)) + np.einsum("ij,ija->ia", np.abs(crr)
                    * np.einsum("ija,ija->ij", np.abs(u), np.abs(g)), np.abs(u)) + np.abs(f[k]) + np.abs(r[k]))
            assert (np.abs(got[k] - want) <= 4.0e-6 * size).all()


@pytest.mark.parametrize("sizes", [(299, 151, 33, 1520), (130,) * 70 + (2400,), (3300,) * 12, (1600, 1590, 40) * 40,
                                   (5600,) * 30], ids=lambda v: f"{len(v)}x{max(v)}")
def test_a_trajectory_gets_the_same_bits_in_every_batch(sizes):
    """A batch on one engine and cut over four, where the whole takes equal runs cut at fine or at coarse
    segments and the parts others or the small form: state, noise streams and C_i."""
    from mt_gb300 import engine
    b = batch(sizes, 94)
    with engine.Engine(b) as e, engine.ShardedEngine(b, [0] * 4) as s:
        e.upload_state(b.coords)
        s.upload_state(b.coords)
        e.step(0, 3)
        s.step(0, 3)
        x = e.download_state()
        assert np.isfinite(x).all() and np.array_equal(x, s.download_state())
        assert np.array_equal(e.download_rng(), s.download_rng())
        whole, parts = e.tea_update(), [k.tea_update() for k in s.engines]
        for v in range(3):
            assert np.array_equal(whole[v], np.concatenate([p[v] for p in parts]))
