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
