"""The one-launch cell-list rebuild against the tiled one (the same FP32
decisions, so the lists agree entry for entry), where it can go wrong: sizes
around the CTA, the table and the key limits, more hits than a bead keeps,
cells far out, coordinates that are not numbers, LJ without assembly lists."""
import numpy as np
import pytest

from mt_gb300 import synth

pytestmark = pytest.mark.gpu


def cloud(sizes, seed=1, box=30.0, **over):
    """Trajectories of free beads at random places, dimers in order."""
    rng = np.random.default_rng(seed)
    n = int(sum(sizes))
    off = np.zeros(len(sizes) + 1, np.int32)
    off[1:] = np.cumsum(sizes)
    c = np.zeros((n, 7), np.float32)
    local = np.concatenate([np.arange(k) for k in sizes])
    side = np.concatenate([np.full(k, box * max(1.0, k / 150.0) ** (1.0 / 3.0)) for k in sizes])
    c[:, :3] = rng.uniform(-0.5, 0.5, (n, 3)) * side[:, None]
    c[:, 3:6] = rng.uniform(-3.1, 3.1, (n, 3))
    last = np.concatenate([np.arange(k) == k - 1 for k in sizes])
    pair = ~(last & (local % 2 == 0))
    harm = np.where(local % 2 == 0, -(local + 1), local - 1).astype(np.int32)
    p = synth.default_params(seed=seed, **over)
    return synth.Batch(params=p, offsets=off, coords=c, mon_type=(local % 2).astype(np.int32),
                       fixed=np.zeros(n, np.uint8), extra=np.zeros(n, np.uint8), gtp=np.ones(n, np.int32),
                       on_tubule=np.zeros(n, np.int32), harmonic_count=pair.astype(np.int32),
                       harmonic=np.where(pair, harm, -1).astype(np.int32), zs=np.full(len(sizes), 160.0, np.float32))


def both(b, static=None):
    from mt_gb300 import engine
    out = []
    with engine.Engine(b, static_lists=static, force_ragged=True) as e:
        e.upload_state(b.coords)
        for method in (1, 2):
            e.set_list_method(method)
            try:
                e.rebuild_pairs()
                full = False
            except engine.MtgError as ex:   # too many bonds for the lists: both cut them off at the same entry
                assert ex.code == -3
                full = True
            out.append({"full": full} | {k: (v[0].copy(), [v[1][v[2] * i:v[2] * i + v[0][i]].tolist() for i in range(e.nb)])
                        for k, v in e.lists().items()})
    return out


def same(b, static=None):
    tiles, cells = both(b, static)
    assert tiles["full"] == cells["full"]
    for k in ("lj", "long", "lat"):
        assert np.array_equal(tiles[k][0], cells[k][0]), k
        assert tiles[k][1] == cells[k][1], k
    return tiles


@pytest.mark.parametrize("sizes", [(1, 2, 3, 31, 32, 33, 64), (511, 512, 513), (1024, 1025, 150), (8191, 8192), (8193,)],
                         ids=str)
def test_sizes(sizes):
    t = same(cloud(sizes))
    assert sum(sizes) < 40 or t["lj"][0].max() > 3


@pytest.mark.parametrize("box", [22.0, 14.0, 9.0])
def test_many_hits(box):
    """8, 16 and 32 hits a bead are passed, also past the keys a bead keeps."""
    t = same(cloud((150, 97), seed=3, box=box, ljpairscutoff=7.0))
    assert t["lj"][0].max() > (8, 16, 32)[(22.0, 14.0, 9.0).index(box)]


@pytest.mark.parametrize("sizes,box", [((150, 31) * 85, 14.0), ((150, 31) * 85, 9.0), ((300, 257) * 100, 14.0),
                                       ((600, 513) * 165, 22.0)], ids=["two", "two-many", "one", "full"])
def test_threads_a_bead(sizes, box):
    """Batches large enough for two threads a bead, one, and a thread for every bead of a CTA (the small ones have four)."""
    t = same(cloud(sizes, seed=4, box=box, ljpairscutoff=7.0))
    assert t["lj"][0].max() > 8


@pytest.mark.parametrize("over", [dict(ljpairscutoff=6.6), dict(ljpairscutoff=13.7), dict(is_wall=1)], ids=str)
def test_cutoffs(over):
    same(cloud((700, 300), seed=5, **over))


@pytest.mark.parametrize("cut", [11.0, 12.0, 17.0, 26.0])
def test_long_cutoffs(cut):
    """More hits than a bead's slots, several times as many, and more than the list holds; small
    trajectories with most beads past the slots take the tiles by themselves."""
    from mt_gb300 import engine
    same(synth.uniform_batch(synth.default_params(seed=9, ljpairscutoff=cut), 3, 40, 100, seed=9, radius=8.12,
                             psi_mode="make_mt", cube=60.0, thermal=0.05))
    t = same(cloud((450, 150, 3), seed=9, ljpairscutoff=cut))
    assert t["lj"][0].max() > 32 and t["full"] == (cut > 20)
    with engine.Engine(cloud((450, 150, 3), seed=9, ljpairscutoff=cut), force_ragged=True) as e:
        assert e.list_method() == (2 if cut <= 11.0 else 1)


def test_lj_without_assembly_lists():
    b = cloud((600, 41), seed=6, is_assembly=0, ljpairscutoff=5.0)

    class Static:
        long_count = np.zeros(b.nbeads, np.int32)
        lat_count = np.zeros(b.nbeads, np.int32)
        lon = np.zeros(b.nbeads * b.max_long, np.int32)
        lat = np.zeros(b.nbeads * b.max_lat, np.int32)
    same(b, Static)


def test_odd_coordinates():
    """Extra beads, clusters far out (past the clamped cells too), infinities and NaN."""
    b = cloud((400, 260, 90), seed=7)
    b.extra[5:400:7] = 1
    b.coords[100:140, :3] += np.float32(4.0e6)
    b.coords[140:180, :3] -= np.float32(3.0e8)
    b.coords[450:460, 0] = np.nan
    b.coords[460:465, 1] = np.inf
    b.coords[465:470, 4] = np.nan
    same(b)


def far_pairs(points, ends, **over):
    """One trajectory of pairs of monomers without a partner (points and ends [n, 3]), each with its axis
    along the pair, so that the longitudinal sites of the two face each other; every pair
    30 nm from the next along z."""
    n = 2 * len(points)
    b = cloud((n,), **over)
    b.coords[0::2, :3], b.coords[1::2, :3] = points, ends
    d = (b.coords[1::2, :3].astype(np.float64) - b.coords[0::2, :3])
    u = -d / np.linalg.norm(d, axis=1)[:, None]
    b.coords[:, 3] = 0
    b.coords[:, 4] = np.repeat(np.arccos(u[:, 2]), 2)
    b.coords[:, 5] = np.repeat(np.arctan2(u[:, 1], u[:, 0]), 2)
    b.harmonic_count[:] = 0
    b.harmonic[:] = -1
    return b


@pytest.mark.parametrize("offset", [2.0e5, 9.0e5, 3.9e6])
def test_sites_far_out(offset):
    """Bonds near the longest there are, so far out that a site's coordinates keep few digits."""
    rng = np.random.default_rng(int(offset))
    n = 1500
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    a = offset * rng.choice([-1.0, 1.0], (n, 3)) + rng.uniform(-50, 50, (n, 3))
    a[:, 2] += 30.0 * np.arange(n)
    a = a.astype(np.float32)
    t = same(far_pairs(a, (a + rng.uniform(6.0, 6.5, (n, 1)) * u).astype(np.float32)))
    assert t["long"][0].sum() > n / 8
