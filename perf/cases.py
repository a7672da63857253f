"""What a user of the engine has it do, as cases that can be timed and checked.

Six kinds of work, each through the public Python binding (mt_gb300.engine):

  plain    assembly-mode Brownian dynamics without hydrodynamics: a call of
           mtg_step over `steps` MD steps (pair lists rebuilt every 10), then the
           state read back, which is how a program's output loop uses it
  static   the same with the lists given once (non-assembly mode), lateral and
           longitudinal barriers and walls on, and the work of an output stride:
           energy totals, microtubule lengths, the state
  frames   re-analysis of stored frames: upload, pair lists, forces, energies per bead
  tea      exact TEA hydrodynamics (all-pairs mobility product)
  learned  learned TEA: the network's coefficients, the far field of the
           mobility product, the exact re-check every 100 steps
  fit      one sample of training data from the engine (descriptors, exact
           targets) and the loss gradient of the network on a batch of it

Sizes are those of the benchmark's workloads and of the tests: trajectories of
a 13-protofilament lattice of `pf` monomers per protofilament plus `free` free
monomers, `ntraj` of them (`ragged`: sizes uneven up to these).  `exact` gives
the same results in 64 bits from plain torch operations.
"""
import ctypes
import math

import numpy as np
import torch

from mt_gb300 import engine, synth

KB = 0.0019872041


def listed():
    return [
        # one microtubule seed, one pair-list period per call: a program that
        # looks at the state after every few steps; latency and launches count
        dict(name="plain_seed_call", kind="plain", ntraj=1, pf=12, free=0, ragged=False, steps=10, persistent=0),
        # the same seed run for long between two looks, with the tuned launch shape
        dict(name="plain_seed_run", kind="plain", ntraj=1, pf=12, free=0, ragged=False, steps=1000, persistent=1),
        # one microtubule growing from free tubulin: the reference program's ordinary run
        dict(name="plain_one_1520", kind="plain", ntraj=1, pf=40, free=1000, ragged=False, steps=200, persistent=0),
        # a batch of replicas of it
        dict(name="plain_batch_256x1520", kind="plain", ntraj=256, pf=40, free=1000, ragged=False, steps=100,
             persistent=0),
        # the largest: a thousand uneven trajectories, odd sizes
        dict(name="plain_ragged_1024", kind="plain", ntraj=1024, pf=120, free=2000, ragged=True, steps=50,
             persistent=0),
        # lattices with fixed partner lists, barriers and walls, one output stride
        dict(name="static_stride_101x780", kind="static", ntraj=101, pf=60, free=0, ragged=False, steps=100),
        # stored frames of uneven trajectories analysed again
        dict(name="frames_97", kind="frames", ntraj=97, pf=91, free=1501, ragged=True, steps=0),
        # hydrodynamics of one small system: few CTAs, latency
        dict(name="tea_one_299", kind="tea", ntraj=1, pf=15, free=104, ragged=False, steps=100, slices=0, jparts=0),
        # the benchmark's exact-TEA configuration, with its tuned launch shapes
        dict(name="tea_16x3300", kind="tea", ntraj=16, pf=100, free=2000, ragged=False, steps=20, slices=4, jparts=4),
        # exact TEA at the size of the learned comparison
        dict(name="tea_64x5600", kind="tea", ntraj=64, pf=200, free=3000, ragged=False, steps=10, slices=0, jparts=0),
        # learned TEA at that size: a re-check period
        dict(name="learned_64x5600", kind="learned", ntraj=64, pf=200, free=3000, ragged=False, steps=100),
        # training data of uneven systems and a gradient on one batch of 4096
        dict(name="fit_8_ragged", kind="fit", ntraj=8, pf=140, free=1500, ragged=True, steps=0, samples=4096),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "static", "frames", "tea", "tea", "learned", "fit"])
    if kind == "plain":
        ragged = rng.random() < 0.5
        pf, free = rng.randint(8, 120), rng.choice([0, rng.randint(1, 1000) * 2])
        n = 13 * pf + free
        # a call's work: at most that of the largest listed case
        ntraj = _logint(rng, 1, max(1, min(1024, 1_900_000 // n)))
        steps = max(1, min(_logint(rng, 10, 1000), 90_000_000 // (n * ntraj)))
        return dict(kind=kind, ntraj=ntraj, pf=pf, free=free, ragged=ragged, steps=steps,
                    persistent=int(n <= 2048 and rng.random() < 0.3))
    if kind == "static":
        return dict(kind=kind, ntraj=_logint(rng, 1, 256), pf=rng.randint(8, 120), free=0, ragged=False,
                    steps=_logint(rng, 10, 200))
    if kind == "frames":
        return dict(kind=kind, ntraj=_logint(rng, 1, 256), pf=rng.randint(8, 120), free=2 * rng.randint(0, 1000),
                    ragged=True, steps=0)
    if kind == "tea":
        pf, free = _logint(rng, 8, 200), 2 * rng.randint(0, 1500)
        n = 13 * pf + free
        ntraj = _logint(rng, 1, max(1, min(64, int(2.0e9 // (n * n)))))
        tuned = rng.random() < 0.5
        return dict(kind=kind, ntraj=ntraj, pf=pf, free=free, ragged=rng.random() < 0.5,
                    steps=max(10, min(100, int(2.0e10 // (n * n * ntraj)))),
                    slices=rng.choice([2, 4, 8]) if tuned else 0, jparts=rng.choice([1, 2, 4]) if tuned else 0)
    if kind == "learned":
        return dict(kind=kind, ntraj=_logint(rng, 4, 64), pf=rng.randint(60, 200), free=2 * rng.randint(300, 1500),
                    ragged=rng.random() < 0.5, steps=100)
    return dict(kind=kind, ntraj=rng.randint(2, 8), pf=rng.randint(40, 140), free=2 * rng.randint(0, 750),
                ragged=True, steps=0, samples=rng.randint(33, 5000))


# ------------------------------------------------------------------ inputs
TEMPLATES = 12     # distinct placements of a batch; every trajectory is one of them, cut, turned and jittered


def _system(case, seed):
    """The batch (numpy arrays of a synth.Batch), its noise streams and, for
    the static kind, its partner lists, from the seed alone."""
    rng = np.random.default_rng([seed, case["ntraj"], case["pf"], case["free"]])
    sizes = np.random.default_rng([case["ntraj"], case["pf"], case["free"]])     # a case's sizes are the same for every seed
    kind, nt, pf, free = case["kind"], case["ntraj"], case["pf"], case["free"] // 2 * 2
    tea = kind in ("tea", "learned", "fit")
    over = {}
    if kind == "static":
        over = dict(is_assembly=0, barrier=1, is_wall=1, rep_r=60.0, rep_eps=0.05)
    p = synth.default_params(seed=1 + seed % 1000, hdi_on=int(tea), tea_a=2.0, tea_epsilon_freq=10, **over)
    lattice = dict(radius=8.12, psi_mode="make_mt") if kind in ("static", "frames") else {}
    cube = 150.0 if 13 * pf + free > 3400 or case["ragged"] else 100.0
    temps, ntemp = [], min(nt, TEMPLATES)
    for k in range(ntemp):
        n_mon = pf
        if case["ragged"] and k:
            n_mon = int(sizes.integers(8, pf + 1))
        bent = case["ragged"] and rng.random() < 0.3
        temps.append(synth.make_trajectory(n_mon, free, seed=int(rng.integers(1 << 30)), cube=cube,
                                           tail=min(n_mon, 6) if bent else 0,
                                           bend=float(rng.uniform(0.1, 0.3)) if bent else 0.0, **lattice))
    trajs = []
    for t in range(nt):
        T = temps[t % ntemp]
        n = T.n
        if case["ragged"] and t:
            n = T.n_lattice + int(sizes.integers(0, (T.n - T.n_lattice) // 2 + 1)) * 2
        c = T.coords[:n].copy()
        turn = 2 * math.pi * float(rng.random())
        cs, sn = math.cos(turn), math.sin(turn)
        c[:, 0], c[:, 1] = cs * T.coords[:n, 0] - sn * T.coords[:n, 1], sn * T.coords[:n, 0] + cs * T.coords[:n, 1]
        c[:, 5] += turn if kind in ("static", "frames") else 0.0
        c[:, :6] += rng.normal(0.0, 0.03, size=(n, 6)).astype(np.float32)
        trajs.append((T, n, c))
    counts = [n for _, n, _ in trajs]
    off = np.zeros(nt + 1, np.int32)
    off[1:] = np.cumsum(counts)

    def cat(f):
        return np.concatenate([f(T)[:n] for T, n, _ in trajs])

    harm, count = {}, {}
    for T in temps:     # dimers: neighbours in order with the same residue and chain
        i = np.arange(T.n)
        same = (T.resid[:-1] == T.resid[1:]) & (T.chain[:-1] == T.chain[1:])
        h, hc = np.full(T.n, -1, np.int32), np.zeros(T.n, np.int32)
        h[:-1][same], hc[:-1][same] = -i[1:][same], 1
        h[1:][same], hc[1:][same] = i[:-1][same], 1
        harm[id(T)], count[id(T)] = h, hc
    b = synth.Batch(
        params=p, offsets=off, coords=np.ascontiguousarray(np.concatenate([c for _, _, c in trajs])),
        mon_type=cat(lambda T: T.mon_type).astype(np.int32), fixed=cat(lambda T: (T.resid <= 1).astype(np.uint8)),
        extra=cat(lambda T: T.extra), gtp=cat(lambda T: T.gtp).astype(np.int32),
        on_tubule=np.zeros(int(off[-1]), np.int32), harmonic_count=cat(lambda T: count[id(T)]),
        harmonic=cat(lambda T: harm[id(T)]), zs=np.array([T.zs for T, _, _ in trajs], np.float32))
    if len(set(counts)) == 1 and kind != "static":
        b.uniform_ntot = counts[0]
    streams = rng.integers(128, 1 << 32, size=8 * b.nbeads, dtype=np.uint32)
    lists = _static_lists(temps[0], nt, b) if kind == "static" else None
    return b, streams, lists


class _Lists:
    pass


def _static_lists(T, nt, b):
    """Partners of the ideal lattice: along the protofilament between dimers,
    and the facing lateral sites (the sign says which site)."""
    n = T.n
    n_mon = n // 13
    lc, lon = np.zeros(n, np.int32), np.zeros((n, b.max_long), np.int32)
    for g in range(n):
        m = g % n_mon
        if m % 2 == 1 and m + 1 < n_mon:
            lon[g, 0], lc[g] = -(g + 1), 1
        elif m % 2 == 0 and m > 0:
            lon[g, 0], lc[g] = g - 1, 1
    ideal = synth.make_lattice(n_mon, 8.12, "make_mt")[0]
    R = _Ref.sites(torch.from_numpy(ideal[:, :6].astype(np.float64)))
    x = torch.from_numpy(ideal[:, :3].astype(np.float64))
    tc, lat = np.zeros(n, np.int32), np.zeros((n, b.max_lat), np.int32)
    near1 = torch.cdist(x + R[1], x + R[2]) < 1.0
    near2 = torch.cdist(x + R[2], x + R[1]) < 1.0
    for near, sign in ((near1, -1), (near2, 1)):
        for i, j in near.nonzero().tolist():
            if i != j:
                lat[i, tc[i]] = sign * (j if j else synth.ZERO_CODE)
                tc[i] += 1
    L = _Lists()
    L.long_count, L.lat_count = np.tile(lc, nt), np.tile(tc, nt)
    L.lon, L.lat = np.ascontiguousarray(np.tile(lon.reshape(-1), nt)), np.ascontiguousarray(np.tile(lat.reshape(-1), nt))
    return L


def _network(seed, X, T):
    """Weights of a network that has not been trained yet and the
    normalisation of a sample (three significant digits)."""
    g = torch.Generator().manual_seed(seed)
    parts = []
    for out, inp in ((128, 32), (128, 128), (128, 128), (4, 128)):
        parts.append(torch.randn(out * inp, generator=g, dtype=torch.float64) * math.sqrt(2.0 / (out + inp)))
    for out in (128, 128, 128, 4):
        parts.append(torch.randn(out, generator=g, dtype=torch.float64) * 0.05)
    params = torch.cat(parts).numpy().astype(np.float32)

    def three(a):
        return np.array([float("%.3g" % v) for v in a], np.float32)

    X, T = np.asarray(X, np.float64), np.asarray(T, np.float64)
    sx, st = X.std(0), T.std(0)
    norm = np.concatenate([three(X.mean(0)), three(np.where(sx > 1e-6, 1.0 / np.maximum(sx, 1e-6), 1.0)),
                           three(T.mean(0)), three(np.where(st > 1e-6, st, 1.0))])
    return params, norm


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    b, streams, lists = _system(case, seed)
    eng = engine.Engine(b, static_lists=lists)
    eng.upload_state(b.coords)
    eng.upload_rng(streams)
    s = dict(case=case, engine=eng, step=0, out=torch.empty((b.nbeads, 7), dtype=torch.float32, pin_memory=True))
    kind = case["kind"]
    tune = eng.tuning()
    if case.get("persistent"):
        tune["plain_persistent"] = 1
        eng.set_tuning(**tune)
    if case.get("slices"):
        tune.update(tea_slices=case["slices"], tea_jparts=case["jparts"])
        eng.set_tuning(**tune)
    if kind == "frames":
        s["frames"] = [torch.from_numpy(b.coords).pin_memory().numpy()]
    elif kind == "learned":
        X, T = eng.tea_training_data()
        net = engine.Surrogate(seed=1 + seed % 97)
        net.train(X, T, epochs=4, batch=4096 if len(X) >= 8192 else 512, lr=1e-3, seed=seed % 1009)
        eng.set_surrogate(net, recheck_every=100, max_err=0.1)
        eng.set_tea_farfield(True, 0.85, refresh_every=1000)
    elif kind == "fit":
        X, T = eng.tea_training_data()
        s["net"] = engine.Surrogate(seed=1)
        s["net"].set_params(*_network(seed, X, T))
    return s


def _state(s):
    """The state into the program's page-locked buffer."""
    ptr = ctypes.cast(s["out"].data_ptr(), ctypes.POINTER(ctypes.c_float))
    engine.check(s["engine"].lib.mtg_download_state(s["engine"].h, ptr, None))
    return s["out"]


def run(s):
    case, eng = s["case"], s["engine"]
    kind = case["kind"]
    if kind == "frames":
        eng.upload_state(s["frames"][0])
        eng.rebuild_pairs()
        total, per_bead = eng.energies(per_bead=True)
        return dict(forces=eng.compute_forces(), energies=per_bead, totals=total)
    if kind == "fit":
        X, T = eng.tea_training_data()
        n = min(case["samples"], len(X))
        loss, grad = s["net"].loss_grad(X[:n], T[:n])
        return dict(X=X, T=T, loss=loss, grad=grad)
    eng.step(s["step"], case["steps"])
    s["step"] += case["steps"]
    if kind == "static":
        # the numbers of a stride's log lines
        return dict(totals=eng.energies().astype(np.float32), length=eng.mt_length(True), state=_state(s))
    return dict(state=_state(s))


def work(case):
    """Bytes: every bead's state and noise streams in and out once, and what is
    returned.  Operations: the pair and bead arithmetic of every step."""
    grow = 0.5 if case["ragged"] and case["ntraj"] > 1 else 1.0
    n = 13 * case["pf"] * (0.56 if grow < 1 else 1.0) + case["free"] * grow
    nb, steps, kind = case["ntraj"] * n, case["steps"], case["kind"]
    if kind == "frames":
        return dict(bytes=nb * (28 + 28 + 56), flops=nb * 600)
    if kind == "fit":
        return dict(bytes=nb * (24 + 36 * 4) + 37764 * 4, flops=nb * n * 44 + case["samples"] * 74752 * 3)
    state = nb * (24 + 24 + 32 + 32)
    if kind == "tea":
        return dict(bytes=state, flops=nb * n * (45 * steps + 44 * steps / 10) + nb * 400 * steps)
    if kind == "learned":
        near = min(n, 600)
        return dict(bytes=state, flops=nb * steps * (45 * near + 90 * 95 + 400) + nb * 74752 * steps / 10 +
                    nb * n * 89 * steps / 100)
    return dict(bytes=state, flops=nb * steps * 400)


# ------------------------------------------------------------------ 64 bits
class _Ref:
    """The engine's steps in 64 bits with torch operations."""

    def __init__(self, b, streams, lists):
        d = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.d, self.nb, self.nt = b.params, d, b.nbeads, b.ntraj
        self.off = b.offsets.tolist()
        self.traj = torch.from_numpy(np.repeat(np.arange(b.ntraj), np.diff(b.offsets))).to(d)
        self.base = torch.from_numpy(b.offsets[:-1].astype(np.int64)).to(d)[self.traj]
        self.local = torch.arange(self.nb, device=d) - self.base
        self.s = torch.from_numpy(b.coords[:, :6].astype(np.float64)).to(d)     # x y z fi theta psi

        def dev(a):
            return torch.from_numpy(np.asarray(a).astype(np.int64)).to(d)

        self.extra, self.fixed = dev(b.extra).bool(), dev(b.fixed).bool()
        self.beta, self.gtp, self.on = dev(b.mon_type) != 0, dev(b.gtp) == 1, dev(b.on_tubule) != 0
        self.h = dev(b.harmonic)
        self.has_h = dev(b.harmonic_count) > 0
        self.zs = torch.from_numpy(b.zs.astype(np.float64)).to(d)[self.traj]
        self.seeds = dev(streams).reshape(2, self.nb, 4)
        self.static = lists is not None
        empty = torch.zeros(0, dtype=torch.int64, device=d)
        self.lj = self.lon = self.lat = (empty, empty, empty)
        if lists is not None:
            i, k = dev(np.nonzero(np.arange(b.max_long) < lists.long_count[:, None])).unbind()
            e = dev(lists.lon).reshape(self.nb, -1)[i, k]
            self.lon = (i, self.base[i] + e.abs(), torch.where(e < 0, 2, -2))
            i, k = dev(np.nonzero(np.arange(b.max_lat) < lists.lat_count[:, None])).unbind()
            e = dev(lists.lat).reshape(self.nb, -1)[i, k]
            j = torch.where(e.abs() == synth.ZERO_CODE, torch.zeros_like(e), e.abs())
            self.lat = (i, self.base[i] + j, (e <= 0).long())

    @staticmethod
    def sites(s):
        """Axis, lateral site 1, lateral site 2 in the lab frame."""
        sf, cf = torch.sin(s[:, 3]), torch.cos(s[:, 3])
        st, ct = torch.sin(s[:, 4]), torch.cos(s[:, 4])
        sp, cp = torch.sin(s[:, 5]), torch.cos(s[:, 5])
        c0 = torch.stack([cp * ct, sp * ct, -st], 1)
        c1 = torch.stack([cp * st * sf - sp * cf, sp * st * sf + cp * cf, ct * sf], 1)
        c2 = torch.stack([cp * st * cf + sp * sf, sp * st * cf - cp * sf, ct * cf], 1)
        a = 2.0 * math.pi / 13.0
        px, py, pz = 0.5 * 8.12 * (math.cos(a) - 1.0), 0.5 * 8.12 * math.sin(a), -6.0 / 13.0
        return c2, px * c0 + py * c1 + pz * c2, px * c0 - py * c1 - pz * c2

    def near(self, cut):
        """All ordered pairs of a trajectory closer than cut, several trajectories at a time."""
        order = sorted(range(self.nt), key=lambda t: self.off[t + 1] - self.off[t])
        found, k = [], 0
        while k < self.nt:
            m, n = k, 0
            while m < self.nt:
                n1 = self.off[order[m] + 1] - self.off[order[m]]
                if m > k and (m + 1 - k) * n1 * n1 > 40_000_000:
                    break
                n, m = n1, m + 1
            ts = torch.tensor(order[k:m], device=self.d)
            o0 = torch.tensor(self.off, device=self.d)
            idx = o0[ts][:, None] + torch.arange(n, device=self.d)
            ok = idx < o0[ts + 1][:, None]
            x = torch.where(ok[:, :, None], self.s[idx.clamp(max=self.nb - 1), :3], torch.tensor(1e9, device=self.d, dtype=torch.float64))
            x = x + torch.where(ok, 0.0, 1e3 * torch.arange(n, device=self.d))[:, :, None]
            d2 = (x[:, :, None, 0] - x[:, None, :, 0]) ** 2
            d2 += (x[:, :, None, 1] - x[:, None, :, 1]) ** 2
            d2 += (x[:, :, None, 2] - x[:, None, :, 2]) ** 2
            t, i, j = (d2 < cut * cut).nonzero().unbind(1)
            keep = ok[t, i] & ok[t, j]
            found.append((idx[t, i][keep], idx[t, j][keep]))
            k = m
        i, j = (torch.cat(v) for v in zip(*found))
        return i, j

    def rebuild(self):
        p = self.p
        if not (p.lj_on or p.is_assembly):
            return
        i, j = self.near(max(p.ljpairscutoff if p.lj_on else 0.0, 6.6 if p.is_assembly else 0.0))
        keep = ~self.extra[i]
        i, j = i[keep], j[keep]
        x = self.s[:, :3]
        dist = (x[i] - x[j]).norm(dim=1)
        if p.lj_on:
            m = (i != j) & (dist < p.ljpairscutoff)
            self.lj = (i[m], j[m], None)
        if p.is_assembly:
            m = (dist < 6.6) & (self.local[j] != self.h[i].abs())
            i, j = i[m], j[m]
            uz, s1, s2 = self.sites(self.s)
            r = torch.where(self.h[i] < 0, -2.0, 2.0)[:, None]
            m = (self.beta[i] != self.beta[j]) & ((x[j] - r * uz[j] - x[i] - r * uz[i]).norm(dim=1) < 2.5)
            side = torch.where((self.h[i] >= 0) & (self.local[j] != 0), 2, -2)
            self.lon = (i[m], j[m], side[m])
            a = (i != j) & ((x[j] + s2[j] - x[i] - s1[i]).norm(dim=1) < 2.5)
            c = (i != j) & ((x[j] + s1[j] - x[i] - s2[i]).norm(dim=1) < 2.5)
            self.lat = (torch.cat([i[a], i[c]]), torch.cat([j[a], j[c]]),
                        torch.cat([torch.ones_like(i[a]), torch.zeros_like(i[c])]))

    def bonds(self):
        """Axial bonds (harmonic, longitudinal) and lateral bonds with their site vectors."""
        x = self.s[:, :3]
        uz, s1, s2 = self.sites(self.s)
        hi = (self.has_h & ~self.extra).nonzero()[:, 0]
        out = []
        for i, j, r in ((hi, self.base[hi] + self.h[hi].abs(), torch.where(self.h[hi] < 0, 2, -2)), self.lon):
            m = ~self.extra[i]
            i, j, r = i[m], j[m], r[m].double()[:, None]
            out.append((i, j, r[:, 0], r * uz[i], x[j] - r * uz[j] - x[i] - r * uz[i]))
        i, j, first = self.lat
        m = ~self.extra[i]
        i, j, first = i[m], j[m], first[m].bool()[:, None]
        w = torch.where(first, s1[i], s2[i])
        out.append((i, j, None, w, x[j] + torch.where(first, s2[j], s1[j]) - x[i] - w))
        return out

    def th0(self, g):
        return torch.where(self.gtp[g], float(self.p.theta0_gtp), float(self.p.theta0_gdp))

    def forces(self):
        p, s = self.p, self.s
        x = s[:, :3]
        f, t, a = (torch.zeros(self.nb, 3, dtype=torch.float64, device=self.d) for _ in range(3))   # a: fi theta psi

        def pair(i, dU, d, w):
            f.index_add_(0, i, dU[:, None] * d)
            t.index_add_(0, i, dU[:, None] * torch.linalg.cross(w, d))

        def bend(i, j, r, dr, th0):
            m = dr < 1.0
            i, j, sg, th0 = i[m], j[m], torch.sign(r[m]), th0[m]
            v = torch.stack([p.B_fi * sg * torch.sin(sg * (s[j, 3] - s[i, 3]) - p.fi_0),
                             p.B_theta * sg * torch.sin(sg * (s[j, 4] - s[i, 4]) - th0),
                             p.B_psi * sg * torch.sin(sg * (s[j, 5] - s[i, 5]) - p.psi_0)], 1)
            a.index_add_(0, i, v)

        def morse(D, A, r):
            e = torch.exp(-A * r)
            return 2.0 * A * D * (1.0 - e) * e

        def barrier(h, r0, w, r):
            return -h * torch.exp(-(r - r0) ** 2 / (2.0 * w * w)) * (r - r0) / (w * w)

        H, L, T = self.bonds()
        i, j, r, w, d = H
        pair(i, torch.full_like(r, float(p.C)), d, w)
        bend(i, j, r, d.norm(dim=1), self.th0(i))
        i, j, r, w, d = L
        dr = d.norm(dim=1)
        off = ~self.on[i] & ~self.on[j]
        dU = morse(p.D_long, p.A_long, dr)
        if p.barrier:
            dU = dU + off * barrier(p.a_barr_long, p.r_barr_long, p.w_barr_long, dr)
        pair(i, dU / dr, d, w)
        bend(i, j, r, dr, torch.where(x[i, 2] > x[j, 2], self.th0(i), self.th0(j)))
        i, j, _, w, d = T
        dr = d.norm(dim=1)
        off = ~self.on[i] & ~self.on[j]
        dU = morse(torch.where(self.beta[i] != self.beta[j], p.D_lat / p.seam_coeff, p.D_lat), p.A_lat, dr)
        if p.barrier:
            dU = dU + off * barrier(p.a_barr_lat, p.r_barr_lat, p.w_barr_lat, dr)
        pair(i, dU / dr, d, w)
        if p.lj_on:
            i, j, _ = self.lj
            d = x[i] - x[j]
            r2 = (d * d).sum(1)
            m = r2 < 36.0
            f.index_add_(0, i[m], (p.ljscale * p.ljsigma6 * 6.0 / r2[m] ** 4)[:, None] * d[m])
        if p.is_wall:
            z, top = x[:, 2], self.zs + p.rep_leftborder
            f[:, 2] += torch.where(z < p.rep_leftborder, p.rep_eps * (z - p.rep_leftborder).abs(),
                                   torch.where(z > top, -p.rep_eps * (z - top).abs(), 0.0)) * ~self.extra
            rad = x[:, :2].norm(dim=1)
            f[:, :2] += torch.where((rad > p.rep_r) & ~self.extra, -p.rep_eps * (rad - p.rep_r) / rad, 0.0)[:, None] * x[:, :2]
        st, ct, sp, cp = torch.sin(s[:, 4]), torch.cos(s[:, 4]), torch.sin(s[:, 5]), torch.cos(s[:, 5])
        a[:, 0] += cp * ct * t[:, 0] + sp * ct * t[:, 1] - st * t[:, 2]
        a[:, 1] += -sp * t[:, 0] + cp * t[:, 1]
        a[:, 2] += t[:, 2]
        f[self.extra], a[self.extra] = 0.0, 0.0
        return f, a

    def energies(self):
        p, s = self.p, self.s
        U = torch.zeros(self.nb, 7, dtype=torch.float64, device=self.d)

        def add(k, i, v):
            U[:, k].index_add_(0, i, v)

        def bend(i, j, dr, dth):
            m = dr < 1.0
            i, j = i[m], j[m]
            add(3, i, p.B_psi * (1.0 - torch.cos(s[i, 5] - s[j, 5] - p.psi_0)))
            add(4, i, p.B_fi * (1.0 - torch.cos(s[i, 3] - s[j, 3] - p.fi_0)))
            add(5, i, p.B_theta * (1.0 - torch.cos(dth[m])))

        def morse(D, A, r):
            return D * (1.0 - torch.exp(-A * r)) ** 2 - D

        H, L, T = self.bonds()
        i, j, _, _, d = H
        dr = d.norm(dim=1)
        add(0, i, p.C / 2.0 * dr * dr)
        bend(i, j, dr, s[j, 4] - s[i, 4] - self.th0(i))
        i, j, _, _, d = L
        dr = d.norm(dim=1)
        add(1, i, morse(p.D_long, p.A_long, dr))
        bend(i, j, dr, s[i, 4] - s[j, 4] - torch.where(s[i, 2] > s[j, 2], self.th0(i), self.th0(j)))
        if p.barrier:
            off = ~self.on[i] & ~self.on[j]
            add(1, i, off * p.a_barr_long * torch.exp(-(dr - p.r_barr_long) ** 2 / (2.0 * p.w_barr_long ** 2)))
        i, j, _, _, d = T
        dr = d.norm(dim=1)
        add(2, i, morse(torch.where(self.beta[i] != self.beta[j], p.D_lat / p.seam_coeff, p.D_lat), p.A_lat, dr))
        if p.barrier:
            off = ~self.on[i] & ~self.on[j]
            add(2, i, off * p.a_barr_lat * torch.exp(-(dr - p.r_barr_lat) ** 2 / (2.0 * p.w_barr_lat ** 2)))
        if p.lj_on:
            i, j, _ = self.lj
            r2 = ((s[i, :3] - s[j, :3]) ** 2).sum(1)
            m = r2 < 36.0
            add(6, i[m], p.ljscale * p.ljsigma6 / r2[m] ** 3)
        return U / 2.0

    def totals(self, U):
        out = torch.zeros(self.nt, 7, dtype=torch.float64, device=self.d)
        return out.index_add_(0, self.traj, U)

    def normals(self, half, who):
        """Four normal deviates of each stream of `who`, the streams advanced."""
        z = self.seeds[half][who]
        mask32 = 0xffffffff

        def word():
            v = torch.zeros_like(z[:, 0])
            for c, (s1, s2, s3, m) in enumerate(((13, 19, 12, 4294967294), (2, 25, 4, 4294967288), (3, 11, 17, 4294967280))):
                b = ((((z[:, c] << s1) & mask32) ^ z[:, c]) >> s2)
                z[:, c] = (((z[:, c] & m) << s3) & mask32) ^ b
                v ^= z[:, c]
            z[:, 3] = (1664525 * z[:, 3] + 1013904223) & mask32
            v ^= z[:, 3]
            u = (v & 0x7fffff).double() / (1 << 23)
            return torch.where(u == 0.0, 1.0e-8, u)

        out = []
        for _ in range(2):
            u1, u2 = word(), word()
            r, a = torch.sqrt(-2.0 * torch.log(u1)), 2.0 * math.pi * u2
            out += [r * torch.sin(a), r * torch.cos(a)]
        self.seeds[half][who] = z
        return torch.stack(out, 1)

    def turn(self, who, a, g):
        p = self.p
        kfi, nfi = p.dt / (p.gammaTheta * p.alpha), p.varTheta * math.sqrt(p.freeze_temp / p.alpha)
        self.s[who, 3] += kfi * a[who, 0] + nfi * g[:, 0]
        self.s[who, 5] += kfi * a[who, 2] + nfi * g[:, 1]
        self.s[who, 4] += p.dt / p.gammaTheta * a[who, 1] + p.varTheta * g[:, 2]

    def step(self, k):
        p = self.p
        if k % p.ljpairsupdatefreq == 0:
            self.rebuild()
        f, a = self.forces()
        moving = (~self.extra & ~self.fixed).nonzero()[:, 0]
        if not p.hdi_on:
            gx, ga = self.normals(0, moving), self.normals(1, moving)
            self.s[moving, :3] += p.dt / p.gammaR * f[moving] + p.varR * gx[:, :3]
            self.turn(moving, a, ga)
            return
        every = torch.arange(self.nb, device=self.d)
        R = self.normals(0, every)[:, :3] * math.sqrt(2.0 * KB * p.Temp * p.gammaR / p.dt)
        if k % p.tea_epsilon_freq == 0:
            self.coefficients()
        move = f + self.C * R
        for t, i0, i1, act, cii, crr, u in self.tensors():
            j = act
            g = f[j][None] + self.beta_t[t] * self.C[i0:i1][:, None, :] * R[j][None]
            move[i0:i1] += (cii[:, :, None] * g + (crr * (u * g).sum(2))[:, :, None] * u).sum(1)
        ga = self.normals(1, every)[moving]
        self.s[moving, :3] += p.dt / p.gammaR * move[moving]
        self.turn(moving, a, ga)

    def tensors(self):
        """Blocks of rows of each trajectory's mobility tensor T = cii I + crr u u^T (zero where j is i)."""
        aa = self.p.tea_a
        for t in range(self.nt):
            b0, b1 = self.off[t], self.off[t + 1]
            act = torch.arange(b0, b1, device=self.d)
            act = act[~self.extra[b0:b1]]
            rows = max(32, 4_000_000 // (b1 - b0))
            for i0 in range(b0, b1, rows):
                i1 = min(b1, i0 + rows)
                u = self.s[act, :3][None] - self.s[i0:i1, None, :3]
                r = u.norm(dim=2)
                me = act[None] == torch.arange(i0, i1, device=self.d)[:, None]
                r = torch.where(me, 1.0, r)
                u = u / r[:, :, None]
                ra = r / aa
                far = ra > 2.0
                cii = torch.where(far, 0.75 / ra * (1.0 + 2.0 / (3.0 * ra * ra)), 1.0 - 9.0 * ra / 32.0)
                crr = torch.where(far, 0.75 / ra * (1.0 - 2.0 / (ra * ra)), 3.0 * ra / 32.0)
                yield t, i0, i1, act, torch.where(me, 0.0, cii), torch.where(me, 0.0, crr), u

    def coefficients(self):
        ci = torch.zeros(self.nb, 3, dtype=torch.float64, device=self.d)
        eps = torch.zeros(self.nt, dtype=torch.float64, device=self.d)
        for t, i0, i1, act, cii, crr, u in self.tensors():
            on = ~self.extra[i0:i1]
            ci[i0:i1] = (cii[:, :, None] ** 2 + ((2.0 * cii + crr) * crr)[:, :, None] * u * u).sum(1) * on[:, None]
            eps[t] += ((3.0 * cii + crr * u.sum(2) ** 2).sum(1) * on).sum()
        n = torch.zeros(self.nt, dtype=torch.float64, device=self.d).index_add_(0, self.traj, (~self.extra).double())
        e = (eps / (3.0 * n * (3.0 * n - 3.0))).clamp(max=1.0)
        a = (3.0 * n - 1.0) * e * e - (3.0 * n - 2.0) * e
        self.beta_t = torch.where(a.abs() < 1e-7, 0.5, (1.0 - torch.sqrt(1.0 - a)) / a)
        self.C = 1.0 / torch.sqrt(1.0 + self.beta_t[self.traj][:, None] ** 2 * ci)

    def descriptors(self):
        X = torch.zeros(self.nb, 32, dtype=torch.float64, device=self.d)
        for t in range(self.nt):
            b0, b1 = self.off[t], self.off[t + 1]
            act = torch.arange(b0, b1, device=self.d)
            act = act[~self.extra[b0:b1]]
            centre = self.s[act, :3].mean(0)
            for i0 in range(b0, b1, 1024):
                i1 = min(b1, i0 + 1024)
                u = self.s[act, :3][None] - self.s[i0:i1, None, :3]
                r = u.norm(dim=2)
                me = act[None] == torch.arange(i0, i1, device=self.d)[:, None]
                q = torch.where(me, 0.0, 1.0 / torch.where(me, 1.0, r))
                u = u * q[:, :, None]
                for k, (lo, hi) in enumerate(((0.0, 5.0), (5.0, 10.0), (10.0, 20.0))):
                    m = (~me & (r >= lo) & (r < hi)).double()
                    w = m * q
                    v = [m, w, w * q, w * q * q, w * u[:, :, 0] ** 2, w * u[:, :, 1] ** 2, w * u[:, :, 2] ** 2,
                         w * u[:, :, 0] * u[:, :, 1], w * u[:, :, 0] * u[:, :, 2], w * u[:, :, 1] * u[:, :, 2]]
                    X[i0:i1, 10 * k:10 * k + 10] = torch.stack([c.sum(1) for c in v], 1)
            X[b0:b1, 30] = math.log(max(len(act), 1))
            X[b0:b1, 31] = (self.s[b0:b1, :3] - centre).norm(dim=1) * 0.01
        X[self.extra] = 0.0
        return X

    def state(self):
        return torch.cat([self.s, torch.zeros(self.nb, 1, dtype=torch.float64, device=self.d)], 1)


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    n = 13 * case["pf"] + case["free"]
    if kind == "learned":
        return None     # the approximation itself has no 64-bit value but exact TEA's, which takes minutes
    if kind == "tea" and n * n * case["ntraj"] * steps > 2.1e10:
        steps_ok = False    # over 20 seconds of 64-bit pairs
    else:
        steps_ok = steps * max(1.0, n * case["ntraj"] / 2e5) < 3000
    if not steps_ok:
        return None
    b, streams, lists = _system(case, seed)
    R = _Ref(b, streams, lists)
    if kind == "frames":
        R.rebuild()
        U = R.energies()
        f, a = R.forces()
        return dict(forces=torch.cat([f, a[:, [0]], a[:, [1]], a[:, [2]], torch.zeros_like(a[:, [0]])], 1), energies=U,
                    totals=R.totals(U))
    if kind == "fit":
        X = R.descriptors()
        R.coefficients()
        T = torch.cat([R.C, R.beta_t[R.traj][:, None]], 1)
        params, norm = (torch.from_numpy(v.astype(np.float64)).to(R.d) for v in _network(seed, X.cpu().numpy(), T.cpu().numpy()))
        m = min(case["samples"], len(X))
        params.requires_grad_(True)
        at, W = 0, []
        for shape in ((128, 32), (128, 128), (128, 128), (4, 128), (128,), (128,), (128,), (4,)):
            k = math.prod(shape)
            W.append(params[at:at + k].reshape(shape))
            at += k
        h = (X[:m] - norm[:32]) * norm[32:64]
        for k in range(3):
            h = torch.nn.functional.silu(h @ W[k].T + W[4 + k])
        y = h @ W[3].T + W[7]
        loss = ((y - (T[:m] - norm[64:68]) / norm[68:72]) ** 2).mean()
        loss.backward()
        return dict(X=X, T=T, loss=loss.item(), grad=params.grad)
    for k in range(steps):
        R.step(k)
    if kind == "static":
        return dict(totals=R.totals(R.energies()), length=None, state=R.state())
    return dict(state=R.state())
