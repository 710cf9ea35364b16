"""Performance cases: what a program built on this package asks of it, over the range of sizes it is used at.

Every case goes through a public entry point with the arrays that such a program holds: the fine-scale
kick (PM3 + PP) on device arrays and on the host arrays of a Fortran driver, the drift with its buffer
rebuild, and the learned shell's kick and training.  Inputs are made on the GPU from a seed, in the
particle layout of ``cube2_b200.layout``.  ``exact`` restates every path in 64 bits with torch alone.
"""
import copy
import math

import numpy as np
import torch

from cube2_b200 import learned
from cube2_b200.drift import DeviceImage
from cube2_b200.kick import CUBE_PM3_PERIODIC, CUBE_PM3_SUBTILE, CUBE_PM3_TILE_PERIODIC, FineKick, green_table
from cube2_b200.layout import RATIO_SF, Image, Layout, apm3_table, classify_subtiles, ixyz3_table

DEV = "cuda"
APP = 0.1                                   # PP softening, fine cells
RCS = 4                                     # fine cells per coarse cell
A_MID = float(np.float32(6 * np.pi))        # with dt = 1 the velocity change is the force
KICK = float(np.float32(np.float32(A_MID) / np.float32(6.0))) / math.pi
MODES = {"periodic": CUBE_PM3_PERIODIC, "tiles": CUBE_PM3_TILE_PERIODIC, "subtile": CUBE_PM3_SUBTILE}
F64 = torch.float64


def listed():
    return [
        # one small periodic box of a time loop or of a parameter study: launches and latency count
        {"name": "box32", "do": "kick", "geometry": "periodic", "arrays": "device", "ng": 32, "nnt": 1, "nns": 1,
         "field": "zeldovich", "sigma": 0.0, "apm3f": 4.0},
        # the 64^3 Zel'dovich box: the smallest simulation of the workloads
        {"name": "zeldovich64", "do": "kick", "geometry": "periodic", "arrays": "device", "ng": 64, "nnt": 1, "nns": 2,
         "field": "zeldovich", "sigma": 0.0, "apm3f": 4.0},
        # a box of ragged size (15 coarse cells a tile, a 240^3 mesh), moderately clustered
        {"name": "ragged120", "do": "kick", "geometry": "periodic", "arrays": "device", "ng": 120, "nnt": 2, "nns": 5,
         "field": "lognormal", "sigma": 1.0, "apm3f": 4.0},
        # the headline workload: 16.8 M clustered particles, resident on the device
        {"name": "clustered256", "do": "kick", "geometry": "periodic", "arrays": "device", "ng": 256, "nnt": 2,
         "nns": 2, "field": "lognormal", "sigma": 1.5, "apm3f": 4.0},
        # the largest time loop: 134 M particles on a 1024^3 mesh
        {"name": "loop512", "do": "kick", "geometry": "periodic", "arrays": "device", "ng": 512, "nnt": 2, "nns": 2,
         "field": "zeldovich", "sigma": 0.0, "apm3f": 4.0},
        # a batch of 64 independent uneven boxes in one call
        {"name": "batch64", "do": "kick", "geometry": "tiles", "arrays": "device", "ng": 128, "nnt": 4, "nns": 2,
         "field": "boxes", "sigma": 1.0, "apm3f": 4.0},
        # the reference driver's own geometry and arrays: buffered subtile meshes of mixed levels, host memory
        {"name": "driver128", "do": "kick", "geometry": "subtile", "arrays": "host", "ng": 128, "nnt": 2, "nns": 2,
         "field": "lognormal", "sigma": 1.5, "apm3f": 3.5},
        # the headline workload from (pinned) host arrays and back, as a driver without device memory calls it
        {"name": "host256", "do": "kick", "geometry": "periodic", "arrays": "host", "ng": 256, "nnt": 2, "nns": 2,
         "field": "lognormal", "sigma": 1.5, "apm3f": 4.0},
        # the other half of a time step: drift, buffer rebuild and buffer velocities of 16.8 M particles
        {"name": "drift256", "do": "drift", "ng": 256, "nnt": 2, "field": "zeldovich", "sigma": 0.0},
        # inference of the learned shell on every particle of a 7 M particle box
        {"name": "shell192", "do": "shell", "ng": 192, "nnt": 2, "field": "lognormal", "sigma": 1.0},
        # training of the shell: a run of Adam steps on random batches
        {"name": "train8192", "do": "train", "batch": 8192, "steps": 16, "rows": 262144},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi, tiles=(1, 2, 3)):  # a box of nnt tiles of nt coarse cells a side, ng fine cells within [lo, hi]
        nnt = rng.choice(tiles)
        nt = max(3, min(hi // (RCS * nnt), log_int(lo, hi) // (RCS * nnt)))
        return {"ng": RCS * nnt * nt, "nnt": nnt, "nns": rng.choice([s for s in (1, 2, 3, 4, 5) if nt % s == 0])}

    def field():
        return rng.choice([{"field": "zeldovich", "sigma": 0.0},
                           {"field": "lognormal", "sigma": round(rng.uniform(0.5, 1.5), 2)}])

    do = rng.choice(["kick", "kick", "kick", "tiles", "subtile", "host", "drift", "shell", "train"])
    if do == "kick":
        return {"do": "kick", "geometry": "periodic", "arrays": "device", **box(24, 288), **field(),
                "apm3f": rng.choice([4.0, 4.0, 3.5, 2.0])}
    if do == "tiles":
        side, nnt = rng.choice([16, 20, 24, 32, 36, 40]), rng.choice([2, 3, 4])
        return {"do": "kick", "geometry": "tiles", "arrays": "device", "ng": side * nnt, "nnt": nnt, "nns": 1,
                "field": "boxes", "sigma": round(rng.uniform(0.3, 1.0), 2), "apm3f": 4.0}
    if do == "subtile":
        return {"do": "kick", "geometry": "subtile", "arrays": rng.choice(["host", "device"]),
                **box(48, 144, (1, 2)), **field(), "apm3f": 3.5}
    if do == "host":
        return {"do": "kick", "geometry": "periodic", "arrays": "host", **box(48, 192), **field(), "apm3f": 4.0}
    if do == "drift":
        b = box(32, 256)
        return {"do": "drift", "ng": b["ng"], "nnt": b["nnt"], **field()}
    if do == "shell":
        b = box(32, 160)
        return {"do": "shell", "ng": b["ng"], "nnt": b["nnt"], **field()}
    return {"do": "train", "batch": 16 * log_int(32, 512), "steps": rng.choice([4, 8, 16]), "rows": 131072}


# ---- inputs, on the GPU ----------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _wave(n):
    k1 = torch.fft.fftfreq(n, d=1.0 / n, device=DEV)
    kr = torch.fft.rfftfreq(n, d=1.0 / n, device=DEV)
    return k1[:, None, None], k1[None, :, None], kr[None, None, :]


def _gaussian_k(n, gen):
    """Transform of a real Gaussian field on n^3 with P(k) ~ k^-2 (not normalised)."""
    wk = torch.fft.rfftn(torch.randn((n, n, n), generator=gen, device=DEV))
    kz, ky, kx = _wave(n)
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    wk *= k2 ** -0.5
    wk[0, 0, 0] = 0
    return wk, k2


def _zeldovich(m, side, gen, rms=0.5):
    """An m^3 lattice in a box of `side` fine cells, displaced by its Zel'dovich field: positions, displacements."""
    wk, k2 = _gaussian_k(m, gen)
    kz, ky, kx = _wave(m)
    psi = torch.stack([torch.fft.irfftn(1j * kc * wk / k2, s=(m, m, m)).reshape(-1) for kc in (kx, ky, kz)], -1)
    psi *= rms / max(float((psi * psi).sum(-1).mean().sqrt()), 1e-30)
    g = (torch.arange(m, device=DEV, dtype=F64) + 0.5) * (side / m)
    q = torch.stack(torch.meshgrid(g, g, g, indexing="ij")[::-1], -1).reshape(-1, 3)
    return torch.remainder(q + psi.double(), side), psi


def _lognormal(n, sigma, gen):
    """A Poisson sample (one particle a cell on average) of a lognormal density: positions, velocities."""
    wk, _ = _gaussian_k(n, gen)
    g = torch.fft.irfftn(wk, s=(n, n, n))
    rho = torch.exp(g * (sigma / g.std()))
    counts = torch.poisson(rho * (n ** 3 / rho.sum()), generator=gen).reshape(-1).long()
    cell = torch.repeat_interleave(torch.arange(n ** 3, device=DEV), counts)
    pos = torch.stack([cell % n, (cell // n) % n, cell // (n * n)], -1).double()
    pos += torch.rand(pos.shape, generator=gen, device=DEV, dtype=F64)
    return torch.remainder(pos, n), 0.05 * torch.randn(pos.shape, generator=gen, device=DEV)


def _boxes(side, nnt, sigma, gen):
    """nnt^3 independent boxes of uneven particle counts, box t at tile t of one image."""
    rng = np.random.default_rng(3000)
    cnt = np.clip(side ** 3 * np.exp(sigma * rng.standard_normal(nnt ** 3)), side ** 3 / 16, side ** 3 * 6)
    ps, vs = [], []
    for t, m in enumerate(np.maximum(np.rint(np.cbrt(cnt)).astype(int), 2)):
        p, v = _zeldovich(int(m), side, gen)
        ps.append(p + torch.tensor([t % nnt, (t // nnt) % nnt, t // nnt ** 2], device=DEV, dtype=F64) * side)
        vs.append(v)
    return torch.cat(ps), torch.cat(vs)


def _layout(c):
    return Layout(ng=c["ng"], nnt=c["nnt"], nns=c.get("nns", 1), ratio_cs=RCS, ngb=RCS, app=APP)


def _ext_cells(L, per_tile):
    """The coarse cell of the image that every stored (extended) cell holds, and whether it is the tile's own."""
    t, e = torch.arange(L.nnt, device=DEV), torch.arange(L.nte, device=DEV) - L.ncb
    w = torch.remainder(e, L.nt) if per_tile else e
    a = t[:, None] * L.nt + w[None, :]
    a = torch.remainder(a, L.nc)

    def axis(x, d):  # [tile, cell] of axis d (0: z) into [tz, ty, tx, k, j, i]
        shape = [1] * 6
        shape[d], shape[3 + d] = L.nnt, L.nte
        return x.reshape(shape)
    g = ((axis(a, 0) * L.nc + axis(a, 1)) * L.nc + axis(a, 2)).reshape(-1)
    own = ((e >= 0) & (e < L.nt))[None, :].expand(L.nnt, -1)
    return g, (axis(own, 0) & axis(own, 1) & axis(own, 2)).reshape(-1)


def _spread(counts, L, per_tile):
    """rhoc and idx_b_r of an image with `counts` particles in its coarse cells, and for every stored copy
    the place of its particle among the particles sorted by cell."""
    gext, _ = _ext_cells(L, per_tile)
    rhoc = counts[gext]
    starts = torch.cumsum(counts, 0) - counts
    src = torch.repeat_interleave(starts[gext] - (torch.cumsum(rhoc, 0) - rhoc), rhoc)
    src += torch.arange(src.numel(), device=DEV)
    idx = torch.cumsum(rhoc.reshape(-1, L.nte).sum(1), 0)
    return rhoc.int(), idx, src


def _capacity(c, L, n):
    """Rows of a program's particle arrays: the reference allocates its image once, with room for the copies."""
    return int(n * ((L.nt + 2.0) / L.nt) ** 3 * (1.1 + 0.6 * c["sigma"])) // 4096 * 4096 + 8192


def _padded(t, rows):
    out = torch.zeros((rows, *t.shape[1:]), dtype=t.dtype, device=DEV)
    out[:t.shape[0]] = t
    return out


def _image(c, seed):
    """rhoc, idx_b_r, xp, vp, particle number (arrays with room to spare) and number of the stored copies."""
    L, gen = _layout(c), _gen(seed)
    if c["field"] == "zeldovich":
        pos, vel = _zeldovich(L.ng, L.ng, gen)
    elif c["field"] == "lognormal":
        pos, vel = _lognormal(L.ng, c["sigma"], gen)
    else:
        pos, vel = _boxes(L.ng // L.nnt, L.nnt, c["sigma"], gen)
    u = torch.floor(pos * (65536.0 / RCS)).long().clamp_(0, L.nc * 65536 - 1)  # fixed point, 16 bits in the cell
    del pos
    cell = u >> 16
    gcell = (cell[:, 2] * L.nc + cell[:, 1]) * L.nc + cell[:, 0]
    del cell
    u &= 65535
    xp = torch.where(u >= 32768, u - 65536, u).short()
    del u
    order = torch.argsort(gcell, stable=True)
    rhoc, idx, src = _spread(torch.bincount(gcell, minlength=L.nc ** 3), L, c.get("geometry") == "tiles")
    pid = order[src]
    del order, src, gcell
    rows = _capacity(c, L, vel.shape[0] if c["field"] == "boxes" else L.ng ** 3)
    if pid.numel() > rows:
        raise ValueError("more stored copies than the image has room for")
    return rhoc, idx, _padded(xp[pid], rows), _padded(vel.float()[pid], rows), _padded(pid, rows), pid.numel()


_GREENS = {}  # a driver tabulates its Green functions once


def _greens(L, levels, apm3f):
    for lev in levels:
        r = int(RATIO_SF[lev - 1])
        if (lev, L.ntt, apm3f) not in _GREENS:
            _GREENS[lev, L.ntt, apm3f] = green_table((L.ntt + 2) * RCS * r, apm3f, 3.5 * r, 1.0 / r)
    return {lev: _GREENS[lev, L.ntt, apm3f] for lev in levels}


def _pinned(t, shape):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy().reshape(shape)


def prepare(case, seed):
    c = dict(case)
    if c["do"] == "train":
        gen = _gen(seed)
        X = torch.randn((c["rows"], learned.K_PAD), generator=gen, device=DEV)
        X[:, learned.K_IN:] = 0.0
        mix = torch.randn((learned.K_IN, 3), generator=gen, device=DEV) / 8.0
        T = torch.tanh(X[:, :learned.K_IN] @ mix) + 0.3 * torch.randn((c["rows"], 3), generator=gen, device=DEV)
        rows = torch.randint(0, c["rows"], (c["steps"], c["batch"]), generator=gen, device=DEV, dtype=torch.int32)
        return {"case": c, "X": X.bfloat16(), "T": T.contiguous(), "rows": rows,
                "net": learned.ShellNet(batch_cap=c["batch"], seed=seed), "loss": torch.zeros(1, device=DEV)}
    L = _layout(c)
    rhoc, idx, xp, vp, pid, n = _image(c, seed)
    s = {"case": c, "n": n}
    if c["do"] == "drift":
        tiny = Image(L, np.zeros((0, 3), np.int16), np.zeros((0, 3), np.float32), np.zeros(1, np.int32),
                     np.zeros(1, np.int64), np.zeros(0, np.int64), np.zeros(0, bool), n_particles=0)
        di = DeviceImage(tiny, DEV)
        di.rhoc, di.idx, di.xp, di.vp, di.pid = rhoc, idx, xp, vp, pid
        di.n_used, di.cap, di.n_physical = n, xp.shape[0], int(pid.max()) + 1
        di._alloc_spare(di.cap)  # the time loop's second set of arrays
        for k in ("xp", "vp", "pid"):
            di._spare[k].zero_()
        return {**s, "di": di, "fk": FineKick(L), "vz": float(vp[:, 2].abs().max())}
    if c["do"] == "shell":
        return {**s, "rhoc": rhoc, "idx": idx, "xp": xp, "vp": vp, "fk": FineKick(L),
                "net": learned.ShellNet(seed=seed, batch_cap=16)}
    s["fk"] = FineKick(L, pm3_mode=MODES[c["geometry"]], apm3f=c["apm3f"])
    shape = (L.nnt,) * 3 + (L.nte,) * 3
    if c["geometry"] == "subtile":
        ires, isort = classify_subtiles(rhoc.cpu().numpy().reshape(shape), L)
        s["greens"] = _greens(L, sorted(set(ires.tolist())), c["apm3f"])
    else:
        ires, isort = np.full(L.ns3, 2, np.int32), np.arange(1, L.ns3 + 1, dtype=np.int32)
        s["greens"] = None
    s["tables"] = (isort, ires, ixyz3_table(L), apm3_table(c["apm3f"]), RATIO_SF.copy())
    if c["arrays"] == "host":
        s["img"] = Image(L, _pinned(xp, xp.shape), _pinned(vp, vp.shape), _pinned(rhoc, shape), _pinned(idx, shape[:5]),
                         np.zeros(0, np.int64), np.zeros(0, bool), n_particles=0)
    else:
        s.update(rhoc=rhoc, idx=idx, xp=xp, vp=vp, out=torch.zeros(8, device=DEV))
    return s


# ---- one pass ---------------------------------------------------------------------------------------


def run(s):
    c = s["case"]
    if c["do"] == "train":
        for k in range(c["steps"]):
            s["net"].train_step(s["X"], s["T"], s["rows"][k], c["batch"], 1e-3, s["loss"])
        return {"params": s["net"].params(), "loss": s["loss"]}
    s["fk"].configure()
    if c["do"] == "drift":
        di = copy.copy(s["di"])  # the drift swaps the two sets of arrays: the next pass starts from the same image
        di.drift(0.1, s["vz"])
        di.buffer_v()
        return {"rhoc": di.rhoc, "idx": di.idx, "xp": di.xp, "vp": di.vp, "pid": di.pid}
    if c["do"] == "shell":
        s["net"].kick(s["rhoc"], s["idx"], s["xp"], s["n"], s["vp"], 1.0, A_MID, 1.0)
        return {"vp": s["vp"]}
    if c["arrays"] == "host":
        vp, out = s["fk"].kick_fine(s["img"], *s["tables"], 1.0, A_MID, 1.0, greens=s["greens"], vp=s["img"].vp)
        return {"vp": vp, "out": out}
    s["fk"].kick_fine_device(s["rhoc"], s["idx"], s["xp"], s["n"], s["vp"], s["out"], *s["tables"], 1.0, A_MID, 1.0,
                             greens=s["greens"])
    return {"vp": s["vp"], "out": s["out"][:5]}


def work(case):
    c = case
    if c["do"] == "train":
        # the rows of X and T that the batches name, the parameters and Adam's two moments; forward and two
        # backward products of the four layers
        per = 2 * (67 * 128 + 2 * 128 * 128 + 128 * 3)
        return {"bytes": c["steps"] * (c["batch"] * (160.0 + 12 + 4) + 43779 * 24.0),
                "flops": 3.0 * per * c["batch"] * c["steps"]}
    n = float(c["ng"]) ** 3
    nt = c["ng"] // RCS // c["nnt"]
    stored = n * ((nt + 2.0) / nt) ** 3
    if c["do"] == "drift":
        return {"bytes": 2.0 * 26 * stored, "flops": 30.0 * n}
    if c["do"] == "shell":
        return {"bytes": 6.0 * n + 24.0 * n + 8.0 * n,
                "flops": 2.0 * n * (67 * 128 + 2 * 128 * 128 + 128 * 3) + 100.0 * n}
    # the pair forces (38 operations each; the neighbours within the PP range of a uniform box, times the
    # excess of a lognormal one), the TSC sums of deposit and gather, the transforms of the mesh
    rc = c["apm3f"] / 2.0
    mesh = 8.0 * n
    near = 4.18879 * rc ** 3
    if c["field"] == "lognormal":
        near *= math.exp(0.33 * c["sigma"] ** 2)
    elif c["field"] == "boxes":  # uneven boxes: the mean count and the mean of its square
        near *= math.exp(1.2 * c["sigma"] ** 2)
        n, stored = n * math.exp(0.5 * c["sigma"] ** 2), stored * math.exp(0.5 * c["sigma"] ** 2)
    return {"bytes": 6.0 * stored + 24.0 * n,
            "flops": 38.0 * near * n + 27 * 10.0 * n + 5.0 * mesh * math.log2(mesh) + 15.0 * mesh}


def tolerance(case):
    # about four times what each path shows against `exact`: the kicks 0.3e-6 to 4.1e-6 (32-bit sums of forces
    # that partly cancel), the shell 5.5e-3, a few Adam steps 1e-3 (BF16 operands)
    if case["do"] == "drift":
        return "exact"
    if case["do"] == "train":
        return {"rel": 4e-3, "max": 0.1}
    if case["do"] == "shell":
        return {"rel": 2e-2, "max": 0.2}
    return {"rel": 2e-5, "max": 5e-4}


# ---- the same in 64 bits ------------------------------------------------------------------------------


def _decode(rhoc, xp, L, per_tile):
    """Of every tile's own copies: their places among the stored ones, the box and the fine position in it."""
    gext, own = _ext_cells(L, per_tile)
    cell = torch.repeat_interleave(torch.arange(rhoc.numel(), device=DEV), rhoc.long())
    I = torch.nonzero(own[cell]).reshape(-1)
    g = gext[cell[I]]
    gc = torch.stack([g % L.nc, (g // L.nc) % L.nc, g // (L.nc * L.nc)], -1)
    del cell
    pos = (gc.double() + ((xp[I].long() & 65535).double() + 0.5) / 65536.0) * RCS
    if not per_tile:
        return I, torch.zeros_like(g), pos
    t = gc // L.nt
    return I, (t[:, 2] * L.nnt + t[:, 1]) * L.nnt + t[:, 0], pos - (t * (L.nt * RCS)).double()


def _tsc(m):
    f = torch.floor(m)
    l = m - f
    w0, w2 = 0.5 * (1 - l) ** 2, 0.5 * l ** 2
    return f.long(), (w0, 1 - w0 - w2, w2)


def _points(m, n, keep_all):
    """The 27 mesh points of each particle, flat (-1: outside a mesh that does not wrap), and their weights."""
    i, w = _tsc(m)
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                x, y, z = i[:, 0] + dx - 1, i[:, 1] + dy - 1, i[:, 2] + dz - 1
                ok = None
                if not keep_all:
                    ok = (x >= 0) & (x < n) & (y >= 0) & (y < n) & (z >= 0) & (z < n)
                at = ((z % n) * n + y % n) * n + x % n
                wt = w[dx][:, 0] * w[dy][:, 1] * w[dz][:, 2]
                yield at, wt if ok is None else wt * ok


def _green64(n, soft, rng_, gs):
    """The Green function of the mesh on its half spectrum [kz][ky][kx] (five alias terms a side)."""
    h = n // 2
    k1 = 2 * math.pi * float(np.float32(1.0) / np.float32(n)) * torch.arange(h + 1, device=DEV, dtype=F64)
    al, c215 = float(np.float32(4.0) / np.float32(3.0)), float(np.float32(2.0) / np.float32(15.0))
    D1 = al * torch.sin(k1) + (1 - al) * torch.sin(2 * k1) / 2
    s1 = torch.sin(k1 / 2) ** 2
    u1 = 1 - s1 + c215 * s1 * s1

    def ax(v, d):
        return v.reshape([-1 if q == d else 1 for q in (2, 1, 0)])

    def soft2(y):
        return (12.0 / y ** 4 * (2 - 2 * torch.cos(y) - y * torch.sin(y))) ** 2
    num = torch.zeros((h + 1,) * 3, device=DEV, dtype=F64)
    for a in range(-2, 3):
        for b in range(-2, 3):
            for c in range(-2, 3):
                kn = [k1 + 2 * math.pi * q for q in (a, b, c)]
                U = [torch.where(k == 0, torch.ones_like(k), torch.sin(k / 2) / (k / 2)) ** 6 for k in kn]
                k2 = ax(kn[0] ** 2, 0) + ax(kn[1] ** 2, 1) + ax(kn[2] ** 2, 2)
                km = torch.sqrt(k2)
                f = soft2(soft * km / 2)
                if rng_:
                    f = f - soft2(rng_ * km / 2)
                dot = ax(D1 * kn[0], 0) + ax(D1 * kn[1], 1) + ax(D1 * kn[2], 2)
                num += ax(U[0], 0) * ax(U[1], 1) * ax(U[2], 2) * dot * f / k2
    den = ax(D1 ** 2, 0) + ax(D1 ** 2, 1) + ax(D1 ** 2, 2)
    G = 4 * math.pi * num / den / (ax(u1, 0) * ax(u1, 1) * ax(u1, 2)) ** 2 / float(np.float32(gs)) ** 2
    G[::h, ::h, ::h] = 0.0
    m = torch.arange(n, device=DEV)
    m = torch.minimum(m, n - m)
    return G[m][:, m]


def _mesh_force(rho, G):
    """Forces [3, ...] on a batch of periodic meshes [b, z, y, x]."""
    n = rho.shape[-1]
    phi = torch.fft.irfftn(torch.fft.rfftn(rho, dim=(1, 2, 3)) * G, s=(n, n, n), dim=(1, 2, 3))
    a = float(np.float32(4.0) / np.float32(3.0))
    w = {-2: (a - 1) / 4, -1: -a / 2, 1: a / 2, 2: (1 - a) / 4}
    return torch.stack([sum(q * torch.roll(phi, -m, dims=3 - d) for m, q in w.items()) for d in range(3)])


def _pm3_periodic(box, pos, nbox, side, apm3f):
    n = 2 * side
    rho = torch.zeros(nbox * n ** 3, device=DEV, dtype=F64)
    for at, w in _points(pos * 2, n, True):
        rho.index_add_(0, box * n ** 3 + at, w)
    F = _mesh_force(rho.reshape(nbox, n, n, n), _green64(n, apm3f, 0.0, 0.5)).reshape(3, -1)
    del rho
    d = torch.zeros_like(pos)
    for at, w in _points(pos * 2, n, True):
        at = at + box * n ** 3
        for q in range(3):
            d[:, q] += F[q][at] * w
    return d, float((F * F).sum(0).max())


def _pm3_subtile(pos, L, ires, apm3f):
    d, f2 = torch.zeros_like(pos), 0.0
    side = L.ntt * RCS
    G = {}
    for (sx, sy, sz, tx, ty, tz), lev in zip(ixyz3_table(L).tolist(), ires.tolist()):
        r = int(RATIO_SF[lev - 1])
        n, b = (side + 2 * RCS) * r, RCS * r
        if r not in G:
            G[r] = _green64(n, apm3f, 3.5 * r, 1.0 / r)
        o = torch.tensor([((t - 1) * L.nns + s - 1) * side for t, s in ((tx, sx), (ty, sy), (tz, sz))], device=DEV,
                         dtype=F64)
        rho = torch.zeros(n ** 3, device=DEV, dtype=F64)
        # the subtile with one coarse cell around it, periodic copies included
        images = [torch.tensor([x, y, z], device=DEV, dtype=F64) * L.ng for x in (-1, 0, 1) for y in (-1, 0, 1)
                  for z in (-1, 0, 1)]
        for im in images:
            rel = pos + (im - o)
            m = rel[((rel >= -RCS) & (rel < side + RCS)).all(1)] * r + b
            if m.numel():
                for at, w in _points(m, n, False):
                    rho.index_add_(0, at, w)
        F = _mesh_force(rho.reshape(1, n, n, n), G[r])
        phys = F[:, 0, b:n - b, b:n - b, b:n - b]
        f2 = max(f2, float((phys * phys).sum(0).max()))
        J = torch.nonzero(((pos >= o) & (pos < o + side)).all(1)).reshape(-1)
        if J.numel():
            F = F.reshape(3, -1)
            for at, w in _points((pos[J] - o) * r + b, n, True):
                for q in range(3):
                    d[J, q] += F[q][at] * w
    return d, f2


def _s2(r, a):
    """The S2 softened force of two unit masses."""
    e = 2 * r / a
    inner = (224 * e - 224 * e ** 3 + 70 * e ** 4 + 48 * e ** 5 - 21 * e ** 6) / (35 * a * a)
    outer = (12 / e ** 2 - 224 + 896 * e - 840 * e ** 2 + 224 * e ** 3 + 70 * e ** 4 - 48 * e ** 5 + 7 * e ** 6) / (35 * a * a)
    return torch.where(e > 2, 1 / (r * r), torch.where(e > 1, outer, inner))


def _pp(box, pos, nbox, side, rc):
    """Pair forces within rc (of each particle) in periodic boxes of `side` fine cells, cells of two fine cells."""
    n = side // 2
    c = (pos * 0.5).long().clamp_(0, n - 1)
    key = ((box * n + c[:, 2]) * n + c[:, 1]) * n + c[:, 0]
    order = torch.argsort(key)
    p, k, r0 = pos[order], key[order], rc[order]
    cnt = torch.bincount(k, minlength=nbox * n ** 3)
    start = torch.cumsum(cnt, 0) - cnt
    x, y, z, b = k % n, (k // n) % n, (k // n ** 2) % n, k // n ** 3
    F = torch.zeros_like(p)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                nb = ((b * n + (z + dz) % n) * n + (y + dy) % n) * n + (x + dx) % n
                m, s = cnt[nb], start[nb]
                cum = torch.cumsum(m, 0)
                total, at = int(cum[-1]), 0
                cuts = torch.searchsorted(cum, torch.arange(0, total, 1 << 25, device=DEV) + (1 << 25)).tolist()
                for end in cuts[:-1] + [k.numel()]:
                    if end <= at:
                        continue
                    mm = m[at:end]
                    i = torch.repeat_interleave(torch.arange(at, end, device=DEV), mm)
                    j = torch.arange(i.numel(), device=DEV) + torch.repeat_interleave(s[at:end] - (torch.cumsum(mm, 0) - mm), mm)
                    d = p[j] - p[i]
                    d -= side * torch.round(d / side)
                    r2 = (d * d).sum(1)
                    ok = torch.nonzero((r2 > 0) & (r2 < r0[i] ** 2)).reshape(-1)
                    i, d = i[ok], d[ok]
                    r = torch.sqrt(r2[ok])
                    f = (_s2(r, float(np.float32(APP))) - _s2(r, r0[i])) / r
                    F.index_add_(0, i, d * f[:, None])
                    at = end
    out = torch.empty_like(F)
    out[order] = F
    return out


def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def _layers(flat):
    """W1, b1 .. W4, b4 of the flat parameters."""
    out, o = [], 0
    for shape in ((128, 80), (128,), (128, 128), (128,), (128, 128), (128,), (3, 128), (3,)):
        k = int(np.prod(shape))
        out.append(flat[o:o + k].reshape(shape))
        o += k
    return out


def _forward(p, X):
    h = X
    for q in range(0, 6, 2):
        h = _gelu(h @ p[q].T + p[q + 1])
    return h @ p[6].T + p[7]


def _exact_train(c, seed):
    s = prepare(c, seed)
    flat = torch.from_numpy(s["net"].params().astype(np.float64)).to(DEV).requires_grad_(True)
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    total = torch.zeros(1, device=DEV, dtype=F64)
    for k in range(c["steps"]):
        rows = s["rows"][k].long()
        loss = ((_forward(_layers(flat), s["X"][rows].double()) - s["T"][rows].double()) ** 2).mean()
        g, = torch.autograd.grad(loss, flat)
        with torch.no_grad():
            total += loss
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            flat -= 1e-3 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
    return {"params": flat.detach(), "loss": total}


def _exact_shell(c, seed):
    s = prepare(c, seed)
    L = _layout(c)
    I, _, pos = _decode(s["rhoc"], s["xp"], L, False)
    n = L.ng
    q = pos - 0.5
    i0, f = torch.floor(q).long(), q - torch.floor(q)
    rho = torch.zeros(n ** 3, device=DEV, dtype=F64)
    for dz in range(2):
        for dy in range(2):
            for dx in range(2):
                w = 1.0
                for a, dd in enumerate((dx, dy, dz)):
                    w = w * (f[:, a] if dd else 1 - f[:, a])
                at = (((i0[:, 2] + dz) % n) * n + (i0[:, 1] + dy) % n) * n + (i0[:, 0] + dx) % n
                rho.index_add_(0, at, w)
    lr = torch.log1p(rho)
    p = _layers(torch.from_numpy(s["net"].params().astype(np.float64)).to(DEV))
    vp = s["vp"].double()
    for a in range(0, I.numel(), 1 << 20):
        i = i0[a:a + (1 << 20)]
        cols = [lr[(((i[:, 2] + dz) % n) * n + (i[:, 1] + dy) % n) * n + (i[:, 0] + dx) % n]
                for dz in range(-1, 3) for dy in range(-1, 3) for dx in range(-1, 3)]
        X = torch.zeros((i.shape[0], 80), device=DEV, dtype=F64)
        X[:, :64] = torch.stack(cols, 1)
        X[:, 64:67] = f[a:a + (1 << 20)]
        vp[I[a:a + (1 << 20)]] += KICK * _forward(p, X)
    return {"vp": vp}


def _exact_drift(c, seed):
    L = _layout(c)
    rhoc, idx, xp, vp, pid, n = _image(c, seed)
    rows, xp, vp, pid = xp.shape[0], xp[:n], vp[:n], pid[:n]
    vz, dt = np.float32(float(vp[:, 2].abs().max())), np.float32(0.1)
    nlayer = 2 * math.ceil(float(np.float32(dt * vz) / np.float32(RCS))) + 2
    n3 = L.nte ** 3
    cell = torch.repeat_interleave(torch.arange(rhoc.numel(), device=DEV), rhoc.long())
    t, e = cell // n3, cell % n3
    ce = torch.stack([e % L.nte, (e // L.nte) % L.nte, e // (L.nte * L.nte)], -1)
    ti = torch.stack([t % L.nnt, (t // L.nnt) % L.nnt, t // (L.nnt * L.nnt)], -1)
    dv = torch.tensor(dt, device=DEV) * vp  # in 32 bits, as the reference's real(4)
    x = (ce - L.ncb).double() + ((xp.long() & 65535).double() + 0.5) / 65536.0 + (dv / 4.0).double()
    stay = ((x > 0) & (x <= L.nt)).all(1)
    g = ti * L.nt + torch.ceil(x).long() - 1
    dest = (g[:, 2] * L.nc + g[:, 1]) * L.nc + g[:, 0]
    K = torch.nonzero(stay).reshape(-1)
    order = K[torch.argsort(dest[K] * nlayer + ce[K, 2] % nlayer, stable=True)]
    q = dv[order].double() / (RCS / 65536.0)
    step = (torch.sign(q) * torch.floor(q.abs() + 0.5)).long()
    new = (xp[order].long() + step) & 65535
    new = torch.where(new >= 32768, new - 65536, new).short()
    rhoc2, idx2, src = _spread(torch.bincount(dest[K], minlength=L.nc ** 3), L, False)
    return {"rhoc": rhoc2, "idx": idx2, "xp": _padded(new[src], rows), "vp": _padded(vp[order][src], rows),
            "pid": _padded(pid[order][src], rows)}


def exact(case, seed):
    c = dict(case)
    if c["do"] == "train":
        return _exact_train(c, seed)
    if c["do"] == "shell":
        return _exact_shell(c, seed)
    if c["do"] == "drift":
        return _exact_drift(c, seed)
    if c["ng"] > 300:
        return None
    L, per_tile = _layout(c), c["geometry"] == "tiles"
    rhoc, idx, xp, vp, _, _ = _image(c, seed)
    I, box, pos = _decode(rhoc, xp, L, per_tile)
    nbox, side = (L.nnt ** 3, L.ng // L.nnt) if per_tile else (1, L.ng)
    apm3 = apm3_table(c["apm3f"]).astype(np.float64)
    if c["geometry"] == "subtile":
        ires, _ = classify_subtiles(rhoc.cpu().numpy().reshape((L.nnt,) * 3 + (L.nte,) * 3), L)
        d, f2 = _pm3_subtile(pos, L, ires, c["apm3f"])
        side_s, m = L.ntt * RCS, L.nnt * L.nns
        loc = torch.zeros(m ** 3, device=DEV, dtype=F64)
        for (sx, sy, sz, tx, ty, tz), lev in zip(ixyz3_table(L).tolist(), ires.tolist()):
            a = [(t - 1) * L.nns + s - 1 for t, s in ((tx, sx), (ty, sy), (tz, sz))]
            loc[(a[2] * m + a[1]) * m + a[0]] = apm3[lev - 1]
        sub = (pos / side_s).long()
        rc = loc[(sub[:, 2] * m + sub[:, 1]) * m + sub[:, 0]]
    else:
        d, f2 = _pm3_periodic(box, pos, nbox, side, c["apm3f"])
        rc = torch.full((pos.shape[0],), float(apm3[1]), device=DEV, dtype=F64)
    a = _pp(box, pos, nbox, side, rc)
    v = vp.double()
    v[I] += KICK * (d + a)
    top = v[I].abs().amax(0).tolist()
    return {"vp": v, "out": torch.tensor([f2, float((a * a).sum(1).max()), *top], device=DEV, dtype=F64)}
