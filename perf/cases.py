"""Measured workloads of the acoustic isotropic operators.

Each case is one call of one operator (nonlinear, Born, extended Born, tomo, WEMVA; forward or
adjoint) on a batch of shots, made the way a user's program makes it: through ``batch.Context`` with
host arrays, or with device-resident traces through ``Context.device_call``. The context (grid,
velocity fields) is the handle that a program keeps; shots, models and data are its inputs.

``exact`` states the same scheme in 64-bit torch: second order in time, tenth order in space, cosine
sponge, linear interpolation between fine and coarse time, and the imaging conditions.
"""
import ctypes as C
import math

import numpy as np
import torch

from acoustic_isotropic_operators_b200.batch import Context, Shot

FAT = 5
STENCIL = (-2.927222222, 1.666666667, -0.238095238, 0.039682539, -0.004960317, 0.000317460)
ALPHA = 0.99
DTS = 0.004


def _case(name, op, nz, nx, shots, nts, sub=4, pad=50, ext=1, axis="time", wavefield="fp32", surface=False, device=False):
    """nz, nx: interior points, sponge included; pad: sponge width; ext: extension length."""
    return {"name": name, "op": op, "nz": nz, "nx": nx, "shots": shots, "nts": nts, "sub": sub, "pad": pad, "ext": ext,
            "axis": axis, "wavefield": wavefield, "surface": surface, "device": device}


def listed():
    return [
        # the smallest calls: one shot on a test-sized grid with a short record
        _case("nl_fwd_small", "nl_fwd", 96, 160, 1, 200, pad=20),
        # modelling one shot (200 x 400 points at 10 m plus sponge, 4 s): what a modelling loop or a
        # served request runs
        _case("nl_fwd_shot", "nl_fwd", 304, 512, 1, 1000),
        # the same shot's adjoint (source estimation, dot-product tests)
        _case("nl_adj_shot", "nl_adj", 304, 512, 1, 1000),
        # modelling on a fine grid (3.3 m: 12 sub-steps), two shots per call
        _case("nl_fwd_fine_grid", "nl_fwd", 560, 1904, 2, 200, sub=12),
        # linearised modelling of a small batch, traces resident on the device
        _case("born_fwd_batch", "born_fwd", 512, 1312, 8, 500, device=True),
        # migration of a full batch (the benchmark's grid and shot count, a shorter record)
        _case("born_adj_batch", "born_adj", 512, 1312, 32, 200, device=True),
        # migration with the stored wavefield in FP16 on a grid of odd size
        _case("born_adj_fp16_odd", "born_adj", 451, 1187, 3, 401, wavefield="fp16"),
        # marine migration: free surface
        _case("born_adj_surface", "born_adj", 462, 1312, 4, 300, surface=True),
        # linearised modelling on a finer grid (5 m: 8 sub-steps), one shot
        _case("born_fwd_fine_grid", "born_fwd", 560, 1904, 1, 250, sub=8),
        # extended migration over 31 time lags, BF16 stored wavefield
        _case("ext_adj_lags_bf16", "ext_adj", 608, 1600, 8, 200, ext=31, wavefield="bf16"),
        # extended linearised modelling over 21 subsurface offsets
        _case("ext_fwd_offsets", "ext_fwd", 512, 1312, 2, 250, ext=21, axis="offset"),
        # tomographic gradient over 41 time lags on the largest grid
        _case("tomo_adj_lags", "tomo_adj", 912, 3104, 1, 200, ext=41),
    ]


PASSES = {"nl_fwd": 1, "nl_adj": 1, "born_fwd": 2, "born_adj": 2, "ext_fwd": 2, "ext_adj": 2, "tomo_fwd": 5, "tomo_adj": 4,
          "wemva_fwd": 4, "wemva_adj": 4}


def draw(rng):
    op = rng.choice(["nl_fwd", "nl_fwd", "nl_adj", "born_fwd", "born_fwd", "born_adj", "born_adj", "ext_fwd", "ext_adj", "tomo_fwd",
                     "tomo_adj", "wemva_fwd", "wemva_adj"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    while True:
        nz, nx, shots, nts = log(64, 1024), log(96, 3104), log(1, 32), log(100, 2000)
        sub = rng.choice([4, 4, 4, 4, 4, 4, 2, 3, 5, 6, 8, 12])
        extended = op.split("_")[0] in ("ext", "tomo", "wemva")
        ext = 2 * rng.randint(1, 20) + 1 if extended else 1
        axis = rng.choice(["time", "time", "time", "offset"]) if extended else "time"
        stored = op not in ("nl_fwd", "nl_adj") and sub == 4 and axis == "time" and op.split("_")[0] in ("born", "ext")
        wavefield = rng.choice(["fp32", "fp32", "bf16", "fp16"]) if stored else "fp32"
        # (the reference's WEMVA has no free surface)
        surface = not op.startswith("wemva") and rng.random() < 0.2
        updates = float(nz) * nx * shots * (nts - 1) * sub * PASSES[op]
        lags = float(nz) * nx * shots * nts * ext
        held = 4.0 * nz * nx * shots * (nts * (0 if op.startswith("nl") else 2) + (ext if op in ("ext_adj", "wemva_fwd") else 1))
        if 2e8 <= updates <= 1.2e10 and lags <= 2.4e10 and held <= 2e10:
            break
    c = _case("", op, nz, nx, shots, nts, sub, rng.choice([10, 20, 25]) if min(nz, nx) < 160 else 50, ext, axis, wavefield,
              surface, rng.random() < 0.5 and not op.startswith("wemva"))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------- inputs
def _step(c):
    """Grid spacing for which the sub-steps hold the Courant number of the 10 m, 4 sub-step grid."""
    return 40.0 / c["sub"]


def _ring(v, fill=0.0):
    return np.pad(v, FAT, constant_values=fill)


def _interfaces(rng, nx, nz, top):
    """20 flat and dipping one-cell interfaces of amplitude U(-0.1, 0.1), the shallow ones closer together."""
    m = np.zeros((nx, nz), np.float32)
    xs = np.arange(nx)
    for k in range(20):
        z0 = top + 4 + (nz - top - 4) * 10.0 ** rng.uniform(-1.6, -0.05)
        dip = 0.0 if k < 10 else math.tan(math.radians(rng.uniform(-15, 15)))
        z = np.round(z0 + dip * (xs - nx / 2)).astype(int)
        ok = (z >= top) & (z < nz)
        m[xs[ok], z[ok]] += rng.uniform(-0.1, 0.1)
    return m


def _inputs(c, seed):
    rng = np.random.default_rng(seed)
    nz, nx, pad, nts, sub, n_ext = c["nz"], c["nx"], c["pad"], c["nts"], c["sub"], c["ext"]
    top = 0 if c["surface"] else pad
    full_nz, full_nx, d = nz + 2 * FAT, nx + 2 * FAT, _step(c)
    # velocity: linear in depth with Gaussian blobs
    z, x = np.arange(nz, dtype=np.float64)[None, :], np.arange(nx, dtype=np.float64)[:, None]
    v = 1500.0 + 2000.0 * np.clip((z - top) / max(1, nz - top - pad), 0, 1) + 0 * x
    for _ in range(8):
        v += rng.choice([-200.0, 200.0]) * np.exp(-((x - rng.uniform(0, nx)) ** 2 + (z - rng.uniform(0, nz)) ** 2) / 200.0)
    v = _ring(v.astype(np.float32), 1500.0)
    dtw = np.float32(DTS) / np.float32(sub)
    v2 = v * v * dtw * dtw
    rs = (2.0 / (v.astype(np.float64) ** 3)).astype(np.float32)
    # acquisition: four grid points per source (on-grid devices: one of them live), and the two rows of
    # points below the receivers
    iz = FAT + top + 2
    xs = np.linspace(pad + 1, nx - pad - 3, c["shots"] + 2)[1:-1].round().astype(int) + FAT
    src = [np.array([i * full_nz + iz, i * full_nz + iz + 1, (i + 1) * full_nz + iz, (i + 1) * full_nz + iz + 1], np.int32) for i in xs]
    cols = np.arange(FAT + pad, FAT + nx - pad)
    rec = np.concatenate([cols * full_nz + iz, cols * full_nz + iz + 1]).astype(np.int32)
    # Ricker wavelets in fine time (Born family: their second derivative), scaled by dtw^2 v^2
    ntw = (nts - 1) * sub + 1
    t = np.arange(ntw) * (DTS / sub)
    sig = np.zeros((c["shots"], 4, ntw), np.float32)
    for s in range(c["shots"]):
        a = (math.pi * 15.0 * rng.uniform(0.9, 1.1)) ** 2
        w = (1 - 2 * a * (t - 0.1) ** 2) * np.exp(-a * (t - 0.1) ** 2)
        if not c["op"].startswith("nl"):
            w = np.gradient(np.gradient(w, DTS / sub), DTS / sub)
        sig[s, 0] = w * v2.reshape(-1)[src[s][0]]
    g = {"c": c, "v2": v2, "rs": rs, "src": src, "rec": rec, "sig": sig, "full": (full_nx, full_nz), "d": d}
    if c["op"] in ("nl_adj", "born_adj", "ext_adj", "tomo_adj", "wemva_fwd", "wemva_adj"):
        # band-limited traces
        f = np.fft.rfftfreq(nts, DTS)
        band = ((f / 15.0) ** 2 * np.exp(-((f / 15.0) ** 2))).astype(np.float32)
        noise = rng.standard_normal((c["shots"], len(rec), nts), dtype=np.float32)
        g["data"] = np.fft.irfft(np.fft.rfft(noise, axis=-1) * band, n=nts, axis=-1).astype(np.float32)
    refl = _interfaces(rng, nx, nz, top)
    refl[:pad] = 0
    refl[nx - pad:] = 0
    h = (n_ext - 1) // 2
    profile = np.exp(-(np.arange(n_ext) - h) ** 2 / 18.0).astype(np.float32)
    extended = lambda: np.stack([_ring(p * refl) for p in profile])  # noqa: E731
    if c["op"] == "born_fwd":
        g["model"] = _ring(refl)
    elif c["op"] in ("ext_fwd",):
        g["model"] = extended()
    elif c["op"] in ("tomo_fwd", "wemva_fwd"):
        dv = sum(rng.choice([-1.0, 1.0]) * np.exp(-((x - rng.uniform(0, nx)) ** 2 + (z - rng.uniform(0, nz)) ** 2) / 1800.0) for _ in range(8))
        g["model"] = _ring((0.05 * 2500.0 * dv).astype(np.float32))
    if c["op"] in ("tomo_fwd", "tomo_adj", "wemva_adj"):
        g["background"] = extended()
    return g


def prepare(case, seed):
    g = _inputs(case, seed)
    nx, nz = g["full"]
    g["ctx"] = Context(nz, nx, case["nts"], DTS, case["sub"], g["d"], g["d"], case["pad"], g["v2"], g["rs"], nExt=case["ext"],
                       alphaCos=ALPHA, wavefield=case["wavefield"], free_surface=int(case["surface"]), extension=case["axis"])
    ns, nr, op = case["shots"], len(g["rec"]), case["op"]
    wemva = op.startswith("wemva")
    if not case["device"]:
        g["shots"] = [Shot(g["src"][s], g["rec"], None if op == "nl_adj" else g["sig"][s], g["data"][s] if "data" in g and not wemva else None,
                           g["data"][s] if wemva else None) for s in range(ns)]
        return g
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    g["dev"] = {k: cuda(g[k]) for k in ("sig", "data", "model", "background") if k in g}
    if op in ("nl_fwd", "born_fwd", "ext_fwd", "tomo_fwd"):
        g["out"] = torch.zeros((ns, nr, case["nts"]), dtype=torch.float32, device="cuda")
    elif op == "nl_adj":
        g["out"] = torch.zeros((ns, 4, (case["nts"] - 1) * case["sub"] + 1), dtype=torch.float32, device="cuda")
    else:
        g["out"] = torch.zeros(((case["ext"],) if op in ("ext_adj", "wemva_fwd") else ()) + (nx, nz), dtype=torch.float32, device="cuda")
    sig, out = g["dev"]["sig"], g["out"]
    data = out if op in ("nl_fwd", "born_fwd", "ext_fwd", "tomo_fwd") else None if wemva else g["dev"]["data"]
    at = lambda a, s: 0 if a is None else a[s].data_ptr()  # noqa: E731
    g["shots"] = [(g["src"][s], g["rec"], at(sig, s), at(data, s), at(g["dev"]["data"] if wemva else None, s), at(out if op == "nl_adj" else None, s))
                  for s in range(ns)]
    torch.cuda.synchronize()
    return g


def run(g):
    op, ctx, shots = g["c"]["op"], g["ctx"], g["shots"]
    if not g["c"]["device"]:
        if op == "nl_fwd":
            return ctx.nonlinear_forward(shots)
        if op == "nl_adj":
            return ctx.nonlinear_adjoint(shots)
        if op == "born_fwd":
            return ctx.born_forward(g["model"], shots)
        if op == "born_adj":
            return ctx.born_adjoint(shots)
        if op == "ext_fwd":
            return ctx.born_ext_forward(g["model"], shots)
        if op == "ext_adj":
            return ctx.born_ext_adjoint(shots)
        if op == "tomo_fwd":
            return ctx.tomo_forward(g["model"], g["background"], shots)
        if op == "tomo_adj":
            return ctx.tomo_adjoint(g["background"], shots)
        if op == "wemva_fwd":
            return ctx.wemva_forward(g["model"], shots)
        return ctx.wemva_adjoint(g["background"], shots)
    p = {k: C.c_void_p(t.data_ptr()) for k, t in g["dev"].items()}
    out, zero = C.c_void_p(g["out"].data_ptr()), C.c_int(0)
    if op == "nl_fwd":
        ctx.device_call("nonlinear_forward", shots=shots)
    elif op == "nl_adj":
        ctx.device_call("nonlinear_adjoint", shots=shots)
    elif op == "born_fwd":
        ctx.device_call("born_forward", p["model"], shots=shots)
    elif op == "born_adj":
        ctx.device_call("born_adjoint", out, zero, shots=shots)
    elif op == "ext_fwd":
        ctx.device_call("born_ext_forward", p["model"], shots=shots)
    elif op == "ext_adj":
        ctx.device_call("born_ext_adjoint", out, zero, shots=shots)
    elif op == "tomo_fwd":
        ctx.device_call("tomo_ext_forward", p["model"], p["background"], shots=shots)
    elif op == "tomo_adj":
        ctx.device_call("tomo_ext_adjoint", out, zero, p["background"], shots=shots)
    elif op == "wemva_fwd":
        ctx.device_call("wemva_ext_forward", p["model"], out, zero, shots=shots)
    else:
        ctx.device_call("wemva_ext_adjoint", out, zero, p["background"], shots=shots)
    return g["out"]


def work(case):
    """Inputs and outputs once; 39 operations per point update (two 11-point lines, the time update, two
    dampings), plus the imaging products of every coarse sample."""
    n, ns, nts, sub, e = float(case["nz"]) * case["nx"], case["shots"], case["nts"], case["sub"], case["ext"]
    op = case["op"]
    nr, ntw = 2 * (case["nx"] - 2 * case["pad"]), (nts - 1) * sub + 1
    b = 4 * n + 4.0 * ns * (nr * nts + 4 * ntw)
    f = 39.0 * n * ns * (nts - 1) * sub * PASSES[op]
    if not op.startswith("nl"):
        b += 4 * n * (2 + (e if e > 1 else 0))
        f += 2.0 * n * ns * nts * ({"tomo_fwd": 2 * e + 2, "wemva_adj": 2 * e + 2, "tomo_adj": 2 * e + 2, "wemva_fwd": 2 * e + 2}.get(op, e))
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the error seen against exact(): FP32 rounding, which grows with the fine steps that
    the waves travel (1e-4 at 2400 steps, 9e-4 at the longest drawn records), plus the stored
    wavefield's (8e-4 in BF16, 1e-4 in FP16). The tomo forward amplifies it: small scattered data."""
    r = 5e-4 * max(1.0, (case["nts"] - 1) * case["sub"] / 2000.0) * (4.0 if case["op"] == "tomo_fwd" else 1.0)
    return {"rel": r + {"fp32": 0.0, "fp16": 4e-4, "bf16": 3e-3}[case["wavefield"]]}


# ------------------------------------------------------------------------- the scheme in 64 bits
class _Scheme:
    def __init__(self, c, g, dev):
        self.c, self.dev = c, dev
        self.nz, self.nx, self.nts, self.sub, self.surface = c["nz"], c["nx"], c["nts"], c["sub"], c["surface"]
        inner = lambda a: self.t(a)[FAT:-FAT, FAT:-FAT].contiguous()  # noqa: E731
        self.v2, self.rs = inner(g["v2"]), inner(g["rs"])
        self.coef = [s / g["d"] ** 2 for s in STENCIL]
        sc = 1.0 / math.sqrt(((self.nts - 1) * self.sub + 1) / self.nts)
        self.hA = [(1 - i / self.sub) * sc for i in range(self.sub + 1)]
        self.hB = [i / self.sub * sc for i in range(self.sub + 1)]
        ix, iz = torch.arange(self.nx, device=dev)[:, None], torch.arange(self.nz, device=dev)[None, :]
        dist = torch.minimum(ix, self.nx - 1 - ix)
        dist = torch.minimum(dist, self.nz - 1 - iz if self.surface else torch.minimum(iz, self.nz - 1 - iz))
        edge = ALPHA + (1 - ALPHA) * torch.cos(math.pi / c["pad"] * (c["pad"] - dist).double())
        self.D = torch.where(dist < c["pad"], edge, torch.ones_like(edge))
        self.B = c["shots"]

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev).double()

    def at(self, pos):
        pos = torch.as_tensor(np.asarray(pos), device=self.dev).long()
        nz = self.nz + 2 * FAT
        return (pos // nz - FAT) * self.nz + pos % nz - FAT

    def start(self):
        shape = (self.B, self.nx + 2 * FAT, self.nz + 2 * FAT)
        self.p = [torch.zeros(shape, dtype=torch.float64, device=self.dev) for _ in range(2)]  # current, old
        self.q = torch.zeros(shape, dtype=torch.float64, device=self.dev)
        self.a, self.b = (torch.empty((self.B, self.nx, self.nz), dtype=torch.float64, device=self.dev) for _ in range(2))

    def advance(self, adjoint, inject):
        """One fine step; inject(n) adds the sources to the undamped new level. Returns the new level."""
        cur, old = self.p
        nx, nz, f = self.nx, self.nz, FAT
        core = lambda u, i=0, j=0: u[:, f + i:f + i + nx, f + j:f + j + nz]  # noqa: E731
        c = cur
        if adjoint:
            core(self.q).copy_(core(cur) * self.v2)
            c = self.q
        elif self.surface:
            c = self.q
            c.copy_(cur)
            c[:, :, f] = 0
            for k in range(1, FAT + 1):
                c[:, :, f - k] = -cur[:, :, f + k]
        lap, tmp = self.a, self.b
        torch.mul(core(c), 2 * self.coef[0], out=lap)
        for k in range(1, 6):
            torch.add(core(c, 0, k), core(c, 0, -k), out=tmp)
            tmp.add_(core(c, k)).add_(core(c, -k))
            lap.add_(tmp, alpha=self.coef[k])
        o = core(old)
        if adjoint:
            if self.surface:  # rows 1-4 drop the terms mirrored at the surface
                for z in range(1, FAT):
                    for k in range(z + 1, 6):
                        lap[:, :, z] -= self.coef[k] * c[:, f:f + nx, f + k - z]
        else:
            lap.mul_(self.v2)
        lap.add_(core(c if not adjoint else cur), alpha=2.0)
        if adjoint and self.surface:
            lap[:, :, 0] = 0
            keep = self.D[:, 0] * o[:, :, 0]
        torch.mul(o, self.D, out=tmp)
        if self.surface and not adjoint:
            tmp[:, :, 0] = 0
        lap.sub_(tmp)
        if adjoint and self.surface:
            lap[:, :, 0] = keep
        inject(lap)
        torch.mul(lap, self.D, out=o)
        self.p = [old, cur]
        return o

    # sparse and dense drives --------------------------------------------------------------
    def forward(self, inject, on_step):
        """inject(n, its, it2), on_step(S, its, it2) over the forward fine steps."""
        self.start()
        for its in range(self.nts - 1):
            for i in range(1, self.sub + 1):
                on_step(self.advance(False, lambda n: inject(n, its, i)), its, i)

    def backward(self, inject, on_step):
        self.start()
        for its in range(self.nts - 2, -1, -1):
            for i in range(self.sub - 1, -1, -1):
                on_step(self.advance(True, lambda n: inject(n, its, i)), its, i)

    def sources(self, g):
        idx = torch.stack([self.at(p) for p in g["src"]])
        sig = self.t(g["sig"])
        return lambda n, its, i: n.reshape(self.B, -1).scatter_add_(1, idx, sig[:, :, its * self.sub + i - 1])

    def data(self, g):
        idx = self.at(g["rec"])
        d = self.t(g["data"]).permute(2, 0, 1).contiguous()
        return lambda n, its, i: n.reshape(self.B, -1).index_add_(1, idx, d[its] * self.hA[i + 1] + d[its + 1] * self.hB[i + 1])

    def record(self, g):
        idx = self.at(g["rec"])
        out = torch.zeros((self.nts, self.B, len(idx)), dtype=torch.float64, device=self.dev)

        def on_step(S, its, i):
            r = S.reshape(self.B, -1)[:, idx]
            out[its] += r * self.hA[i]
            out[its + 1] += r * self.hB[i]
        return out, on_step

    def field(self):
        return torch.zeros((self.nts, self.B, self.nx, self.nz), dtype=torch.float64, device=self.dev)

    def store(self, W):
        def on_step(S, its, i):
            W[its].add_(S, alpha=self.hA[i])
            W[its + 1].add_(S, alpha=self.hB[i])
        return on_step

    def dense_forward(self, ss):
        return lambda n, its, i: n.add_(ss(its), alpha=self.hA[i - 1]).add_(ss(its + 1), alpha=self.hB[i - 1])

    def dense_backward(self, ss):
        return lambda n, its, i: n.add_(ss(its), alpha=self.hA[i + 1]).add_(ss(its + 1), alpha=self.hB[i + 1])

    def cached(self, f):
        """The last two coarse slices that f formed."""
        kept = {}

        def get(t):
            if t not in kept:
                for k in [k for k in kept if abs(k - t) > 1]:
                    del kept[k]
                kept[t] = f(t)
            return kept[t]
        return get

    # extensions ---------------------------------------------------------------------------
    def spread(self, m, F, sign=1):
        """ss(t) = sum_e m_e F: time lags F[t - sign 2 (e - h)], offsets m_s(x - s) F(x - 2 s) v2(x) (sign 1)
        or m_s(x + s) F(x + 2 s) v2(x + 2 s) (sign -1), model points within [h, nx - h)."""
        h, nx = (self.c["ext"] - 1) // 2, self.nx

        def f(t):
            out = torch.zeros_like(F[0])
            for e in range(2 * h + 1):
                s = e - h
                if self.c["axis"] == "time":
                    u = t - sign * 2 * s
                    if 0 <= u < self.nts:
                        out.addcmul_(m[e].expand_as(out), F[u])
                else:
                    lo, hi = max(h, -s if sign > 0 else h, s if sign > 0 else 0), nx - h
                    # model point x, source point x - sign s, output point x + sign s
                    x = torch.arange(lo, hi, device=self.dev)
                    ok = (x - sign * s >= 0) & (x - sign * s < nx) & (x + sign * s >= 0) & (x + sign * s < nx)
                    x = x[ok]
                    w = F[t][:, x - sign * s]
                    if sign < 0:
                        w = w * self.v2[x - sign * s]
                    out[:, x + sign * s] += m[e][x] * w
            if self.c["axis"] == "offset" and sign > 0:
                out *= self.v2
            return out
        return self.cached(f)

    def image(self, img, R, t, F, sign=1):
        """Extended image of sample R of time t: lags R F[t - sign 2 (e - h)]; offsets (R v2)(x + s) F(x - s) (sign 1)
        or R(x - s) F(x + s) v2(x + s) (sign -1)."""
        h, nx = (self.c["ext"] - 1) // 2, self.nx
        for e in range(2 * h + 1):
            s = e - h
            if self.c["axis"] == "time":
                u = t - sign * 2 * s
                if 0 <= u < self.nts:
                    img[e] += (R * F[u]).sum(0)
            elif sign > 0:
                img[e, h:nx - h] += ((R * self.v2)[:, h + s:nx - h + s] * F[t][:, h - s:nx - h - s]).sum(0)
            else:
                img[e, h:nx - h] += (R[:, h - s:nx - h - s] * (F[t] * self.v2)[:, h + s:nx - h + s]).sum(0)

    def samples(self, post, backward):
        """on_step that hands each finished coarse sample (t, R) to post."""
        acc = {}

        def on_step(S, its, i):
            for t, w in ((its, self.hA[i]), (its + 1, self.hB[i])):
                if t not in acc:
                    acc[t] = torch.zeros((self.B, self.nx, self.nz), dtype=torch.float64, device=self.dev)
                acc[t].add_(S, alpha=w)
            if backward and i == 0:
                post(its + 1, acc.pop(its + 1))
                if its == 0:
                    post(0, acc.pop(0))
            if not backward and i == self.sub:
                post(its, acc.pop(its))
                if its == self.nts - 2:
                    post(its + 1, acc.pop(its + 1))
        return on_step


def exact(case, seed):
    with torch.no_grad():
        g = _inputs(case, seed)
        return _exact(case, g, torch.device("cuda" if torch.cuda.is_available() else "cpu"))


def _exact(c, g, dev):
    s, op = _Scheme(c, g, dev), c["op"]
    nx, nz = g["full"]
    traces = lambda d: _as_run(c, d.permute(1, 2, 0))  # noqa: E731
    if op == "nl_fwd":
        out, on_step = s.record(g)
        s.forward(s.sources(g), on_step)
        return traces(out)
    if op == "nl_adj":
        idx = torch.stack([s.at(p) for p in g["src"]])
        out = torch.zeros((s.B, 4, (s.nts - 1) * s.sub + 1), dtype=torch.float64, device=dev)

        def on_step(S, its, i):
            out[:, :, its * s.sub + i] = S.reshape(s.B, -1).gather(1, idx)
        s.backward(s.data(g), on_step)
        return _as_run(c, out)
    inner = lambda a: s.t(a)[..., FAT:-FAT, FAT:-FAT].contiguous()  # noqa: E731
    lag = c["axis"] == "time"
    W = s.field()
    s.forward(s.sources(g), s.store(W))
    scale = s.v2 * s.rs
    ext_scale = scale if lag else s.rs
    if op == "born_fwd":
        dm = inner(g["model"]) * scale
        out, on_step = s.record(g)
        s.forward(s.dense_forward(s.cached(lambda t: W[t] * dm)), on_step)
        return traces(out)
    if op == "ext_fwd":
        out, on_step = s.record(g)
        s.forward(s.dense_forward(s.spread(inner(g["model"]) * ext_scale, W)), on_step)
        return traces(out)
    img = torch.zeros((c["ext"], s.nx, s.nz), dtype=torch.float64, device=dev)
    zero_lag = torch.zeros((s.nx, s.nz), dtype=torch.float64, device=dev)

    def whole(a):
        out = torch.zeros(a.shape[:-2] + (nx, nz), dtype=torch.float64, device=dev)
        out[..., FAT:-FAT, FAT:-FAT] = a
        return out if c["device"] else out.cpu().numpy()

    def correlate(F):
        def post(t, R):
            zero_lag.add_((R * F[t]).sum(0))
        return post
    if op == "born_adj":
        s.backward(s.data(g), s.samples(correlate(W), True))
        return whole(zero_lag * scale)
    if op == "ext_adj":
        s.backward(s.data(g), s.samples(lambda t, R: s.image(img, R, t, W), True))
        return whole(img * ext_scale)
    # tomo and WEMVA work on the second time derivative of the source wavefield
    prev = torch.zeros_like(W[0])
    for t in range(s.nts):
        here = W[t].clone()
        W[t] = (prev - 2 * here + (W[t + 1] if t + 1 < s.nts else 0)) / DTS ** 2
        prev = here
    if op == "tomo_fwd":
        dm, ex = inner(g["model"]) * scale, inner(g["background"]) * ext_scale
        out, on_step = s.record(g)
        W1 = s.field()
        s.forward(s.dense_forward(s.spread(ex, W)), s.store(W1))
        s.forward(s.dense_forward(s.cached(lambda t: W1[t] * dm)), on_step)
        W1.zero_()
        s.forward(s.dense_forward(s.cached(lambda t: W[t] * dm)), s.store(W1))
        s.forward(s.dense_forward(s.spread(ex, W1)), on_step)
        return traces(out)
    R = s.field()
    s.backward(s.data(g), s.store(R))
    if op == "wemva_fwd":
        dm = inner(g["model"]) * scale
        s.forward(s.dense_forward(s.cached(lambda t: W[t] * dm)), s.samples(lambda t, r: s.image(img, r, t, R, -1), False))
        s.backward(s.dense_backward(s.cached(lambda t: R[t] * dm)), s.samples(lambda t, r: s.image(img, r, t, W, 1), True))
        return whole(img * ext_scale)
    ex = inner(g["background"]) * ext_scale
    s.forward(s.dense_forward(s.spread(ex, W)), s.samples(correlate(R), False))
    s.backward(s.dense_backward(s.spread(ex, R, -1)), s.samples(correlate(W), True))
    return whole(zero_lag * scale)


def _as_run(c, out):
    """Traces as run() returns them: one tensor on the device, or a list of host arrays."""
    return out.contiguous() if c["device"] else [o.cpu().numpy() for o in out]
