"""Performance cases of the measurement path, through its public entry points.

Each listed case is a call a user's program makes: one configuration measured
(HYP smearing of all links, operator smearing over several levels, plaquette
after every level, all Wilson loops W(sl1, sl2; t, r; x0)), a batch of
configurations, or a field smeared and handed back.  Kinds:

  stream    the field comes from host memory on every pass (ms10's loop over
            configurations: read, measure)
  resident  the field is on the device (restored from the context's snapshot,
            since a measurement smears the field in place)
  batch     many lattices of two sizes in one Batch
  smear     smearing entry points one by one, the plaquette, and the field
            downloaded (a program that uses the smeared links itself)

Fields are U = exp(i eps sum_a h_a lambda_a) with Gaussian h_a, the synthetic
fields of the workloads, drawn here with torch from the seed; with open
boundary conditions the temporal links of the last slice are zero.
"""
import math

import numpy as np
import torch

from wloop_b200.api import APE, HYP, Batch, Context, WloopParms

HYP2 = (1.0, 1.0, 0.5)


def _case(name, kind, n, bc, precision, eps, nss, t, r, op="ape", proj_iter=4, count=0, n_b=None):
    c = {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "n3": n[3], "bc": bc,
         "precision": precision, "eps": eps, "nss": ",".join(str(s) for s in nss), "t": t, "r": r,
         "op": op, "proj_iter": proj_iter}
    if kind == "batch":  # count lattices n, then count // 4 of the larger size
        c["count"] = count
        c["m0"], c["m1"] = n_b[0], n_b[1]
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: an 8^4 test lattice streamed from the host,
        # where launches and latency count
        _case("stream_8x8x8x8_mixed", "stream", (8, 8, 8, 8), 3, "mixed", 0.3, [0, 5, 5, 5], 4, 4),
        # a small open lattice at the reference's own precision
        _case("stream_24x12x12x12_open_fp64", "stream", (24, 12, 12, 12), 0, "fp64", 0.25,
              [0, 5, 5], 8, 6),
        # the smaller volume of the batch and serving workloads, on its own
        _case("resident_32x16x16x16_mixed", "resident", (32, 16, 16, 16), 3, "mixed", 0.2,
              [0, 5, 5, 5], 8, 8),
        # odd, unequal extents: tiles and row blocks end in the middle
        _case("resident_26x17x15x23_mixed", "resident", (26, 17, 15, 23), 3, "mixed", 0.25,
              [1, 4, 7], 11, 7),
        # spatial HYP as the operator smearing (ms10's other choice)
        _case("resident_32x20x20x20_hyp_fp64", "resident", (32, 20, 20, 20), 3, "fp64", 0.2,
              [1, 3, 3, 3], 10, 8, op="hyp"),
        # an ordinary production lattice, open boundaries, streamed and
        # resident, at both precisions
        _case("stream_48x24x24x24_open_mixed", "stream", (48, 24, 24, 24), 0, "mixed", 0.25,
              [0, 10, 10, 10, 10], 16, 12),
        _case("resident_48x24x24x24_open_fp64", "resident", (48, 24, 24, 24), 0, "fp64", 0.25,
              [0, 10, 10, 10, 10], 16, 12),
        # the headline configuration at both precisions
        _case("resident_64x32x32x32_mixed", "resident", (64, 32, 32, 32), 3, "mixed", 0.2,
              [0, 10, 10, 10, 10, 10], 24, 16),
        _case("resident_64x32x32x32_fp64", "resident", (64, 32, 32, 32), 3, "fp64", 0.2,
              [0, 10, 10, 10, 10, 10], 24, 16),
        # a larger volume with the serving workload's parameters
        _case("resident_72x36x36x36_open_mixed", "resident", (72, 36, 36, 36), 0, "mixed", 0.2,
              [0, 5, 5, 5], 18, 18),
        # throughput runs: many configurations of two volumes together
        _case("batch_12x32x16x16x16_3x48x24x24x24_mixed", "batch", (32, 16, 16, 16), 3, "mixed",
              0.2, [0, 5, 5, 5], 8, 8, count=12, n_b=(48, 24)),
        # smearing on its own, the smeared field read back
        _case("smear_24x12x12x12_fp64", "smear", (24, 12, 12, 12), 3, "fp64", 0.3, [10, 10], 1, 1),
    ]


def _flops(c):
    return work(c)["flops"]


def draw(rng):
    """One more case: sizes over 2^12 .. 2 million sites (log-uniform), any
    extents, 1-6 levels, both boundaries, precisions and operator smearings."""
    cap = max(_flops(c) for c in listed())
    while True:
        kind = rng.choice(["stream"] * 2 + ["resident"] * 5 + ["batch"] * 2 + ["smear"])
        most = {"resident": 2.1e6, "stream": 7e5, "batch": 1.3e5, "smear": 4.2e4}[kind]
        sites = math.exp(rng.uniform(math.log(4096), math.log(most)))
        aspect = rng.uniform(1.0, 2.2)  # time extent over the mean spatial one
        ns = (sites / aspect) ** 0.25
        n = [max(4, round(ns * aspect))] + [max(4, round(ns * rng.uniform(0.85, 1.18)))
                                            for _ in range(3)]
        if rng.random() < 0.5:
            n = [v + (v & 1) for v in n]
        msl = rng.randint(1, 6)
        nss = [rng.choice([0, 0, 1, 2])] + [rng.randint(1, 10) for _ in range(msl - 1)]
        tmax, rmax = n[0] // 2, min(n[1:]) // 2
        t = max(1, round(tmax * rng.uniform(0.4, 1.0)))
        r = max(1, round(rmax * rng.uniform(0.4, 1.0)))
        precision = rng.choice(["mixed", "mixed", "fp64"])
        bc = rng.choice([0, 3])
        eps = round(rng.uniform(0.15, 0.3), 3)
        if kind == "smear":
            c = _case(None, kind, n, bc, precision, eps, [rng.randint(0, 8), rng.randint(1, 8)],
                      1, 1)
        elif kind == "batch":
            c = _case(None, kind, n, bc, precision, eps, nss, t, r, count=rng.choice([4, 8]),
                      n_b=(n[0] + 4, min(n[1:]) + 3))
        else:
            c = _case(None, kind, n, bc, precision, eps, nss, t, r,
                      op="hyp" if rng.random() < 0.25 else "ape")
        if 6.0e7 <= _flops(c) <= 0.9 * cap:
            return c


# --- what a pass needs -------------------------------------------------------
def _nss(c):
    return [int(s) for s in c["nss"].split(",")]


def _parms(c):
    nss = _nss(c)
    return WloopParms(msl=len(nss), nss=nss, mwlt=c["t"], mwlr=c["r"],
                      op_smear=HYP if c["op"] == "hyp" else APE, alpha_action=HYP2, alpha_ape=0.5,
                      alpha_hyp=(0.75, 0.6), proj_iter=c["proj_iter"])


def _lattices(c):
    n = (c["n0"], c["n1"], c["n2"], c["n3"])
    if c["kind"] != "batch":
        return [n]
    m = (c["m0"], c["m1"], c["m1"], c["m1"])
    return [n] * c["count"] + [m] * (c["count"] // 4)


def work(case):
    """Bytes: the field read once, the result written once.  Flops: 198 a 3x3
    complex product, piter-fold projection, the loops as dot products of 18
    numbers per (site, direction, t, r, level pair)."""
    c = case
    nss, pit = _nss(c), c["proj_iter"]
    msl = len(nss)
    proj = 76 + 531 * pit
    nbytes = flops = 0
    link = 144 if c["precision"] == "fp64" or c["kind"] in ("stream", "smear") else 72
    for n in _lattices(c):
        v = n[0] * n[1] * n[2] * n[3]
        hyp = (48 * 828 + 28 * proj) * v
        nbytes += 4 * link * v
        if c["kind"] == "smear":
            flops += hyp + nss[0] * (12 * 828 + 4 * proj) * v
            flops += nss[1] * (12 * 828 + 9 * proj) * v + 2592 * v
            nbytes += 4 * 144 * v
            continue
        sweep = (6 * 828 + 3 * proj) if c["op"] == "ape" else (12 * 828 + 9 * proj)
        flops += hyp + sweep * sum(nss) * v + 2592 * v * (msl if c["kind"] != "batch" else 0)
        flops += 3 * msl * 198 * (c["r"] - 1) * v + 108 * msl * msl * c["t"] * c["r"] * v
        nbytes += 8 * msl * msl * c["t"] * c["r"] * n[0]
    return {"bytes": nbytes, "flops": flops}


# --- fields ------------------------------------------------------------------
def _mm(a, b, dag_a=False, dag_b=False):
    """Products of 3x3 matrices in the first two dimensions."""
    if dag_a:
        a = a.transpose(0, 1).conj()
    if dag_b:
        b = b.transpose(0, 1).conj()
    out = a[:, 0, None] * b[None, 0]
    for k in (1, 2):
        out += a[:, k, None] * b[None, k]
    return out


def _unit(like):
    one = torch.eye(3, dtype=like.dtype, device=like.device)
    return one.reshape((3, 3) + (1,) * (like.dim() - 2))


def _field(n, bc, eps, seed):
    """The four directions, each [3, 3, N0, N1, N2, N3] complex128."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    out = []
    for mu in range(4):
        h = torch.randn((8,) + tuple(n), dtype=torch.float64, device=dev, generator=gen) * eps
        a = torch.zeros((3, 3) + tuple(n), dtype=torch.complex128, device=dev)
        s3 = 1.0 / math.sqrt(3.0)
        a[0, 0] = 1j * (h[2] + s3 * h[7])
        a[1, 1] = 1j * (-h[2] + s3 * h[7])
        a[2, 2] = -2j * s3 * h[7]
        for i, j, p, q in ((0, 1, 0, 1), (0, 2, 3, 4), (1, 2, 5, 6)):
            a[i, j] = torch.complex(h[q], h[p])
            a[j, i] = torch.complex(-h[q], h[p])
        a *= 1.0 / 16.0
        u = _unit(a) + a / 11.0
        for k in range(10, 0, -1):  # Taylor series of exp(a), then squared 4 times
            u = _unit(a) + _mm(a, u) / k
        for _ in range(4):
            u = _mm(u, u)
        if bc == 0 and mu == 0:
            u[:, :, n[0] - 1] = 0.0
        out.append(u)
    return out


def _host(field, pin):
    """su3_dble order (V, 4, 3, 3) in host memory."""
    v = field[0][0, 0].numel()
    dev = torch.empty((v, 4, 3, 3), dtype=torch.complex128, device=field[0].device)
    for mu in range(4):
        dev[:, mu] = field[mu].reshape(3, 3, v).permute(2, 0, 1)
    if not pin or not dev.is_cuda:
        return dev.cpu().numpy()
    host = torch.empty(dev.shape, dtype=dev.dtype, pin_memory=True)
    host.copy_(dev)
    return host.numpy()


def prepare(case, seed):
    c = case
    lats = _lattices(c)
    fields = []
    for i, n in enumerate(lats):
        fields.append(_host(_field(n, c["bc"], c["eps"], 1000 * seed + i), c["kind"] == "stream"))
    if torch.cuda.is_available():
        torch.cuda.empty_cache()
    if c["kind"] == "batch":
        b = Batch([(n, c["bc"], _parms(c)) for n in lats], precision=c["precision"])
        for i, u in enumerate(fields):
            b.upload(i, u)
        b.snapshot()
        return {"case": c, "batch": b}
    ctx = Context(lats[0], bc=c["bc"], precision=c["precision"])
    state = {"case": c, "ctx": ctx, "parms": _parms(c)}
    if c["kind"] == "stream":
        state["u"] = fields[0]
    else:
        ctx.upload(fields[0])
        ctx.snapshot()
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        b = state["batch"]
        b.restore()
        b.run()
        return [b.result(i) for i in range(len(b))]
    ctx = state["ctx"]
    if c["kind"] == "stream":
        ctx.upload(state["u"])
    else:
        ctx.restore()
    if c["kind"] == "smear":
        nss = _nss(c)
        ctx.hyp_links(*HYP2, proj=1, piter=c["proj_iter"])
        if nss[0]:
            ctx.ape_links(0.1, proj=1, piter=c["proj_iter"], nsweeps=nss[0])
        ctx.hyp_spatial_links(0.75, 0.6, proj=1, piter=c["proj_iter"], nsweeps=nss[1])
        return [ctx.average_plaquette(), ctx.download()]
    wl, plaq = ctx.measure(state["parms"], plaq=True)
    return [wl, plaq]


# --- the same in 64 bits -----------------------------------------------------
def _project(u, piter):
    d = (u.real.square() + u.imag.square()).sum((0, 1))
    live = d >= 4.242640687119285 * np.finfo(np.float64).eps
    s = torch.where(live, 1.0 / torch.sqrt(torch.where(live, d, torch.ones_like(d)) / 3.0),
                    torch.ones_like(d))
    u = u * s
    for _ in range(piter):
        x = _mm(u, u, dag_a=True) * -0.5 + 1.5 * _unit(u)
        y = _mm(u, x)
        det = (y[0, 0] * (y[1, 1] * y[2, 2] - y[1, 2] * y[2, 1])
               - y[0, 1] * (y[1, 0] * y[2, 2] - y[1, 2] * y[2, 0])
               + y[0, 2] * (y[1, 0] * y[2, 1] - y[1, 1] * y[2, 0]))
        u = y * torch.complex(torch.ones_like(d), det.imag / -3.0)
    return u


def _up(u, mu):
    return torch.roll(u, -1, 2 + mu)


def _staples(u1, u2, mu, nu):
    """u1(x,nu) u2(x+nu,mu) u1(x+mu,nu)^dag and the one below."""
    side = _up(u1, mu)
    out = _mm(u1, _mm(_up(u2, nu), side, dag_b=True))
    return out + torch.roll(_mm(u1, _mm(u2, side), dag_a=True), 1, 2 + nu)


def _hyp(u, alpha, piter):
    a1, a2, a3 = alpha

    def level1(mu, eta):
        return _project((1 - a3) * u[mu] + a3 / 2 * _staples(u[eta], u[mu], mu, eta), piter)

    bar = {(mu, eta): level1(mu, eta) for mu in range(4) for eta in range(4) if mu != eta}
    til = {}
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            s = 0
            for rho in range(4):
                if rho not in (mu, nu):
                    eta = 6 - mu - nu - rho
                    s = s + _staples(bar[rho, eta], bar[mu, eta], mu, rho)
            til[mu, nu] = _project((1 - a2) * u[mu] + a2 / 4 * s, piter)
    out = []
    for mu in range(4):
        s = 0
        for nu in range(4):
            if nu != mu:
                s = s + _staples(til[nu, mu], til[mu, nu], mu, nu)
        out.append(_project((1 - a1) * u[mu] + a1 / 6 * s, piter))
    return out


def _ape(u, alpha, piter, dirs):
    out = list(u)
    for mu in dirs:
        s = 0
        for nu in dirs:
            if nu != mu:
                s = s + _staples(u[nu], u[mu], mu, nu)
        out[mu] = _project(u[mu] + alpha * s, piter)
    return out


def _hyp_spatial(u, a1, a2, piter):
    bar = {(mu, nu): _project((1 - a2) * u[mu] + a2 / 2 * _staples(u[nu], u[mu], mu, nu), piter)
           for mu in (1, 2, 3) for nu in (1, 2, 3) if mu != nu}
    out = list(u)
    for mu in (1, 2, 3):
        s = 0
        for nu in (1, 2, 3):
            if nu != mu:
                s = s + _staples(bar[nu, mu], bar[mu, nu], mu, nu)
        out[mu] = _project((1 - a1) * u[mu] + a1 / 4 * s, piter)
    return out


def _plaq(u, n, bc):
    """Sum of Re tr over the plaquettes."""
    total = 0.0
    for mu in range(1, 4):
        for nu in range(mu):
            p = _mm(u[mu], _up(u[nu], mu))
            q = _mm(u[nu], _up(u[mu], nu))
            # with open time the plaquettes above the last slice hold its zero
            # temporal links
            total += float((p.real * q.real + p.imag * q.imag).sum())
    return total


def _measure(c, n, seed):
    u = _hyp(_field(n, c["bc"], c["eps"], seed), HYP2, c["proj_iter"])
    nss = _nss(c)
    msl, vs = len(nss), n[1] * n[2] * n[3]
    levels, plaq = [], []
    for sweeps in nss:
        for _ in range(sweeps):
            if c["op"] == "hyp":
                u = _hyp_spatial(u, 0.75, 0.6, c["proj_iter"])
            else:
                u = _ape(u, 0.5, c["proj_iter"], (1, 2, 3))
        levels.append(u[1:])
        plaq.append(_plaq(u, n, c["bc"]))
    wl = torch.zeros((n[0], c["r"], c["t"], msl, msl), dtype=torch.float64, device=u[0].device)
    # per direction: [3, 3, N0, msl, vs]; the temporal lines are carried from
    # both sides, C(x0, T) = U0(x0+T-1)^dag C(x0, T-1) U0(x0+T-1, +R k)
    for k in range(3):
        lev = [levels[s][k] for s in range(msl)]
        line = list(lev)
        for r in range(1, c["r"] + 1):
            if r > 1:
                line = [_mm(line[s], torch.roll(lev[s], -(r - 1), 3 + k)) for s in range(msl)]
            flat = torch.stack(line, 3).reshape(3, 3, n[0], msl, vs)
            left = u[0].reshape(3, 3, n[0], 1, vs)
            right = torch.roll(u[0], -r, 3 + k).reshape(3, 3, n[0], 1, vs)
            # rows (x0, entry), so that one product serves every slice
            real = torch.view_as_real(flat.permute(2, 0, 1, 3, 4).contiguous())
            real = real.reshape(n[0], 9, msl, 2 * vs)
            car = flat
            for t in range(1, c["t"] + 1):
                lt, rt = (torch.roll(x, -(t - 1), 2) for x in (left, right))
                car = _mm(_mm(lt, car, dag_a=True), rt)
                cr = torch.view_as_real(car.permute(2, 0, 1, 3, 4).contiguous())
                cr = cr.reshape(n[0], 9, msl, 2 * vs)
                top = torch.roll(real, -t, 0)
                wl[:, r - 1, t - 1] += torch.matmul(top, cr.transpose(2, 3)).sum(1)
    wl /= 9.0 * vs
    return wl.reshape(-1).cpu().numpy(), np.array(plaq)


def exact(case, seed):
    c = case
    lats = _lattices(c)
    if c["kind"] == "smear":
        n = lats[0]
        nss = _nss(c)
        u = _hyp(_field(n, c["bc"], c["eps"], 1000 * seed), HYP2, c["proj_iter"])
        for _ in range(nss[0]):
            u = _ape(u, 0.1, c["proj_iter"], (0, 1, 2, 3))
        for _ in range(nss[1]):
            u = _hyp_spatial(u, 0.75, 0.6, c["proj_iter"])
        count = (6 * n[0] - (3 if c["bc"] == 0 else 0)) * n[1] * n[2] * n[3]
        return [_plaq(u, n, c["bc"]) / count, _host(u, False)]
    got = [_measure(c, n, 1000 * seed + i) for i, n in enumerate(lats)]
    return [wl for wl, _ in got] if c["kind"] == "batch" else list(got[0])
