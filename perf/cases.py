"""Performance cases: the work a user of this package has it do, through its public entry points.

A case is a dict of plain values; ``kind`` names the entry point and the rest are its sizes.  The listed sizes are
those of the package's own workloads (``swfwi_b200.survey.config``, the preconditioner's demonstration grids and the
reference's 533 x 193 stencil check) with shorter time axes; ``draw`` spreads the same kinds over odd sizes.

Inputs come from a seed alone: layered velocity models with dipping interfaces and smooth perturbations, Ricker
wavelets, band-limited reflection traces.  ``exact`` restates each path in FP64 with torch.
"""
import math

import numpy as np
import torch

import swfwi_b200 as S
from swfwi_b200.precond import Preconditioner

NB = 30   # sponge cells of every survey here


def listed():
    return [
        # the drop-in stencil step, one call on the grid of the reference's own stencil check: launch latency
        dict(name="step", kind="step", nx=533, nz=193, damped=True),
        # modelling one shot of the plain-FWI survey in the default (reference-identical) arithmetic
        dict(name="forward", kind="forward", nx=461, nz=151, nt=500, ns=1, arith="ref", dx=25.0, dt=0.002, fm=10.0),
        # the ensemble filter's modelling loop: one encoded supershot for every member's velocity
        dict(name="members", kind="members", nx=461, nz=201, nt=400, ns=16, n=64, dx=20.0, dt=0.002, fm=10.0),
        # the encoded-source gradient of the 921 x 301 survey: one supershot of 96 sources
        dict(name="encoded", kind="encoded", nx=921, nz=301, nt=1000, ns=96, strips="f32", dx=10.0, dt=0.001, fm=15.0),
        # the plain-FWI gradient of the 461 x 151 survey: 20 shots on one receiver line
        dict(name="gradient", kind="gradient", nx=461, nz=151, nt=800, ns=20, strips="f32", uneven=False, dx=25.0,
             dt=0.002, fm=10.0),
        # the largest: the batched gradient of 96 shots with uneven receiver spreads
        dict(name="gradient_batch", kind="gradient", nx=921, nz=301, nt=1000, ns=96, strips="f32", uneven=True,
             dx=10.0, dt=0.001, fm=15.0),
        # one whole encoded-source inversion epoch (gradient, direction, step-length search, update)
        dict(name="epoch", kind="epoch", nx=461, nz=151, nt=800, ns=20, dx=25.0, dt=0.002, fm=10.0),
        # the ensemble Kalman analysis: gain and member update
        dict(name="analysis", kind="analysis", nx=461, nz=201, nt=1000, ng=461, n=64),
        # least-squares migration's operator, both directions
        dict(name="born", kind="lsrtm", nx=461, nz=151, nt=500, ns=20, adj=False, exact_adj=False, arith="fast"),
        dict(name="migrate", kind="lsrtm", nx=461, nz=151, nt=500, ns=20, adj=True, exact_adj=True, arith="fast"),
        # the learned preconditioner: a proposal inside an epoch (one image), and a training step (a batch)
        dict(name="propose", kind="propose", nx=480, nz=160),
        dict(name="train", kind="train", N=16, H=480, W=160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "forward", "members", "encoded", "gradient", "epoch", "analysis", "lsrtm", "propose",
                       "train"])
    phys = dict(dx=25.0, dt=0.002, fm=10.0)
    if kind == "step":
        return dict(kind=kind, nx=_log_int(rng, 120, 1000), nz=_log_int(rng, 100, 400), damped=rng.random() < 0.7)
    nx, nz = _log_int(rng, 150, 921), _log_int(rng, 80, 301)
    if kind == "forward":
        return dict(kind=kind, nx=nx, nz=nz, nt=rng.randint(200, 600), ns=_log_int(rng, 1, 20),
                    arith=rng.choice(["ref", "fast"]), **phys)
    if kind == "members":
        return dict(kind=kind, nx=rng.randint(150, 461), nz=rng.randint(80, 201), nt=rng.randint(150, 400),
                    ns=rng.randint(4, 24), n=rng.randint(4, 64), **phys)
    if kind == "encoded":
        return dict(kind=kind, nx=nx, nz=nz, nt=rng.randint(300, 1000), ns=rng.randint(4, 96),
                    strips=rng.choice(["f32", "f32", "f16", "bf16"]), **phys)
    if kind == "gradient":
        return dict(kind=kind, nx=nx, nz=nz, nt=rng.randint(300, 800), ns=_log_int(rng, 2, 48),
                    strips=rng.choice(["f32", "f32", "f16", "bf16"]), uneven=rng.random() < 0.5, **phys)
    if kind == "epoch":
        return dict(kind=kind, nx=nx, nz=nz, nt=rng.randint(300, 800), ns=rng.randint(4, 48), **phys)
    if kind == "analysis":
        return dict(kind=kind, nx=rng.randint(150, 461), nz=rng.randint(80, 201), nt=rng.randint(300, 1000),
                    ng=rng.randint(100, 461), n=rng.randint(8, 64))
    if kind == "lsrtm":
        return dict(kind=kind, nx=rng.randint(150, 461), nz=rng.randint(80, 151), nt=rng.randint(200, 500),
                    ns=_log_int(rng, 1, 20), adj=rng.random() < 0.5, exact_adj=rng.random() < 0.7,
                    arith=rng.choice(["fast", "fast", "ref"]))
    if kind == "propose":
        return dict(kind=kind, nx=_log_int(rng, 150, 921), nz=_log_int(rng, 80, 301))
    return dict(kind=kind, N=rng.randint(2, 16), H=8 * rng.randint(15, 60), W=8 * rng.randint(8, 20))


# ---------------------------------------------------------------- inputs
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _model(nx, nz, seed, lo=1500.0, hi=4700.0):
    """Seven layers with dipping interfaces, plus a smooth +-150 m/s perturbation: [nx][nz] float32."""
    rng = np.random.default_rng(seed)
    x = np.arange(nx)[:, None] - nx / 2.0
    z = np.arange(nz)[None, :]
    depth = np.sort(rng.uniform(0.12, 0.92, 6)) * nz
    dip = rng.uniform(-0.12, 0.12, 6) * nz / nx
    vel = np.sort(rng.uniform(lo, hi, 7))
    v = np.full((nx, nz), vel[0])
    for k in range(6):
        v = np.where(z >= depth[k] + dip[k] * x, vel[k + 1], v)
    coarse = torch.from_numpy(rng.uniform(-150.0, 150.0, (1, 1, max(2, nx // 10), max(2, nz // 10))))
    fine = torch.nn.functional.interpolate(coarse, size=(nx, nz), mode="bicubic", align_corners=True)
    return np.clip(v + fine[0, 0].numpy(), lo, hi).astype(np.float32)


def _ricker(nt, dt, fm):
    a = (np.pi * fm * (np.arange(nt) * dt - 1.0 / fm)) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _traces(n, nt, ng, dt, dx, fm, seed, jitter=0.0):
    """Reflection traces [n][nt][ng] float32: six hyperbolic Ricker arrivals per trace from a source that moves
    along the line, with `jitter` seconds of spread between the n gathers."""
    rng = np.random.default_rng(seed + 7919)
    dev = _dev()
    out = torch.zeros((n, nt, ng), dtype=torch.float32, device=dev)
    t = torch.arange(nt, device=dev, dtype=torch.float32)[:, None] * dt
    g = torch.arange(ng, device=dev, dtype=torch.float32)[None, :]
    t0, v, a = rng.uniform(0.1, 0.9, 6) * nt * dt, rng.uniform(1800, 4000, 6), rng.uniform(-0.5, 0.5, 6)
    for i in range(n):
        sx = 0.5 * ng if jitter else (i + 0.5) * ng / n
        shift = rng.normal(0.0, 1.0, 6) * jitter
        for k in range(6):
            tau = torch.sqrt(float(t0[k] + shift[k]) ** 2 + ((g - sx) * (dx / float(v[k]))) ** 2)
            w = (math.pi * fm * (t - tau)) ** 2
            out[i] += float(a[k]) * (1.0 - 2.0 * w) * torch.exp(-w)
    return out


def _blob(n, nx, nz, seed):
    """Two smooth wavefields [n][nx][nz] one step apart: Gaussian pulses."""
    rng = np.random.default_rng(seed)
    x, z = np.arange(nx)[:, None], np.arange(nz)[None, :]
    out = []
    pulses = [(rng.uniform(0.1, 0.9) * nx, rng.uniform(0.1, 0.9) * nz, rng.uniform(4, 9), rng.uniform(-1, 1))
              for _ in range(8)]
    for step in range(2):
        f = np.zeros((nx, nz))
        for cx, cz, w, a in pulses:
            f += a * np.exp(-(((x - cx - 0.2 * step) ** 2 + (z - cz) ** 2) / (w * w)))
        out.append(torch.from_numpy(f.astype(np.float32)).to(_dev())[None].repeat(n, 1, 1).contiguous())
    return out


def _survey(c):
    """Source and receiver lines of a survey case."""
    jsx = max(1, (c["nx"] - 2) // c["ns"])
    return dict(ns=c["ns"], sxbeg=(c["nx"] - 1 - (c["ns"] - 1) * jsx) // 2, jsx=jsx, szbeg=6, ng=c["nx"], gzbeg=6)


def _spreads(c, seed):
    """Per-shot receiver spreads of seeded lengths around each source, as offsets and coordinates."""
    s = _survey(c)
    rng = np.random.default_rng(seed + 11)
    off, gx = [0], []
    for i in range(s["ns"]):
        m = int(rng.integers(max(2, c["nx"] // 5), c["nx"] + 1))
        a = min(max(s["sxbeg"] + i * s["jsx"] - m // 2, 0), c["nx"] - m)
        gx.append(np.arange(a, a + m))
        off.append(off[-1] + m)
    gx = np.concatenate(gx)
    return np.asarray(off, np.int32), gx.astype(np.int32), np.full(gx.size, s["gzbeg"], np.int32)


def _observed(c, ngmax, spreads, seed):
    """Observed gathers [ns][nt][ngmax], zero past each shot's own spread."""
    d = _traces(c["ns"], c["nt"], ngmax, c["dt"], c["dx"], c["fm"], seed)
    if spreads is not None:
        for i, m in enumerate(np.diff(spreads[0])):
            d[i, :, int(m):] = 0.0
    return d


def _propagator(c, arith, spreads=None):
    s = _survey(c)
    m = S.Damp4t10d(S.ShotPosition(s["szbeg"], s["sxbeg"], 0, s["jsx"], s["ns"], c["nz"]),
                    S.ShotPosition(s["gzbeg"], 0, 0, 1, s["ng"], c["nz"]), c["dt"], c["dx"], c["fm"], NB, c["nt"],
                    arith=arith)
    m.setModelSize(c["nx"], c["nz"])
    if spreads is not None:
        m.setReceiversPerShot(*spreads)
    return m


def _codes(ns, seed):
    return (np.random.default_rng(seed + 3).integers(0, 2, ns) * 2 - 1).astype(np.int32)


def _encoded_source(c, seed):
    return torch.from_numpy(_ricker(c["nt"], c["dt"], c["fm"])[:, None]
                            * _codes(c["ns"], seed)[None, :].astype(np.float32)).to(_dev())


def _net_params(widths, seed):
    """He-uniform convolutions, small biases: (flat parameters, [(cin, cout, weight offset, bias offset)])."""
    a, b, c, d = widths
    io = [(16, a), (a, a), (a, b), (b, b), (b, c), (c, c), (c, d), (d, d), (d + c, c), (c, c), (c + b, b), (b, b),
          (b + a, a), (a, a)]
    rng = np.random.default_rng(seed + 5)
    parts, layers, off = [], [], 0
    for ci, co in io:
        lim = math.sqrt(6.0 / (9.0 * ci))
        layers.append((ci, co, off, off + co * 9 * ci))
        parts += [rng.uniform(-lim, lim, co * 9 * ci), rng.uniform(-0.05, 0.05, co)]
        off += co * 9 * ci + co
    layers.append((a, 1, off, off + a))
    parts += [rng.uniform(-1, 1, a) / math.sqrt(a), np.zeros(1)]
    return np.concatenate(parts).astype(np.float32), layers


def _image(N, H, W, ch, seed):
    """Smooth unit-RMS images [N][H][W][ch] with some fine-scale noise."""
    g = torch.Generator().manual_seed(seed)
    coarse = torch.randn((N, ch, max(2, H // 12), max(2, W // 12)), generator=g)
    x = torch.nn.functional.interpolate(coarse, size=(H, W), mode="bilinear", align_corners=True)
    x = x + 0.2 * torch.randn((N, ch, H, W), generator=g)
    x = x / x.square().mean(dim=(2, 3), keepdim=True).sqrt()
    return x.permute(0, 2, 3, 1).contiguous().to(_dev())


def _fields3(c, seed):
    """Padded gradient, transformed velocity and illumination of a survey grid: float32 [nxpad][nzpad]."""
    nxp, nzp = c["nx"] + 2 * NB + 12, c["nz"] + NB + 12
    x = _image(1, nxp, nzp, 2, seed)[0]
    grad = x[..., 0].contiguous() * 3.0e4
    vel = torch.from_numpy(_expand(_model(c["nx"], c["nz"], seed), 25.0, 0.002)).to(_dev())
    z = torch.arange(nzp, device=_dev(), dtype=torch.float32)[None, :]
    illum = (x[..., 1].square() + 0.1) * torch.exp(-z / 40.0)
    return grad, vel, illum.contiguous()


def _hona(c, seed):
    """Member seismograms [n][ng*nt] and the observed data [ng*nt], trace by trace."""
    d = _traces(c["n"] + 1, c["nt"], c["ng"], 0.002, 20.0, 10.0, seed, jitter=0.02)
    d = d.transpose(1, 2).reshape(c["n"] + 1, -1)
    return d[1:].contiguous(), d[0].contiguous()


def _member_models(c, seed):
    base = _model(c["nx"], c["nz"], seed, 1700.0, 4300.0)
    ex = torch.from_numpy(_expand(base, 20.0, 0.002)).to(_dev())
    g = torch.Generator().manual_seed(seed)
    p = torch.randn((1, c["n"], max(2, c["nx"] // 10), max(2, c["nz"] // 10)), generator=g) * 0.03
    p = torch.nn.functional.interpolate(p, size=tuple(ex.shape), mode="bilinear", align_corners=True)[0]
    return (ex[None] * (1.0 + p.clamp(-0.1, 0.1).to(_dev()))).contiguous()


def _expand(v, dx, dt):
    """The padded transformed model: sponge on three sides, a 6-cell halo, dx^2 / (v^2 dt^2)."""
    v = np.pad(v.astype(np.float32), ((NB, NB), (0, NB)), mode="edge")
    dx, dt = np.float32(dx), np.float32(dt)
    return np.ascontiguousarray(np.pad((dx * dx) / (v * v * dt * dt), 6, mode="edge"))


# ---------------------------------------------------------------- prepare / run
ARITH = {"ref": S.ARITH_REF, "fast": S.ARITH_FAST}
STRIPS = {"f32": S.STRIP_F32, "f16": S.STRIP_F16, "bf16": S.STRIP_BF16}


def prepare(case, seed):
    c, k = case, case["kind"]
    dev = _dev()
    if k == "step":
        vt = torch.from_numpy(_expand(_model(c["nx"] - 2 * NB - 12, c["nz"] - NB - 12, seed), 25.0, 0.002)).to(dev)
        p0, p1 = _blob(1, c["nx"], c["nz"], seed)
        return dict(case=c, prev=p0[0], curr=p1[0], vel=vt)
    if k in ("forward", "members", "encoded", "gradient"):
        spreads = _spreads(c, seed) if c.get("uneven") else None
        m = _propagator(c, ARITH[c.get("arith", "fast")], spreads)
        vt = torch.from_numpy(m.expandDomain(_model(c["nx"], c["nz"], seed))).to(dev)
        m.bindVelocity(vt)
        st = dict(case=c, m=m, vel=vt, wlt=torch.from_numpy(_ricker(c["nt"], c["dt"], c["fm"])).to(dev))
        ngmax = m.getng()
        if k == "forward":
            st["dcal"] = torch.zeros((c["ns"], c["nt"], ngmax), device=dev)
        elif k == "members":
            st["vels"] = _member_models(c, seed)
            st["encsrc"] = _encoded_source(c, seed)
            st["hona"] = torch.empty((c["n"], ngmax * c["nt"]), device=dev)
        else:
            m.set_strip_format(STRIPS[c["strips"]])
            st["grad"] = torch.zeros_like(vt)
            if k == "encoded":
                st["encsrc"] = _encoded_source(c, seed)
                tr = _traces(1, c["nt"], ngmax, c["dt"], c["dx"], c["fm"], seed)
                st["vsrc"] = _trans64(tr.to(F64))[0].float().contiguous()
            else:
                st["dobs"] = _observed(c, ngmax, spreads, seed)
        return st
    if k == "epoch":
        m = _propagator(c, S.ARITH_REF)
        true = torch.from_numpy(m.expandDomain(_model(c["nx"], c["nz"], seed))).to(dev)
        m.bindVelocity(true)
        wlt = _ricker(c["nt"], c["dt"], c["fm"])
        dobs = torch.zeros((c["ns"], c["nt"], c["nx"]), device=dev)
        m.forward_batch(torch.from_numpy(wlt).to(dev), dobs, np.arange(c["ns"], dtype=np.int32))
        v0 = torch.from_numpy(_model(c["nx"], c["nz"], seed))[None, None]
        v0 = torch.nn.functional.avg_pool2d(torch.nn.functional.pad(v0, (15, 15, 15, 15), mode="replicate"), 31, 1)
        m = _propagator(c, S.ARITH_FAST)
        start = m.expandDomain(v0[0, 0].numpy())
        fw = S.EssFwiFramework(m, start, 1500.0, 4700.0, 5, 200.0, wlt, dobs.cpu().numpy())
        return dict(case=c, m=m, fw=fw, it=0)
    if k == "analysis":
        hona, dobs = _hona(c, seed)
        return dict(case=c, hona=hona, dobs=dobs, vels=_member_models(c, seed), seed=seed)
    if k == "lsrtm":
        vel = torch.from_numpy(_model(c["nx"], c["nz"], seed, 1500.0, 4000.0)).to(dev)
        s = _survey(c)
        op = S.Prtm2d(vel, 25.0, 25.0, 0.002, 1.0, 10.0, NB, c["nt"], c["ns"], c["nx"], s["sxbeg"], 1, s["jsx"], 0, 0,
                      1, 1, 0, arith=ARITH[c["arith"]])
        if c["exact_adj"]:
            op.set_adjoint(S.PRTM_ADJ_EXACT)
        mod, dat = _lsrtm_arrays(c, seed)
        return dict(case=c, op=op, mod=mod, dat=dat)
    net = Preconditioner()
    net.set_params(_net_params(net.widths, seed)[0])
    if k == "propose":
        m = _propagator(dict(c, nt=8, ns=1, dt=0.002, dx=25.0, fm=10.0), S.ARITH_FAST)
        grad, vel, illum = _fields3(c, seed)
        return dict(case=c, net=net, m=m, grad=grad, vel=vel, illum=illum)
    return dict(case=c, net=net, x=_image(c["N"], c["H"], c["W"], 3, seed),
                t=_image(c["N"], c["H"], c["W"], 1, seed + 1)[..., 0].contiguous())


def _lsrtm_arrays(c, seed):
    """A reflectivity model for modelling; reflection gathers [ns][ng][nt] for migration."""
    v = _model(c["nx"], c["nz"], seed, 1500.0, 4000.0)
    mod = np.zeros_like(v)
    mod[:, 1:] = np.diff(v, axis=1) / 4000.0
    mod = torch.from_numpy(mod).to(_dev())
    if c["adj"]:
        d = _traces(c["ns"], c["nt"], c["nx"], 0.002, 25.0, 10.0, seed)
        return torch.zeros_like(mod), d.transpose(1, 2).contiguous()
    return mod, torch.zeros((c["ns"], c["nx"], c["nt"]), device=_dev())


def run(st):
    c, k = st["case"], st["case"]["kind"]
    if k == "step":
        if c["damped"]:
            S.fd4t10s_damp_zjh_2d_vtrans(st["prev"], st["curr"], st["vel"], NB + 6)
        else:
            S.fd4t10s_zjh_2d_vtrans(st["prev"], st["curr"], st["vel"])
        st["prev"], st["curr"] = st["curr"], st["prev"]
        return st["curr"]
    if k == "forward":
        m = st["m"]
        if c["ns"] == 1:
            m.FwiForwardModeling(st["wlt"], st["dcal"], 0)
        else:
            m.forward_batch(st["wlt"], st["dcal"], np.arange(c["ns"], dtype=np.int32))
        return st["dcal"]
    if k == "members":
        st["m"].ess_forward_members(st["encsrc"], st["vels"], st["hona"])
        return st["hona"]
    if k == "encoded":
        st["grad"].zero_()
        st["m"].calgradient_ess(st["encsrc"], st["vsrc"], st["grad"])
        return st["grad"]
    if k == "gradient":
        obj = st["m"].gradient_batch(st["wlt"], st["dobs"], np.arange(c["ns"], dtype=np.int32), st["grad"])
        return [st["grad"], obj]
    if k == "epoch":
        st["fw"].epoch(st["it"])
        st["it"] += 1
        return [st["fw"].velocity(), st["fw"].getUpdateObj()]
    if k == "analysis":
        t4, sigma, clip = S.enkf_analyze(st["hona"], st["dobs"], st["vels"], 20.0, 0.002, None, 0.1, 0.0, st["seed"])
        return [st["vels"], t4, sigma, clip]
    if k == "lsrtm":
        st["op"].lop(c["adj"], False, st["mod"], st["dat"])
        return st["mod"] if c["adj"] else st["dat"]
    if k == "propose":
        return st["net"].propose(st["m"], st["grad"], st["vel"], st["illum"])
    loss = st["net"].train_step(st["x"], st["t"], 1e-3)
    return [loss, st["net"].grads()]


# ---------------------------------------------------------------- work
def work(case):
    """What a pass cannot do without: inputs read once, outputs written once, the scheme's own operations
    (31 a point-update of the tenth-order step, 15 of the fourth-order one)."""
    c, k = case, case["kind"]
    if k == "step":
        p = (c["nx"] - 12) * (c["nz"] - 12)
        return dict(bytes=16 * p, flops=31 * p)
    if k == "analysis":
        rows, model = c["nt"] * c["ng"], (c["nx"] + 72) * (c["nz"] + 42)
        n = c["n"]
        return dict(bytes=4 * (n + 1) * rows + 8 * n * model, flops=6 * n * n * rows + 2 * n * n * model)
    if k == "lsrtm":
        p = (c["nx"] + 2 * NB) * (c["nz"] + 2 * NB) * c["nt"] * c["ns"]
        steps = 3 if c["adj"] else 2
        return dict(bytes=4 * (c["nx"] * c["nz"] * 2 + c["ns"] * c["nx"] * c["nt"]), flops=15 * p * steps)
    if k in ("propose", "train"):
        N, H, W = (c["N"], c["H"], c["W"]) if k == "train" else (1, -(-c["nx"] // 8) * 8, -(-c["nz"] // 8) * 8)
        p = N * H * W
        mac = 9 * p * (16 * 16 * 2 + 48 * 16 + 16 * 16 + (16 * 32 + 32 * 32 + 96 * 32 + 32 * 32) / 4
                       + (32 * 64 + 64 * 64 + 128 * 64 + 64 * 64) / 16 + 2 * 64 * 64 / 64)
        return dict(bytes=16 * p + 8 * 304721, flops=2 * mac * (3 if k == "train" else 1))
    nxp, nzp = c["nx"] + 2 * NB + 12, c["nz"] + NB + 12
    p, traces = (nxp - 12) * (nzp - 12), c["nx"] * c["nt"]
    if k == "members":
        return dict(bytes=4 * (c["n"] * (nxp * nzp + traces)), flops=31 * p * c["nt"] * c["n"])
    if k == "forward":
        return dict(bytes=4 * (nxp * nzp + c["ns"] * traces), flops=31 * p * c["nt"] * c["ns"])
    n = c["ns"] if k == "gradient" else 1
    sweeps = 5 if k == "epoch" else 3
    return dict(bytes=4 * (3 * nxp * nzp + (c["ns"] if k != "encoded" else 1) * traces),
                flops=31 * p * c["nt"] * n * sweeps)


# ---------------------------------------------------------------- exact
F64 = torch.float64
A = [float(np.float32(v)) for v in (1.53400796, 1.78858721, -0.31660756, 0.07612173, -0.01626042, 0.00216736)]


def _sponge(nx, nz, nb):
    """delta = 0.05 dist^2 on the left, right and bottom ramps, [nx][nz]."""
    d = np.zeros((nx, nz))
    ix, iz = np.arange(nx)[:, None], np.arange(nz)[None, :]
    d = np.where(ix < nb, (nb - ix) / nb, d)
    d = np.where(ix >= nx - nb, (ix - (nx - nb) + 1) / nb, d)
    d = np.where(iz >= nz - nb, (iz - (nz - nb) + 1) / nb, d)
    return torch.from_numpy(0.05 * d * d).to(_dev())


def _step64(p0, p1, r, delta):
    """The next field of [n][nx][nz] (in place over p0)."""
    nx, nz = p1.shape[-2:]
    core = p1[:, 5:nx - 5, 5:nz - 5]
    u = torch.mul(core, -4.0 * A[0])
    for k in range(1, 6):
        s = p1[:, 5:nx - 5, 5 - k:nz - 5 - k] + p1[:, 5:nx - 5, 5 + k:nz - 5 + k]
        s += p1[:, 5 - k:nx - 5 - k, 5:nz - 5]
        s += p1[:, 5 + k:nx - 5 + k, 5:nz - 5]
        u.add_(s, alpha=A[k])
    uc = u[:, 1:-1, 1:-1]
    lap = u[:, 1:-1, :-2] + u[:, 1:-1, 2:]
    lap += u[:, :-2, 1:-1]
    lap += u[:, 2:, 1:-1]
    lap.add_(uc, alpha=-4.0)
    i = (slice(None), slice(6, nx - 6), slice(6, nz - 6))
    rr = r[..., 6:nx - 6, 6:nz - 6]
    lap.mul_(rr / 12.0).add_(uc).mul_(rr)
    if delta is None:
        p0[i] = 2.0 * p1[i] - p0[i] + lap
    else:
        d = delta[6:nx - 6, 6:nz - 6]
        p0[i] = (2.0 - 2.0 * d + d * d) * p1[i] - (1.0 - 2.0 * d) * p0[i] + lap
    return p0


class _Survey64:
    """Modelling and gradient of the listed sources in FP64."""

    def __init__(self, c, vt, spreads=None):
        s = _survey(c)
        self.c, self.nt = c, c["nt"]
        self.nxp, self.nzp = c["nx"] + 2 * NB + 12, c["nz"] + NB + 12
        self.r = 1.0 / vt.to(F64)
        self.delta = _sponge(self.nxp, self.nzp, NB + 6)
        self.src = (np.arange(s["ns"]) * s["jsx"] + s["sxbeg"] + NB + 6) * self.nzp + s["szbeg"] + 6
        if spreads is None:
            self.rec = np.tile((np.arange(s["ng"]) + NB + 6) * self.nzp + s["gzbeg"] + 6, (s["ns"], 1))
            self.used = np.ones(self.rec.shape, bool)
        else:
            off, gx, _ = spreads
            m = int(np.max(np.diff(off)))
            self.rec, self.used = np.zeros((s["ns"], m), np.int64), np.zeros((s["ns"], m), bool)
            for i in range(s["ns"]):
                g = gx[off[i]:off[i + 1]].astype(np.int64)
                self.rec[i, :g.size], self.used[i, :g.size] = (g + NB + 6) * self.nzp + s["gzbeg"] + 6, True
        self.x0, self.x1, self.z0, self.z1 = NB + 6, self.nxp - NB - 6, 6, self.nzp - NB - 6
        band = torch.zeros((self.nxp, self.nzp), dtype=torch.bool)
        band[self.x0 - 6:self.x1 + 6, self.z0:self.z1 + 6] = True
        band[self.x0:self.x1, self.z0:self.z1] = False
        self.band = band.reshape(-1).nonzero()[:, 0].to(_dev())

    def fields(self, n):
        return [torch.zeros((n, self.nxp, self.nzp), dtype=F64, device=_dev()) for _ in range(2)]

    def forward(self, n, src, vals, rec, keep):
        """src [n][m] positions with vals [nt][n or 1][m]; returns the traces [n][nt][ng], the strips and the last two
        fields.  As in the scheme, step `it` records and saves the field it advances from, its source added."""
        src, rec = torch.as_tensor(src, device=_dev()), torch.as_tensor(rec, device=_dev())
        p0, p1 = self.fields(n)
        d = torch.zeros((n, self.nt, rec.shape[1]), dtype=F64, device=_dev())
        strips = []
        for it in range(self.nt):
            p1.view(n, -1).scatter_add_(1, src, vals[it].expand(n, -1))
            p0, p1 = p1, _step64(p0, p1, self.r, self.delta)
            d[:, it] = p0.view(n, -1).gather(1, rec)
            if keep:
                strips.append(p0.view(n, -1)[:, self.band])
        return d, strips, p0, p1

    def gradient(self, n, src, vals, rec, vsrc, strips, p0, p1):
        """The image of a backward sweep: the source field rebuilt from its strips, the residual injected."""
        src, rec = torch.as_tensor(src, device=_dev()), torch.as_tensor(rec, device=_dev())
        g0, g1 = self.fields(n)
        img = torch.zeros((n, self.nxp, self.nzp), dtype=F64, device=_dev())
        s0, s1 = p0, p1
        dt = np.float32(self.c["dt"])
        for it in range(self.nt - 1, -1, -1):
            s0.view(n, -1)[:, self.band] = strips[it]
            s0, s1 = s1, s0
            _step64(s0, s1, self.r, None)
            s0.view(n, -1).scatter_add_(1, src, -vals[it].expand(n, -1))
            g1.view(n, -1).scatter_add_(1, rec, vsrc[:, it])
            g0, g1 = g1, _step64(g0, g1, self.r, self.delta)
            t = float(dt * np.float32(it))
            scale = 1.0 if t > 0.4 else (t - 0.3) / 0.1 if t > 0.3 else None
            if scale is None:
                break
            img.addcmul_(s0, g0, value=-scale)
        return img


def _mute(c, vt, sxz, rec, used, nt):
    """The direct-arrival window of each trace: a bool [nt][ng] that is True where data are zeroed.  Window edges
    are whole samples of single-precision times, so they are formed in single precision here too."""
    half = int(np.float32(1.5 / float(np.float32(c["fm"]))) / np.float32(c["dt"]))
    nxp, nzp = vt.shape
    sx, sz = sxz
    gx, gz = rec // nzp, rec % nzp
    lo, hi = min(sz, int(gz[0])), max(sz, int(gz[0]))
    total = np.cumsum(vt[:, lo:hi + 1].reshape(-1).astype(np.float32), dtype=np.float32)[-1]
    avg = np.float32(total / np.float32(nxp * (hi - lo + 1)))
    t = np.sqrt(((gx - sx) ** 2 + (gz - sz) ** 2).astype(np.float32) * avg).astype(np.int64)
    it = np.arange(nt)[:, None]
    return torch.from_numpy(used[None, :] & (it >= t[None, :]) & (it < t[None, :] + 2 * half)).to(_dev())


def _trans64(r):
    v = torch.zeros_like(r)
    v[:, 2:-2] = (-r[:, :-4] + 16.0 * r[:, 1:-3] - 30.0 * r[:, 2:-2] + 16.0 * r[:, 3:-1] - r[:, 4:]) / 12.0
    return v


def _exact_survey(c, seed):
    k = c["kind"]
    points = (c["nx"] + 72) * (c["nz"] + 42) * c["nt"] * {"gradient": 3 * c["ns"], "forward": c["ns"], "encoded": 3}.get(
        k, c.get("n", 1))
    if points > 9e9:
        return None
    vt_host = _expand(_model(c["nx"], c["nz"], seed), c["dx"], c["dt"])
    vt = torch.from_numpy(vt_host).to(_dev())
    wlt = torch.from_numpy(_ricker(c["nt"], c["dt"], c["fm"])).to(_dev(), F64)[:, None, None]
    spreads = _spreads(c, seed) if c.get("uneven") else None
    if k == "members":
        e = _Survey64(c, _member_models(c, seed))
        n = c["n"]
        enc = _encoded_source(c, seed).to(F64)[:, None, :]
        d, _, _, _ = e.forward(n, np.tile(e.src, (n, 1)), enc, np.tile(e.rec[0], (n, 1)), False)
        return d.transpose(1, 2).reshape(n, -1)
    e = _Survey64(c, vt, spreads)
    if k == "forward":
        d, _, _, _ = e.forward(c["ns"], e.src[:, None], wlt, e.rec, False)
        return d
    if k == "encoded":
        enc = _encoded_source(c, seed).to(F64)[:, None, :]
        tr = _traces(1, c["nt"], c["nx"], c["dt"], c["dx"], c["fm"], seed)
        _, strips, p0, p1 = e.forward(1, e.src[None, :], enc, e.rec[:1], True)
        return e.gradient(1, e.src[None, :], enc, e.rec[:1], _trans64(tr.to(F64)).float().to(F64), strips, p0, p1)[0]
    d, strips, p0, p1 = e.forward(c["ns"], e.src[:, None], wlt, e.rec, True)
    used = torch.from_numpy(e.used).to(_dev())[:, None, :]
    obs = _observed(c, e.rec.shape[1], spreads, seed).to(F64)
    cal = d * used
    for i in range(c["ns"]):
        mute = _mute(c, vt_host, (int(e.src[i]) // e.nzp, int(e.src[i]) % e.nzp), e.rec[i], e.used[i], c["nt"])
        obs[i][mute] = 0.0
        cal[i][mute] = 0.0
    res = obs - cal
    obj = res.square().sum(dim=(1, 2))
    img = e.gradient(c["ns"], e.src[:, None], wlt, e.rec, _trans64(res) * used, strips, p0, p1)
    iz = torch.arange(e.nzp, device=_dev(), dtype=F64) - 6.0
    img = (img * torch.where(iz >= 1, iz.clamp(min=1).sqrt(), torch.ones_like(iz))).sum(0)
    out = torch.zeros_like(img)
    out[e.x0:e.x1, e.z0:e.z1] = img[e.x0:e.x1, e.z0:e.z1]
    return [out, obj.cpu().numpy()]


def _exact_lsrtm(c, seed):
    """Modelling from zero fields, its transpose, or the reference's migration, in FP64; the reference-identical
    arithmetic carries fields from shot to shot and is left out."""
    if c["arith"] == "ref":
        return None
    nx, nz, nt, ns, nb = c["nx"], c["nz"], c["nt"], c["ns"], NB
    nxp, nzp = nx + 2 * nb, nz + 2 * nb
    dev = _dev()
    mod, dat = _lsrtm_arrays(c, seed)
    v = torch.from_numpy(np.pad(_model(nx, nz, seed, 1500.0, 4000.0), nb, mode="edge")).to(dev, F64)
    vv = (v * float(np.float32(0.002))) ** 2
    c1, c2 = 4.0 / (3.0 * 625.0), -1.0 / (12.0 * 625.0)
    c0 = -4.0 * (c1 + c2)
    tap = torch.exp(-(0.015 * (nb - 1 - torch.arange(nb, dtype=F64))) ** 2)

    def edge(n):
        w = torch.ones(n, dtype=F64)
        w[:nb], w[-nb:] = w[:nb] * tap, w[-nb:] * tap.flip(0)
        return w.to(dev)
    W = edge(nxp)[:, None] * edge(nzp)[None, :]
    it = np.arange(nt, dtype=np.float64)
    a = (np.pi * 10.0 * (it * float(np.float32(0.002)) - 0.1)) ** 2
    wl = (1.0 - 2.0 * a) * np.exp(-a)
    s = _survey(c)
    sx, sz = nb + s["sxbeg"] + s["jsx"] * torch.arange(ns, device=dev), nb + 1
    idx = torch.arange(ns, device=dev)
    mi = (slice(None), slice(nb, nb + nx), slice(nb, nb + nz))
    inner = (slice(None), slice(2, nxp - 2), slice(2, nzp - 2))

    def lap(u):
        o = c0 * u[:, 2:-2, 2:-2]
        o += c1 * (u[:, 2:-2, 1:-3] + u[:, 2:-2, 3:-1] + u[:, 1:-3, 2:-2] + u[:, 3:-1, 2:-2])
        o += c2 * (u[:, 2:-2, :-4] + u[:, 2:-2, 4:] + u[:, :-4, 2:-2] + u[:, 4:, 2:-2])
        return o

    def step(u0, u1):
        u0[inner] = 2.0 * u1[inner] - u0[inner] + vv[2:-2, 2:-2] * lap(u1)

    def zeros():
        return torch.zeros((ns, nxp, nzp), dtype=F64, device=dev)
    S0, S1, G0, G1 = zeros(), zeros(), zeros(), zeros()
    m64, d64 = mod.to(F64), dat.to(F64)
    if not c["adj"]:
        out = torch.zeros((ns, nx, nt), dtype=F64, device=dev)
        for t in range(nt):
            G1[mi] += S0[mi] * m64
            G0, G1 = G1, G0
            for f in (G0, G1, S0, S1):
                f *= W
            S1[idx, sx, sz] += wl[t]
            out[:, :, t] = G1[:, nb:nb + nx, nb + 1]
            G0[inner] = 2.0 * G1[inner] - G0[inner] + lap(vv * G1)
            step(S0, S1)
            S0, S1 = S1, S0
        return out
    ring = torch.zeros((nxp, nzp), dtype=torch.bool)
    ring[nb:nb + nx, nb - 2:nb] = True
    ring[nb:nb + nx, nb + nz:nb + nz + 2] = True
    ring[nb - 2:nb, nb:nb + nz] = True
    ring[nb + nx:nb + nx + 2, nb:nb + nz] = True
    ring = ring.reshape(-1).nonzero()[:, 0].to(dev)
    saved = []
    for t in range(nt):
        S1[idx, sx, sz] += wl[t]
        step(S0, S1)
        S0 *= W
        S1 *= W
        S0, S1 = S1, S0
        saved.append(S0.view(ns, -1)[:, ring])
    img = torch.zeros((ns, nx, nz), dtype=F64, device=dev)
    P = torch.zeros((nxp, nzp), dtype=F64, device=dev)
    P[2:-2, 2:-2] = 1.0
    pad = torch.nn.functional.pad
    for t in range(nt - 1, -1, -1):
        S0.view(ns, -1)[:, ring] = saved[t]
        if t + 1 < nt:
            S1[idx, sx, sz] -= wl[t + 1]
        G1[:, nb:nb + nx, nb + 1] += d64[:, :, t]
        S0, S1 = S1, S0
        step(S0, S1)
        if c["exact_adj"]:
            x = G0 * P
            new = W * (2.0 * x + vv * lap(pad(x, (2, 2, 2, 2))) + G1)
            G1 = W * (G0 * (1.0 - P) - x)
            G0 = new
            img += S0[mi] * G1[mi]
        else:
            step(G0, G1)
            G0 *= W
            G1 *= W
            G0, G1 = G1, G0
            img += S0[mi] * G1[mi]
    return img.sum(0)


def _normals(seed, first, n, dev):
    """Standard normals number first .. first+n-1 of a seed: Philox 4x32, ten rounds (Salmon et al. 2011), and the
    Box-Muller transform of its first two words."""
    mask = 0xFFFFFFFF
    i = torch.arange(first, first + n, dtype=torch.int64, device=dev)
    c = [i & mask, i >> 32, torch.zeros_like(i), torch.zeros_like(i)]
    k0, k1 = seed & mask, seed >> 32

    def mul(x, m):
        lo16 = (x & 0xFFFF) * m
        hi16 = (x >> 16) * m + (lo16 >> 16)
        return hi16 >> 16, ((hi16 & 0xFFFF) << 16) | (lo16 & 0xFFFF)
    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u1, u2 = (c[0].to(F64) + 1.0) / 2.0 ** 32, c[1].to(F64) / 2.0 ** 32
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)


def _exact_analysis(c, seed):
    hona, dobs = _hona(c, seed)
    n, rows = hona.shape
    h = hona.to(F64)
    hap = h - h.mean(0)
    key = hap.float().abs().reshape(-1)
    sigma = float(hap.reshape(-1)[int(torch.argmax(key))].abs() * float(np.float32(0.1)))
    pert = torch.stack([_normals(seed, i * rows, rows, hona.device) for i in range(n)]) * sigma
    band = (hap + pert - pert.mean(0)).t()
    res = (dobs.to(F64) + pert - h).t()
    q, r = torch.linalg.qr(band)
    u, s, _ = torch.linalg.svd(r)
    rel, acc, sv = float(np.float32(0.001)), 0.0, s.cpu().numpy()
    pos = 0
    while pos < n - 1:
        acc += abs(sv[pos])
        if rel / (1 - rel) * acc > (n - pos + 1) * sv[pos + 1]:
            break
        pos += 1
    clip = min(pos, n - 1) + 1
    uc = q @ u[:, :clip]
    t4 = (hap @ uc) @ ((uc.t() @ res) / s[:clip, None] ** 2)
    vels = _member_models(c, seed)
    mean = vels[0].clone()
    for j in range(1, n):
        mean += vels[j]
    mean = mean / n
    dev64 = (vels - mean).to(F64)
    t5 = torch.einsum("jxz,ji->ixz", dev64, t4)
    ratio = float(np.float32(20.0)) ** 2 / float(np.float32(0.002)) ** 2
    phys = torch.sqrt(ratio / vels.to(F64)) + t5
    return [ratio / phys.square(), t4.cpu().numpy(), sigma, clip]


def _net64(p, layers, x):
    """The network in FP64: x [N][3][H][W] -> [N][H][W]."""
    F = torch.nn.functional

    def conv(i, z):
        ci, co, wo, bo = layers[i]
        w = p[wo:wo + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        return torch.relu(F.conv2d(z, w, p[bo:bo + co], padding=1))

    def up(z, skip):
        return torch.cat([z.repeat_interleave(2, 2).repeat_interleave(2, 3), skip], 1)
    z = F.pad(x, (0, 0, 0, 0, 0, 13))
    skips = []
    for level in range(3):
        z = conv(2 * level + 1, conv(2 * level, z))
        skips.append(z)
        z = F.avg_pool2d(z, 2)
    z = conv(7, conv(6, z))
    for level in range(3):
        z = conv(9 + 2 * level, conv(8 + 2 * level, up(z, skips[2 - level])))
    ci, _, wo, bo = layers[14]
    return torch.einsum("nchw,c->nhw", z, p[wo:wo + ci]) + p[bo]


def exact(case, seed):
    c, k = case, case["kind"]
    dev = _dev()
    if k == "epoch":
        return None
    if k == "step":
        vt = torch.from_numpy(_expand(_model(c["nx"] - 2 * NB - 12, c["nz"] - NB - 12, seed), 25.0, 0.002)).to(dev)
        p0, p1 = (f.to(F64) for f in _blob(1, c["nx"], c["nz"], seed))
        delta = _sponge(c["nx"], c["nz"], NB + 6) if c["damped"] else None
        return _step64(p0, p1, 1.0 / vt.to(F64), delta)[0]
    if k in ("forward", "members", "encoded", "gradient"):
        return _exact_survey(c, seed)
    if k == "lsrtm":
        return _exact_lsrtm(c, seed)
    if k == "analysis":
        return _exact_analysis(c, seed)
    host, layers = _net_params((16, 32, 64, 64), seed)
    p = torch.from_numpy(host).to(dev, F64)
    if k == "propose":
        grad, vel, illum = (f.to(F64) for f in _fields3(c, seed))
        i = (slice(NB + 6, NB + 6 + c["nx"]), slice(6, 6 + c["nz"]))
        g, v, il = grad[i], vel[i], illum[i]
        f = torch.stack([g / g.square().mean().sqrt(), (v - v.mean()) / (v.square().mean() - v.mean() ** 2).sqrt(),
                         (torch.log10(il.clamp(min=0) / il.max() + 1e-6) + 3.0) / 3.0])
        f = torch.nn.functional.pad(f, (0, -c["nz"] % 8, 0, -c["nx"] % 8))
        out = torch.zeros_like(grad)
        out[i] = _net64(p, layers, f[None])[0, :c["nx"], :c["nz"]]
        return out
    p.requires_grad_(True)
    loss, mean = 0.0, 1.0 / (c["N"] * c["H"] * c["W"])
    x, t = _image(c["N"], c["H"], c["W"], 3, seed), _image(c["N"], c["H"], c["W"], 1, seed + 1)[..., 0]
    for i in range(c["N"]):
        part = (_net64(p, layers, x[i:i + 1].permute(0, 3, 1, 2).to(F64)) - t[i:i + 1].to(F64)).square().sum() * mean
        part.backward()
        loss += float(part.detach())
    return [loss, p.grad.cpu().numpy()]
