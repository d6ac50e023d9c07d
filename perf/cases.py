"""The propagation work that is measured: each case is one call (or one
forward and backward) that an optics program makes through the package's
light classes and optical elements, with its inputs, its arithmetic and what
it gives in 64 bits.

Kinds of case:

* ``rs``     scalar light behind a phase SLM, Rayleigh-Sommerfeld propagation;
* ``vrs``    vector light, VRS propagation; ``masked``: behind an LCD with
             per-pixel settings and a polarizer;
* ``czt``    scalar light behind a thin lens, chirp-z onto another grid;
* ``vczt``   vector light behind an LCD, vectorial chirp-z onto another grid;
* ``focus``  vector light behind a double-phase SLM, through the high-NA lens;
* ``fourf``  4f tables: loss and gradients of the two SLMs' phases;
* ``spot``   high-NA tables: loss on the focal Ez and gradients of the LCD's
             and the SLM's planes;
* ``block``  building block (SLM, VRS over a distance held on the device, LCD):
             loss and gradients of the SLM's and the LCD's planes.
"""
import math

import numpy as np
import torch

from xlumina_gb300 import loss_functions as lf
from xlumina_gb300 import optical_elements as oe
from xlumina_gb300.vectorized_optics import VectorizedLight
from xlumina_gb300.wave_optics import ScalarLight

WL = 0.633          # um
PITCH = 1.95        # um per pixel of an input grid
Z_SET = (1.0e4, 5.0e4, 1.0e5, 2.0e5)


def listed():
    return [
        # the smallest call: one small field, where launches and host work are all there is
        dict(name="rs 64 single", kind="rs", ny=64, nx=64, batch=1, zs=1),
        # the ordinary batched scalar propagation, one distance for the batch
        dict(name="rs 1024 x16", kind="rs", ny=1024, nx=1024, batch=16, zs=1),
        # a camera-sized field that is neither square nor a power of two
        dict(name="rs 1117x1301 x4", kind="rs", ny=1117, nx=1301, batch=4, zs=1),
        # the longest transforms
        dict(name="rs 4096 x2", kind="rs", ny=4096, nx=4096, batch=2, zs=1),
        # the vectorial propagation at the resolution that experiments use, four distances
        dict(name="vrs 2048 x8 masked", kind="vrs", ny=2048, nx=2048, batch=8, zs=4, masked=True),
        # a small vector field of odd size, one distance for each entry, no mask before it
        dict(name="vrs 601 x4", kind="vrs", ny=601, nx=601, batch=4, zs=4, masked=False),
        # a lens and its focal region, scalar
        dict(name="czt 1024-400 x4", kind="czt", ny=1024, nx=1024, my=400, mx=400, batch=4),
        # the same for vector light, sizes that are no powers of two
        dict(name="vczt 1500-301 x2", kind="vczt", ny=1500, nx=1500, my=301, mx=301, batch=2),
        # the high-NA objective's focal field, all three components
        dict(name="focus 2048-1024 x4", kind="focus", ny=2048, nx=2048, my=1024, mx=1024, batch=4),
        # one optimisation step's loss and gradients of a batch of 4f tables
        dict(name="fourf 1024-512 x16", kind="fourf", ny=1024, nx=1024, my=512, mx=512, batch=16),
        # and of high-NA tables
        dict(name="spot 2048-1024 x8", kind="spot", ny=2048, nx=2048, my=1024, mx=1024, batch=8),
        # the element that the large discovery tables are made of, one copy of it
        dict(name="block 1024", kind="block", ny=1024, nx=1024, batch=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("rs", "rs", "vrs", "vrs", "czt", "vczt", "focus", "fourf", "spot", "block"))
    # pixels of a case: within what the listed cases of its kind take
    most = {"rs": 2 * 4096 ** 2, "vrs": 8 * 2048 ** 2, "czt": 4 * 2048 ** 2, "vczt": 4 * 2048 ** 2,
            "focus": 4 * 2048 ** 2, "fourf": 16 * 1024 ** 2, "spot": 8 * 2048 ** 2, "block": 2 * 1024 ** 2}[kind]
    top = {"rs": 4096, "fourf": 1536, "block": 1400}.get(kind, 2048)
    n = _log_int(rng, 64 if kind in ("rs", "vrs") else 128, top)
    ny = n
    if kind in ("rs", "vrs") and rng.random() < 0.5:
        ny = max(48, int(n * rng.uniform(0.6, 1.0)))
    if kind in ("focus", "spot"):
        n += n % 2          # the lens has no value on the axis itself
        ny = n
    batch = max(1, min(_log_int(rng, 1, 32), most // (n * ny)))
    case = dict(kind=kind, ny=ny, nx=n, batch=batch)
    if kind == "rs":
        case["zs"] = rng.choice((1, min(batch, 4)))
    elif kind == "vrs":
        case["zs"] = rng.choice((1, min(batch, 4)))
        case["masked"] = rng.random() < 0.5
    elif kind == "block":
        case["batch"] = 1
    else:
        m = max(16, int(n * rng.uniform(0.2, 0.7)))
        while any(s & (s - 1) == 0 for s in (n + m - 1, 2 * m - 1)):   # sizes that the chirp-z refuses
            m += 1
        case["my"] = case["mx"] = m
    return case


# ------------------------------------------------------------------ inputs --

def _axis(n, pitch=PITCH):
    h = 0.5 * pitch * (n - 1)
    return np.linspace(-h, h, n)


def _grids(case):
    """Axes (x, y) and, where there are any, (xout, yout)."""
    k = case["kind"]
    x, y = _axis(case["nx"]), _axis(case["ny"])
    if "mx" not in case:
        return x, y
    h = {"fourf": 0.6 * x[-1], "czt": 0.25 * x[-1], "vczt": 0.25 * x[-1], "focus": 2.0, "spot": 1.0}[k]
    return x, y, np.linspace(-h, h, case["mx"]), np.linspace(-h, h, case["my"])


def _data(case, seed):
    """The tensors of a case, from its sizes and the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + case["ny"] * 31 + case["nx"])
    B, ny, nx = case["batch"], case["ny"], case["nx"]
    x, y = (torch.tensor(a, device="cuda") for a in _grids(case)[:2])
    w = 0.45 * float(x[-1])
    beam = torch.exp(-(x[None, :] ** 2 + y[:, None] ** 2) / w ** 2).to(torch.complex64)

    def field(*lead):      # a beam with weak speckle on it
        shape = lead + (ny, nx)
        return beam * (1 + 0.3 * torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g))

    def plane(lo, hi, shape):
        return torch.rand(shape, device="cuda", generator=g) * (hi - lo) + lo

    two, kind, d = (B, ny, nx), case["kind"], {}
    if B == 1:
        two = (ny, nx)
    lead = two[:-2]
    if kind == "rs":
        d = dict(field=field(*lead), phase=plane(-math.pi, math.pi, two))
    elif kind == "vrs":
        d = dict(ex=field(*lead), ey=field(*lead))
        if case["masked"]:
            d.update(eta=plane(0, 2 * math.pi, two), theta=plane(0, 2 * math.pi, two), alpha=0.3 + 0.01 * (seed % 100))
    elif kind == "czt":
        d = dict(field=field(*lead))
    elif kind == "vczt":
        d = dict(ex=field(*lead), ey=field(*lead), eta=plane(0, 2 * math.pi, (ny, nx)),
                 theta=plane(0, 2 * math.pi, (ny, nx)))
    elif kind == "focus":
        d = dict(ex=field(*lead), ey=field(*lead), alpha=plane(0, 2 * math.pi, two), phi=plane(0, 2 * math.pi, two))
    elif kind == "fourf":
        m = (case["my"], case["mx"])
        keep = (torch.rand(two, device="cuda", generator=g) > 0.5).to(torch.float32)
        tgt = (torch.rand(lead + m, device="cuda", generator=g) < 0.1).to(torch.float32) + 1e-3
        d = dict(field=field(*lead) * keep, p1=plane(-math.pi, math.pi, two), p2=plane(-math.pi, math.pi, lead + m),
                 target=tgt / tgt.sum(dim=(-2, -1), keepdim=True))
    elif kind == "spot":
        m = (case["my"], case["mx"])
        tgt = torch.rand(m, device="cuda", generator=g) ** 4
        d = dict(ex=field(), ey=field(), target=tgt / tgt.sum())
        d.update((k, plane(0, 2 * math.pi, two)) for k in ("eta", "theta", "alpha", "phi"))
    elif kind == "block":
        d = dict(ex=field(), ey=field(), target=[0.3 * field() for _ in range(3)],
                 z=torch.tensor([3.0e4 + 100.0 * (seed % 50)], dtype=torch.float64, device="cuda"))
        d.update((k, plane(-math.pi, math.pi, (ny, nx))) for k in ("alpha", "phi", "eta", "theta"))
    return d


TRAINED = {"fourf": ("p1", "p2"), "spot": ("eta", "theta", "alpha", "phi"),
           "block": ("alpha", "phi", "eta", "theta")}


def _distances(case):
    """The distance as the propagators take it: a number, or one for each batch entry."""
    if case["zs"] == 1 or case["batch"] == 1:
        return Z_SET[1]
    return [Z_SET[i % case["zs"]] for i in range(case["batch"])]


def _lens(case):
    """(lens radius, focal distance) of the chirp-z cases, (radius, f) of the high-NA ones."""
    h = float(_axis(case["nx"])[-1])
    if case["kind"] in ("focus", "spot"):
        return 0.95 * h, 0.95 * h / 0.9
    return 1.05 * h, 60.0 * h


def prepare(case, seed):
    d = _data(case, seed)
    grids = _grids(case)
    if "field" in d:
        light = ScalarLight(grids[0], grids[1], WL)
        light.field = d["field"]
    else:
        light = VectorizedLight(grids[0], grids[1], WL)
        B = case["batch"]
        lead = (B,) if case["kind"] == "spot" and B > 1 else None
        light.Ex = d["ex"].expand(lead + d["ex"].shape) if lead else d["ex"]
        light.Ey = d["ey"].expand(lead + d["ey"].shape) if lead else d["ey"]
    target = None
    if case["kind"] == "block":
        target = VectorizedLight(grids[0], grids[1], WL)
        target.Ex, target.Ey, target.Ez = d["target"]
    trained = TRAINED.get(case["kind"], ())
    for k in trained:
        d[k].requires_grad_(True)
    return dict(case=case, d=d, grids=grids, light=light, target=target, trained=trained)


# --------------------------------------------------------------- one pass --

def run(state):
    case, d, light = state["case"], state["d"], state["light"]
    kind = case["kind"]
    if kind == "rs":
        return oe.SLM(light, d["phase"], case["nx"])[0].RS_propagation(_distances(case))[0].field
    if kind == "vrs":
        if case["masked"]:
            light = oe.linear_polarizer(oe.LCD(light, d["eta"], d["theta"]), d["alpha"])
        out = light.VRS_propagation(_distances(case))[0]
        return out.Ex, out.Ey, out.Ez
    x, y = state["grids"][:2]
    if kind == "block":
        out = oe.building_block(light, d["alpha"], d["phi"], d["z"], d["eta"], d["theta"])
        return _gradients(torch.mean(lf.vMSE_Intensity(out, state["target"])), state)
    xo, yo = state["grids"][2:]
    r, f = _lens(case)
    if kind == "czt":
        return oe.lens(light, (r, r), (f, f))[0].CZT(f, xo, yo).field
    if kind == "vczt":
        out = oe.LCD(light, d["eta"], d["theta"]).VCZT(f, xo, yo)
        return out.Ex, out.Ey, out.Ez
    if kind == "focus":
        out = oe.VCZT_objective_lens(oe.sSLM(light, d["alpha"], d["phi"]), r, f, xo, yo)
        return out.Ex, out.Ey, out.Ez
    if kind == "fourf":
        a, _ = oe.SLM(light, d["p1"], case["nx"])
        b, _ = a.RS_propagation(f)
        c, _ = oe.lens(b, (r, r), (f, f))
        e, _ = oe.SLM(c.CZT(f, xo, yo), d["p2"], case["mx"])
        out = e.CZT(f).field
        return _gradients(torch.mean(lf.normalized_intensity_mse(out, d["target"])), state)
    masked = oe.sSLM(oe.LCD(light, d["eta"], d["theta"]), d["alpha"], d["phi"])
    ez = oe.VCZT_objective_lens_ez(masked, r, f, xo, yo)
    return _gradients(torch.mean(lf.normalized_intensity_mse(ez, d["target"])), state)


def _gradients(loss, state):
    """The loss and the gradients of what the case trains, as an optimiser reads them."""
    params = [state["d"][k] for k in state["trained"]]
    for p in params:
        p.grad = None
    loss.backward()
    return [loss.detach()] + [p.grad for p in params]


# ------------------------------------------------------------ what it needs --

def _fft_flops(lines, n):
    return 5.0 * lines * n * math.log2(n)


def work(case):
    """Bytes of the inputs read once and the outputs written once, and the
    operations of the transforms: a convolution needs transforms of 2 n - 1
    points a line, a chirp-z two of n + m a line."""
    B, ny, nx, kind = case["batch"], case["ny"], case["nx"], case["kind"]
    pix = float(B * ny * nx)
    opix = float(B * case.get("my", ny) * case.get("mx", nx))

    def conv(comps):
        return comps * B * (2 * _fft_flops(ny, 2 * nx) + 2 * _fft_flops(2 * nx, 2 * ny))

    def chirp(comps, n_y, n_x, m_y, m_x):
        return comps * B * 2 * (_fft_flops(n_y, n_x + m_x) + _fft_flops(m_x, n_y + m_y))

    my, mx = case.get("my", 0), case.get("mx", 0)
    if kind == "rs":
        return {"bytes": pix * (8 + 4 + 8), "flops": conv(1)}
    if kind == "vrs":
        return {"bytes": pix * (16 + (8 if case["masked"] else 0) + 24), "flops": conv(3)}
    if kind == "czt":
        return {"bytes": pix * 8 + opix * 8, "flops": chirp(1, ny, nx, my, mx)}
    if kind == "vczt":
        return {"bytes": pix * 16 + 8.0 * ny * nx + opix * 24, "flops": chirp(3, ny, nx, my, mx)}
    if kind == "focus":
        return {"bytes": pix * 24 + opix * 24, "flops": chirp(3, ny, nx, my, mx)}
    if kind == "fourf":
        return {"bytes": pix * (8 + 4 + 4) + opix * (4 + 4 + 4),
                "flops": 2 * (conv(1) + chirp(1, ny, nx, my, mx) + chirp(1, my, mx, my, mx))}
    if kind == "spot":
        return {"bytes": pix * 32 + 16.0 * ny * nx + 4.0 * my * mx, "flops": 2 * chirp(1, ny, nx, my, mx)}
    # the distance's spectrum is part of a pass
    return {"bytes": pix * (16 + 16 + 24 + 16),
            "flops": 2 * conv(3) + _fft_flops(2 * ny, 2 * nx) + _fft_flops(2 * nx, 2 * ny)}


# ------------------------------------------------------------- in 64 bits --

def _response(X, Y, z, k):
    r = torch.sqrt(X ** 2 + Y ** 2 + z ** 2)
    return torch.exp(1j * k * r) * (z / (2 * math.pi * r ** 2)) * (1 / r - 1j * k)


def _convolve(fields, x, y, z):
    """Each field of (c, ny, nx) convolved with the impulse response at z > 0, cropped."""
    k = 2 * math.pi / WL
    ny, nx = len(y), len(x)

    def offsets(a):
        return torch.cat([a[0] - a.flip(0), a[1:] - a[0]])
    P = [1 << (2 * n - 2).bit_length() for n in (ny, nx)]
    H = _response(offsets(x)[None, :], offsets(y)[:, None], z, k)
    spec = torch.fft.fft2(H, s=P) * ((x[1] - x[0]) * (y[1] - y[0]))
    out = torch.fft.ifft2(torch.fft.fft2(fields, s=P) * spec)
    return out[..., ny - 1:2 * ny - 1, nx - 1:2 * nx - 1]


def _chirp_matrix(m, f1, f2, Dm, M):
    """The M x m matrix of one axis of the chirp-z transform (Bluestein's form)."""
    D1 = f1 + (M * Dm + f2 - f1) / (2 * M)
    D2 = f2 + (M * Dm + f2 - f1) / (2 * M)
    dW = (D2 - D1) / (M * Dm)
    dW -= round(dW)
    n = torch.arange(m, device="cuda", dtype=torch.float64)[None, :]
    q = torch.arange(M, device="cuda", dtype=torch.float64)[:, None]
    lf_ = q / M * (D2 - D1) + D1
    turns = -(D1 / Dm) * n - dW * (n * (q + 1) - q - 0.5) - lf_ * (0.5 - m / 2) / Dm
    a = 2 * math.pi * (turns - torch.round(turns))
    K = torch.complex(torch.cos(a), torch.sin(a))
    if M >= m:
        K[M - 1, 0] = 0     # the inverse chirp is one sample short there (wave_optics.py:404)
    return K


def _chirp(fields, n_y, n_x, xo, yo, Dm):
    My = _chirp_matrix(n_y, yo[0] + Dm / 2, yo[-1] + Dm / 2, Dm, len(yo))
    Mx = _chirp_matrix(n_x, xo[0] + Dm / 2, xo[-1] + Dm / 2, Dm, len(xo))
    return My @ fields @ Mx.T


def _free_chirp(fields, x, y, xo, yo, z):
    """Chirp-z propagation over z from (x, y) onto (xo, yo)."""
    k = 2 * math.pi / WL
    xt, yt, xot, yot = (torch.tensor(a, device="cuda") for a in (x, y, xo, yo))
    dx, dy = x[1] - x[0], y[1] - y[0]
    F, F0 = _response(xt[None, :], yt[:, None], z, k), _response(xot[None, :], yot[:, None], z, k)
    return _chirp(fields * F, len(y), len(x), xo, yo, WL * z / dx) * F0 * (z * dx * dy * WL)


def _retarder(ex, ey, eta, theta):
    ch, sh = torch.cos(eta / 2), torch.sin(eta / 2)
    c2, s2 = torch.cos(2 * theta), torch.sin(2 * theta)
    return (ch - 1j * sh * c2) * ex - 1j * sh * s2 * ey, -1j * sh * s2 * ex + (ch + 1j * sh * c2) * ey


def _focus(ex, ey, case, rows=(0, 1, 2)):
    """The high-NA lens and its focal field: the rows asked for of (Ex, Ey, Ez)."""
    x, y, xo, yo = _grids(case)
    r, f = _lens(case)
    X, Y = torch.tensor(x, device="cuda")[None, :], torch.tensor(y, device="cuda")[:, None]
    rho = torch.sqrt(X ** 2 + Y ** 2)
    s_max = r / math.sqrt(r ** 2 + f ** 2)
    q = rho ** 2 / r ** 2
    th, phi = rho / f, torch.atan2(Y, X)
    w = torch.where(q < 1, torch.sqrt(torch.abs(torch.cos(th)) / torch.abs(1 - q * s_max ** 2)), 0.0)
    ez = ex * X / rho + ey * Y / rho
    ct, st, c, s = torch.cos(th), torch.sin(th), torch.cos(phi), torch.sin(phi)
    R = [[ct * c * c + s * s, ct * c * s - s * c, -c * st],
         [s * ct * c - c * s, ct * s * s + c * c, -s * st],
         [st * c, st * s, ct]]
    Dm = f * WL * (len(x) - 1) / (2 * r)
    cte = -1j * s_max ** 2 / (f * WL)
    return [cte * _chirp(w * (R[i][0] * ex + R[i][1] * ey + R[i][2] * ez), len(y), len(x), xo, yo, Dm) for i in rows]


def _cis(a):
    return torch.complex(torch.cos(a), torch.sin(a))


def _norm_mse(u, target):
    I = u.real ** 2 + u.imag ** 2
    I = I / I.sum()
    return ((I - target) ** 2).sum() / I.numel()


def exact(case, seed):
    d = _data(case, seed)
    kind, B = case["kind"], case["batch"]
    x, y = _grids(case)[:2]
    xt, yt = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    k = 2 * math.pi / WL

    def entry(name, b):
        t = d[name]
        t = t[b] if B > 1 and t.dim() == 3 else t
        return t.to(torch.complex128) if t.is_complex() else t.to(torch.float64)

    def whole(entries):       # the entries of a batch as run() lays them out
        return torch.stack(entries) if B > 1 else entries[0]

    def vector_ez(ex, ey, z):
        r = torch.sqrt(xt[None, :] ** 2 + yt[:, None] ** 2 + z ** 2)
        return ex * xt[None, :] / r + ey * yt[:, None] / r

    def comps(entries):
        return tuple(whole([e[c] for e in entries]).to(torch.complex128) for c in range(3))

    if kind in ("rs", "vrs"):
        z = _distances(case)
        z = list(z) if isinstance(z, list) else [z] * B
    if kind == "rs":
        return whole([_convolve(entry("field", b) * _cis(entry("phase", b)), xt, yt, z[b]) for b in range(B)])
    if kind == "vrs":
        outs = []
        for b in range(B):
            ex, ey = entry("ex", b), entry("ey", b)
            if case["masked"]:
                ex, ey = _retarder(ex, ey, entry("eta", b), entry("theta", b))
                c, s = math.cos(d["alpha"]), math.sin(d["alpha"])
                ex, ey = c * (c * ex + s * ey), s * (c * ex + s * ey)
            outs.append([_convolve(e, xt, yt, z[b]) for e in (ex, ey, vector_ez(ex, ey, z[b]))])
        return comps(outs)
    if kind == "block":
        p = {n: d[n].to(torch.float64).requires_grad_(True) for n in TRAINED["block"]}
        ex = entry("ex", 0) * _cis(p["alpha"])
        ey = entry("ey", 0) * _cis(p["phi"])
        ex, ey, ez = (_convolve(e, xt, yt, d["z"]) for e in (ex, ey, vector_ez(ex, ey, d["z"])))
        ex, ey = _retarder(ex, ey, p["eta"], p["theta"])
        tgt = [t.to(torch.complex128) for t in d["target"]]
        loss = sum((((u.real ** 2 + u.imag ** 2) - (t.real ** 2 + t.imag ** 2)) ** 2).sum() / u.numel()
                   for u, t in zip((ex, ey, ez), tgt)) / 3
        loss.backward()
        return [loss.detach()] + [p[n].grad for n in TRAINED["block"]]
    xo, yo = _grids(case)[2:]
    r, f = _lens(case)
    pupil = ((xt[None, :] / r) ** 2 + (yt[:, None] / r) ** 2 < 1).to(torch.float64)
    lens = pupil * _cis(-k * (xt[None, :] ** 2 + yt[:, None] ** 2) / (2 * f))
    if kind == "czt":
        return whole([_free_chirp(entry("field", b) * lens, x, y, xo, yo, f) for b in range(B)])
    if kind == "vczt":
        outs = []
        for b in range(B):
            ex, ey = _retarder(entry("ex", b), entry("ey", b), entry("eta", b), entry("theta", b))
            ez = vector_ez(ex, ey, f) * f / torch.sqrt(xt[None, :] ** 2 + yt[:, None] ** 2 + f ** 2)
            outs.append([_free_chirp(e, x, y, xo, yo, f) for e in (ex, ey, ez)])
        return comps(outs)
    if kind == "focus":
        return comps([_focus(entry("ex", b) * _cis(entry("alpha", b)), entry("ey", b) * _cis(entry("phi", b)), case)
                      for b in range(B)])
    losses, grads = [], []
    for b in range(B):
        p = {n: entry(n, b).requires_grad_(True) for n in TRAINED[kind]}
        if kind == "fourf":
            u = _convolve(entry("field", b) * _cis(p["p1"]), xt, yt, f) * lens
            u = _free_chirp(u, x, y, xo, yo, f) * _cis(p["p2"])
            u = _free_chirp(u, xo, yo, xo, yo, f)
        else:
            ex, ey = _retarder(entry("ex", b), entry("ey", b), p["eta"], p["theta"])
            u = _focus(ex * _cis(p["alpha"]), ey * _cis(p["phi"]), case, rows=(2,))[0]
        loss = _norm_mse(u, entry("target", b)) / B
        loss.backward()
        losses.append(loss.detach())
        grads.append([p[n].grad for n in TRAINED[kind]])
    return [sum(losses)] + [whole([g[i] for g in grads]) for i in range(len(TRAINED[kind]))]
