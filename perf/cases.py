"""The work that programs have this framework do, as cases to be timed.

Every case goes through the package's public Python entry points, with the
force parameters of the reference's rules (rs = 1.25 cells, rcut = 4.5 rs,
softening 0.03 mean spacings) and seeded particle sets of the three kinds the
repository's workloads use: a jittered grid, a Zel'dovich field, and a uniform
background with NFW halos (and Plummer spheres for the batched boxes).

    listed()            the cases
    draw(rng)           one more of the same ranges
    prepare(case, seed) inputs on the device (or the host, where the entry
                        point takes host arrays) and the context a program keeps
    run(state)          one pass through the entry point, and its outputs
    work(case)          bytes and operations the pass cannot do without
    exact(case, seed)   the outputs in 64 bits, from plain torch

The split-precision pass forms its pair forces and sums in single precision
and hands them out in 64-bit arrays; a program that chose it keeps
accelerations (and, as a Gadget-2 snapshot does, positions and velocities)
in single precision, so those cases return float32.  The FP64 passes, the PM
force and the direct sum return float64.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry

ph = entry.load_package()
from photons_gb300 import ics  # noqa: E402  (the package is loaded above)

CELL = 1.953125  # mean particle spacing of the 256^3 / L = 500 workload; boxes scale with the particle count
_stream = None


def listed():
    return [
        # the smallest call: the 16^3 box of the smoke run, launches and latency count
        dict(name="pass_grid16", kind="pass", dist="grid", n=4096, leaf=16, prec="fp32", theta=0.5),
        # the 32^3 grid workload (leaf 16)
        dict(name="pass_grid32", kind="pass", dist="grid", n=32768, leaf=16, prec="fp32", theta=0.5),
        # an ordinary clustered box, particle count no power of two
        dict(name="pass_nfw64", kind="pass", dist="nfw", n=250047, leaf=24, prec="fp32", theta=0.5),
        # the 128^3 halo workload at its autotuned leaf size
        dict(name="pass_nfw128", kind="pass", dist="nfw", n=2097152, leaf=24, prec="fp32", theta=0.5),
        # the headline: 256^3 Zel'dovich at leaf 64
        dict(name="pass_zel256", kind="pass", dist="zel", n=16777216, leaf=64, prec="fp32", theta=0.5),
        # the reference's arithmetic on halos, odd particle count
        dict(name="pass64_nfw48", kind="pass", dist="nfw", n=110591, leaf=16, prec="fp64", theta=0.5),
        # the reference's arithmetic on a near-uniform field
        dict(name="pass64_zel96", kind="pass", dist="zel", n=884736, leaf=64, prec="fp64", theta=0.5),
        # the reference driver's step on its globals (host part[]), the demo run's theta and MAXLEAF, PM beside it
        dict(name="driver_grid32", kind="driver", dist="grid", n=32768, leaf=8, mesh=32, theta=0.4),
        # many independent boxes in one pass (host arrays), leaf 32
        dict(name="boxes40", kind="boxes", boxes=40, nmin=4096, nmax=32768, leaf=32),
        # a kick-drift-kick step with both force halves on resident arrays
        dict(name="kdk_zel128", kind="kdk", dist="zel", n=2097152, leaf=48, mesh=128, theta=0.5),
        # the long-range force alone, host arrays
        dict(name="pm_nfw100", kind="pm", dist="nfw", n=1000000, mesh=128),
        # the FP64 direct sum over a sample of targets: what the leaf-size autotuner scores its candidates with
        dict(name="direct_nfw64", kind="direct", dist="nfw", n=262144, targets=2000),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _leaf(n, sizes, rng):
    """A leaf size whose balanced tree has leaves filled to at least 0.65:
    the reference's rule allows 2N/MAXLEAF leaves and no more."""
    sizes = list(sizes)
    rng.shuffle(sizes)
    for s in sizes:
        if n / 2.0 ** math.ceil(math.log2(n / s)) / s >= 0.65:
            return s
    return max(sizes, key=lambda s: n / 2.0 ** math.ceil(math.log2(n / s)) / s)


def _count(rng, dist, lo, hi):
    n = _loguniform(rng, lo, hi)
    return n if dist == "nfw" else max(round(lo ** (1 / 3)), round(n ** (1 / 3))) ** 3


def draw(rng):
    kind = rng.choice(["pass", "pass", "pass", "pass", "pass", "pass64", "pass64", "driver", "boxes", "kdk", "pm",
                       "direct"])
    dist = rng.choice(["grid", "zel", "nfw"])
    theta = rng.choice([0.4, 0.5])
    if kind == "pass":
        n = _count(rng, dist, 4096, 1500000 if dist == "nfw" else 10000000)
        # the leaf sizes the autotuner scores; near-uniform boxes run fastest from 48 up, halos below
        leaf = _leaf(n, [16, 24, 32, 48, 64], rng)
        return dict(kind="pass", dist=dist, n=n, leaf=leaf, prec="fp32", theta=theta)
    if kind == "pass64":
        n = _count(rng, dist, 4096, 80000 if dist == "nfw" else 600000)
        return dict(kind="pass", dist=dist, n=n, leaf=_leaf(n, [8, 16, 32, 64], rng), prec="fp64", theta=theta)
    if kind == "driver":
        n = _count(rng, "grid", 4096, 60000)
        return dict(kind="driver", dist="grid", n=n, leaf=_leaf(n, [8, 16], rng), mesh=2 * rng.randint(8, 20),
                    theta=theta)
    if kind == "boxes":
        lo = _loguniform(rng, 1024, 8192)
        return dict(kind="boxes", boxes=rng.randint(4, 48), nmin=lo, nmax=lo * rng.randint(2, 4),
                    leaf=rng.choice([16, 32]))
    if kind == "kdk":
        n = _count(rng, dist, 20000, 1500000)
        return dict(kind="kdk", dist=dist, n=n, leaf=_leaf(n, [24, 32, 48, 64], rng),
                    mesh=2 * max(8, round(n ** (1 / 3) / 2)), theta=theta)
    if kind == "pm":
        n = _count(rng, dist, 10000, 1000000)
        return dict(kind="pm", dist=dist, n=n, mesh=2 * rng.randint(16, 64))
    n = _count(rng, dist, 10000, 262144)
    return dict(kind="direct", dist=dist, n=n, targets=_loguniform(rng, 100, 2000))


# ---- inputs ------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(shape, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(shape, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _iso(m, g):
    v = _randn((m, 3), g)
    return v / v.norm(dim=1, keepdim=True)


def _wrap(pos, side):
    pos = torch.remainder(pos, side)
    return torch.where(pos >= side, pos - side, pos).contiguous()


def _lattice(nside, dx):
    i = (torch.arange(nside, device="cuda", dtype=torch.float64) + 0.5) * dx
    return torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3)


def _grid(n, side, g):
    nside = round(n ** (1 / 3))
    dx = side / nside
    return _wrap(_lattice(nside, dx) + 0.3 * dx * _randn((n, 3), g), side)


def _zeldovich(n, side, g):
    """Lattice displaced by a Gaussian field with P(k) ~ k^-2, rms half a spacing."""
    nside = round(n ** (1 / 3))
    dx = side / nside
    dk = torch.fft.rfftn(_randn((nside,) * 3, g))
    k1 = 2 * math.pi * torch.fft.fftfreq(nside, d=dx, device="cuda", dtype=torch.float64)
    kz = 2 * math.pi * torch.fft.rfftfreq(nside, d=dx, device="cuda", dtype=torch.float64)
    ks = (k1[:, None, None], k1[None, :, None], kz[None, None, :])
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    k2[0, 0, 0] = 1.0
    dk = dk / k2 ** 1.5  # sqrt(P) = 1/k, and the 1/k^2 of the displacement
    dk[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * k * dk, s=(nside,) * 3).reshape(-1) for k in ks], -1)
    psi *= 0.5 * dx / torch.sqrt((psi ** 2).sum(1).mean())
    return _wrap(_lattice(nside, dx) + psi, side)


def _nfw(n, side, g):
    """Half uniform, half in NFW halos (concentration 5-15, masses over two
    decades, one halo per 32768 particles)."""
    nhalo = max(1, round(n / 32768))
    n_bg = n // 2
    n_halo = n - n_bg
    w = 10.0 ** (2.0 * _rand((nhalo,), g))
    edge = torch.floor(torch.cumsum(w, 0) / w.sum() * n_halo).long()
    edge[-1] = n_halo
    counts = torch.diff(edge, prepend=edge.new_zeros(1))
    conc = 5.0 + 10.0 * _rand((nhalo,), g)
    centres = side * _rand((nhalo, 3), g)
    h = torch.repeat_interleave(torch.arange(nhalo, device="cuda"), counts, output_size=n_halo)
    rvir = (3.0 * counts.double() / (4.0 * math.pi * 200.0 * (n / side ** 3))) ** (1.0 / 3.0)
    c = conc[h]
    u = _rand((n_halo,), g) * (torch.log1p(c) - c / (1.0 + c))
    lo, hi = torch.zeros_like(c), c.clone()
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        big = torch.log1p(mid) - mid / (1.0 + mid) > u
        hi = torch.where(big, mid, hi)
        lo = torch.where(big, lo, mid)
    r = 0.5 * (lo + hi) / c * rvir[h]
    return _wrap(torch.cat([side * _rand((n_bg, 3), g), centres[h] + r[:, None] * _iso(n_halo, g)]), side)


def _plummer(n, side, g):
    """70 % in a Plummer sphere of scale 0.05 sides, the rest uniform."""
    m = int(round(0.7 * n))
    u = 0.97 * _rand((m,), g) + 1e-9  # radii within half a side
    r = 0.05 * side / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    return _wrap(torch.cat([0.5 * side + r[:, None] * _iso(m, g), side * _rand((n - m, 3), g)]), side)


def _side(n):
    return CELL * n ** (1 / 3)


def _positions(case, seed):
    make = {"grid": _grid, "zel": _zeldovich, "nfw": _nfw}[case["dist"]]
    return make(case["n"], _side(case["n"]), _gen(seed))


def _params(case):
    n = case["n"]
    mesh = case.get("mesh") or max(1, round(n ** (1 / 3)))
    return ics.force_params(n, _side(n), mesh, theta=case.get("theta", 0.5), maxleaf=case.get("leaf", 16))


def _boxes(case, seed):
    rng = np.random.default_rng(case["boxes"])  # the boxes' sizes are the case's, the particles the seed's
    g = _gen(seed)
    out = []
    for _ in range(case["boxes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        side = rng.uniform(20.0, 100.0)
        p = ics.force_params(n, side, max(1, round(n ** (1 / 3))), maxleaf=case["leaf"])
        out.append((_plummer(n, side, g), p))
    return out


def _context():
    """A context on the program's torch stream, so that the pass and the
    program's own kernels are ordered."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    _stream.wait_stream(torch.cuda.current_stream())
    fp = ph.ForcePass(0)
    fp.set_stream(_stream.cuda_stream)
    return fp


def prepare(case, seed):
    kind = case["kind"]
    if kind == "boxes":
        return dict(kind=kind, fp=ph.ForcePass(0), boxes=[(x.cpu().numpy(), p) for x, p in _boxes(case, seed)])
    p = _params(case)
    pos = _positions(case, seed)
    s = dict(kind=kind, p=p, n=case["n"])
    if kind == "pass":
        s.update(pos=pos, acc=torch.empty_like(pos), prec=ph.FP64 if case["prec"] == "fp64" else ph.FP32_SPLIT)
    elif kind == "kdk":
        s.update(pos=pos, vel=_randn(pos.shape, _gen(seed + 1)), acc=torch.zeros_like(pos),
                 acc_pm=torch.zeros_like(pos), mesh=case["mesh"], dd=5e-4 * CELL)
    elif kind == "driver":
        s.update(pos=pos.cpu().numpy(), ref=ph.Reference(), mesh=case["mesh"])
    elif kind == "pm":
        s.update(pos=pos.cpu().numpy(), fp=ph.ForcePass(0), mesh=case["mesh"])
    elif kind == "direct":
        tgt = np.random.default_rng(seed).choice(case["n"], case["targets"], replace=False).astype(np.int32)
        s.update(pos=pos.cpu().numpy(), targets=tgt)
    if kind in ("pass", "kdk"):
        s["fp"] = _context()
    if kind == "kdk":
        # the forces at the start, as a program's first call makes them, and a
        # kick of a few thousandths of the velocity
        with torch.cuda.stream(_stream):
            _kdk(s, 0.0, 0.0)
            s["dkh"] = 2e-3 / float((s["acc"] + s["acc_pm"]).pow(2).mean().sqrt())
    return s


def _kdk(s, dkh, dd):
    s["fp"].kdk_step_pm_device(s["pos"].data_ptr(), s["vel"].data_ptr(), s["acc"].data_ptr(), s["acc_pm"].data_ptr(),
                               s["n"], s["p"], s["mesh"], dkh, dd)


def run(s):
    kind = s["kind"]
    if kind == "pass":
        with torch.cuda.stream(_stream):
            s["fp"].run_device(s["pos"].data_ptr(), s["acc"].data_ptr(), s["n"], s["p"], precision=s["prec"])
            return s["acc"].float() if s["prec"] == ph.FP32_SPLIT else s["acc"]
    if kind == "kdk":
        with torch.cuda.stream(_stream):
            _kdk(s, s["dkh"], s["dd"])
            return [s[k].float() for k in ("pos", "vel", "acc", "acc_pm")]
    if kind == "boxes":
        return [a.astype(np.float32) for a in s["fp"].run_boxes(s["boxes"])]
    if kind == "driver":
        ref = s["ref"]
        ref.setup(s["pos"], s["p"])
        ref.force_pass(pm_nside=s["mesh"])
        part = ref.part()
        ref.deconstruct()
        return [part["pos"], part["acc"], part["acc_pm"]]
    if kind == "pm":
        return s["fp"].pm_force(s["pos"], s["p"], s["mesh"])
    return ph.direct_sum(s["pos"], s["p"], s["targets"])


# ---- what a pass cannot do without -----------------------------------------

# particles within rcut (5.625 cells) of a particle at mean density, each
# symmetric pair once, 36 operations a pair; clustered sets have more
_PAIR_FLOPS = 0.5 * (4.0 / 3.0) * math.pi * 5.625 ** 3 * 36


def _pm_work(n, mesh):
    cells = mesh ** 3
    # positions in, accelerations out; two FFTs of 2.5 N log2 N, the Green's product, three gradients, two CIC passes
    return n * 48.0, 2 * 2.5 * cells * math.log2(cells) + 20.0 * cells + 60.0 * n


def work(case):
    kind = case["kind"]
    if kind == "boxes":
        n = case["boxes"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        return dict(bytes=n * 48.0, flops=n * _PAIR_FLOPS)
    n = case["n"]
    if kind == "pass":
        return dict(bytes=n * 48.0, flops=n * _PAIR_FLOPS)
    if kind in ("kdk", "driver"):
        b, f = _pm_work(n, case["mesh"])
        # positions and velocities read and written, both accelerations read and written
        return dict(bytes=n * (192.0 if kind == "kdk" else 96.0), flops=n * _PAIR_FLOPS + f)
    if kind == "pm":
        b, f = _pm_work(n, case["mesh"])
        return dict(bytes=b, flops=f)
    # every source's distance is looked at; those within 2 rcut get a force
    near = min(1.0, (4.0 / 3.0) * math.pi * 11.25 ** 3 / n)
    return dict(bytes=n * 24.0 + case["targets"] * 28.0, flops=case["targets"] * n * (9.0 + 36.0 * near))


# ---- the outputs in 64 bits -------------------------------------------------

def _split_sum(pos, p, targets, rmax=None, images=False):
    """Direct sum of the short-range force: m g(r/2rs) dx / max(r, eps)^3,
    g(u) = erfc(u) + (2/sqrt(pi)) u exp(-u^2), nearest images, or all 27."""
    side = p["boxsize"]
    shifts = [(0, 0, 0)]
    if images:
        shifts = [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
    out = torch.zeros((len(targets), 3), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 26) // pos.shape[0])
    for a in range(0, len(targets), step):
        t = pos[targets[a:a + step]]
        for sh in shifts:
            d = pos[None, :, :] + side * torch.tensor(sh, device="cuda", dtype=torch.float64) - t[:, None, :]
            if not images:
                d = d - side * torch.round(d / side)
            r = d.norm(dim=2)
            u = r / (2.0 * p["rs"])
            f = p["mass"] * (torch.special.erfc(u) + 2.0 / math.sqrt(math.pi) * u * torch.exp(-u * u))
            f = f / torch.clamp(r, min=p["eps"]) ** 3
            f = torch.where((r > 0) if rmax is None else (r > 0) & (r <= rmax), f, torch.zeros_like(f))
            out[a:a + step] += torch.einsum("ts,tsc->tc", f, d)
    return out


def _pm_exact(pos, p, mesh):
    """CIC deposit, the Green's function, a 4-point gradient and CIC
    interpolation; pi is the single-precision 3.1415926 of the reference's
    Fortran."""
    pi = float(np.float32(3.1415926))
    N, L = mesh, p["boxsize"]
    c = torch.floor(pos * (N / L)).long()
    w = (pos - (c.double() + 0.5) * (L / N)) * (N / L)
    cn = torch.where(w > 0, c + 1, c - 1) % N
    c = c % N
    w = w.abs()
    corners = []
    for bits in range(8):
        up = [(bits >> d) & 1 for d in range(3)]
        cell = [cn[:, d] if up[d] else c[:, d] for d in range(3)]
        wt = [w[:, d] if up[d] else 1.0 - w[:, d] for d in range(3)]
        corners.append(((cell[0] * N + cell[1]) * N + cell[2], wt[0] * wt[1] * wt[2]))
    rho = torch.zeros(N ** 3, device="cuda", dtype=torch.float64)
    for at, wt in corners:
        rho.index_add_(0, at, p["mass"] * wt)
    rho = rho.reshape(N, N, N) * (N / L) ** 3
    a = torch.arange(N, device="cuda", dtype=torch.float64)
    a = torch.where(a > N // 2, a - N, a)
    b = torch.arange(N // 2 + 1, device="cuda", dtype=torch.float64)
    sinc = lambda q: torch.where(q == 0, torch.ones_like(q), torch.sin(pi * q / N) / (pi * q / N))  # noqa: E731
    k2 = a[:, None, None] ** 2 + a[None, :, None] ** 2 + b[None, None, :] ** 2
    win = sinc(a)[:, None, None] * sinc(a)[None, :, None] * sinc(b)[None, None, :]
    pref = L * L / (pi * float(N) ** 3)
    green = pref * torch.exp(-k2 * (2 * pi * p["rs"] / L) ** 2) / win ** 4 / k2
    green[0, 0, 0] = pref
    psi = torch.fft.irfftn(torch.fft.rfftn(rho) * green, s=(N, N, N)) * float(N) ** 3
    h = 0.5 * N / L
    out = torch.zeros_like(pos)
    for d in range(3):
        grad = (4.0 / 3.0) * h * (torch.roll(psi, -1, d) - torch.roll(psi, 1, d))
        grad = (grad - h / 6.0 * (torch.roll(psi, -2, d) - torch.roll(psi, 2, d))).reshape(-1)
        for at, wt in corners:
            out[:, d] += wt * grad[at]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "boxes":
        return [_split_sum(x, p, torch.arange(len(x), device="cuda")) for x, p in _boxes(case, seed)]
    if kind == "pass" and case["n"] <= 120000:
        pos = _positions(case, seed)
        return _split_sum(pos, _params(case), torch.arange(case["n"], device="cuda"), images=case["n"] <= 8192)
    if kind == "pm":
        return _pm_exact(_positions(case, seed), _params(case), case["mesh"])
    if kind == "direct":
        p = _params(case)
        tgt = np.random.default_rng(seed).choice(case["n"], case["targets"], replace=False)
        return _split_sum(_positions(case, seed), p, torch.from_numpy(tgt).cuda(), rmax=2.0 * p["rcut"])
    # larger passes take too long; the driver's outputs come in its tree's order, a step's after earlier ones
    return None
