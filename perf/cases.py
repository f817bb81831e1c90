"""The measured work of this library: solves as a user's program makes them.

A case is one call of the public Python front-end (``flups_b200.pyflups``,
the same C symbols a FLUPS program links) on a solver that was set up before:
``Solver.solve`` on CUDA or host arrays, or ``Solver.solve_batch``.  Grids are
given by their number of points per direction, boundary conditions by two
letters per direction (U unbounded, P periodic, E even, O odd; ``--`` for the
missing direction of a plane problem), data cell- or node-centred, transforms
in FP32 or FP64 (the library's default), scalar or three-component ROT solves
with the spectral curl.

Sizes are those FFT users choose: transform lengths whose prime factors are
13 or less (the lengths FFTW's manual recommends), even and odd, powers of two
among them.
"""
import math

import numpy as np
import torch

from flups_b200 import pyflups as pf

_BC = {"U": pf.BoundaryType.UNB, "P": pf.BoundaryType.PER, "E": pf.BoundaryType.EVEN, "O": pf.BoundaryType.ODD,
       "-": pf.BoundaryType.NONE}


def _case(name, nx, ny, nz, bc, center, green, bits, kind="device", batch=1, rot=False):
    c = {"nx": nx, "ny": ny, "nz": nz, "bc": bc, "center": center, "green": green, "bits": bits, "kind": kind,
         "batch": batch, "rot": rot}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small free-space solve inside a time step: five short launches
        _case("unb64_fp32", 64, 64, 64, "UUUUUU", "cell", "CHAT_2", 32),
        # free space at the default precision, an ordinary production grid
        _case("unb256_fp64", 256, 256, 256, "UUUUUU", "cell", "HEJ_4", 64),
        # the largest free-space grid of the benchmark
        _case("unb512_fp32", 512, 512, 512, "UUUUUU", "cell", "HEJ_2", 32),
        # free space on a grid that is no power of two, default precision
        _case("unb200_fp64", 200, 200, 200, "UUUUUU", "cell", "HEJ_2", 64),
        # a flow over a wall: symmetry plane below, open above and around
        _case("wall_160x120x100_fp32", 160, 120, 100, "UUUUOU", "cell", "HEJ_4", 32),
        # node-centred data in free space: odd extents, rows of any alignment
        _case("node_unb_145x121x101_fp32", 145, 121, 101, "UUUUUU", "node", "HEJ_2", 32),
        # the benchmark's node-centred mixed problem: even/odd walls, periodic span, open height
        _case("node_eo_per_unb_513x257x257_fp32", 513, 257, 257, "EOPPUU", "node", "HEJ_4", 32),
        # a closed box: Dirichlet, Neumann and periodic faces (pressure solves)
        _case("box_250x150x180_fp64", 250, 150, 180, "OOEEPP", "cell", "CHAT_2", 64),
        # a plane problem: periodic along x, open along y
        _case("plane_1500x700_fp64", 1500, 700, 1, "PPUU--", "cell", "HEJ_2", 64),
        # velocity from vorticity (vortex methods): three components, spectral curl
        _case("rot384_fp32", 384, 384, 384, "UUUUUU", "cell", "HEJ_4", 32, rot=True),
        # many right-hand sides of one solver in one call
        _case("batch64_unb128_fp32", 128, 128, 128, "UUUUUU", "cell", "HEJ_2", 32, kind="batch", batch=64),
        # the reference's own calling convention: host arrays in and out, the call returns with the result
        _case("host_unb160_fp64", 160, 160, 160, "UUUUUU", "cell", "HEJ_2", 64, kind="host"),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi, node):
    """A log-uniform extent in [lo, hi] whose number of intervals has prime factors up to 13."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if _smooth(n - 1 if node else n):
            return n


def draw(rng):
    fam = rng.choice(["unb", "unb", "wall", "node_unb", "node_mixed", "box", "channel", "plane", "rot", "batch", "host"])
    bits = rng.choice([32, 64])
    node = fam.startswith("node") or (fam in ("box", "channel", "wall") and rng.random() < 0.3)
    center = "node" if node else "cell"
    green = rng.choice(["HEJ_2", "HEJ_4", "CHAT_2"])
    if fam in ("unb", "node_unb"):
        n = [_size(rng, 24, 400, node) for _ in range(3)]
        return _case(None, *n, "UUUUUU", center, green, bits)
    if fam == "wall":
        n = [_size(rng, 24, 256, node) for _ in range(3)]
        bc = rng.choice(["UUUUOU", "UUUUEU", "UUUUUO", "EUUUUU"])
        return _case(None, *n, bc, center, green, bits)
    if fam == "node_mixed":
        n = [_size(rng, 33, 513, True), _size(rng, 33, 321, True), _size(rng, 33, 321, True)]
        return _case(None, *n, rng.choice(["EOPPUU", "OEPPUU", "EEPPUU", "OOPPUU"]), "node", green, bits)
    if fam == "box":
        n = [_size(rng, 24, 400, node) for _ in range(3)]
        bc = "".join(rng.choice(["OO", "EE", "PP", "EO", "OE"]) for _ in range(3))
        return _case(None, *n, bc, center, "CHAT_2", bits)
    if fam == "channel":
        n = [_size(rng, 24, 400, node) for _ in range(3)]
        return _case(None, *n, rng.choice(["PPPPUU", "PPUUPP", "UUPPPP", "EEPPUU", "PPOOUU"]), center, green, bits)
    if fam == "plane":
        return _case(None, _size(rng, 64, 2048, False), _size(rng, 64, 1024, False), 1, "PPUU--", "cell", green, bits)
    if fam == "rot":
        n = [_size(rng, 24, 256, False) for _ in range(3)]
        return _case(None, *n, "UUUUUU", "cell", rng.choice(["HEJ_2", "HEJ_4"]), bits, rot=True)
    if fam == "batch":
        n = [_size(rng, 24, 128, False) for _ in range(3)]
        return _case(None, *n, "UUUUUU", "cell", green, bits, kind="batch", batch=rng.randint(2, 16))
    n = [_size(rng, 32, 200, False) for _ in range(3)]
    return _case(None, *n, "UUUUUU", "cell", green, bits, kind="host")


# ------------------------------------------------------------------ geometry
def _dims(case):
    return [case["nx"], case["ny"], case["nz"]]


def _bcs(case):
    return [case["bc"][0:2], case["bc"][2:4], case["bc"][4:6]]


def _h(case):
    """One spacing for every direction (the regularised kernels ask for it); the longest side is 1."""
    node = case["center"] == "node"
    return 1.0 / max(n - 1 if node and n > 1 else n for n in _dims(case))


def _rhs(case, seed, dev):
    """Seeded Gaussian blobs (vorticity or sources of compact support), [batch * lda][z][y][x], FP64."""
    rng = np.random.default_rng(seed)
    node, h = case["center"] == "node", _h(case)
    n = _dims(case)
    shape = [n[2], n[1], n[0]]
    ext = [n[d] * h for d in range(3)]
    xs = [torch.arange(n[d], dtype=torch.float64, device=dev) * h + (0.0 if node else 0.5 * h) for d in range(3)]
    size = min(e for e, m in zip(ext, n) if m > 1)
    lda = 3 if case["rot"] else 1
    out = torch.zeros([case["batch"] * lda] + shape, dtype=torch.float64, device=dev)
    for i in range(out.shape[0]):
        for _ in range(4):
            g = []
            sig = max(rng.uniform(0.05, 0.1) * size, 1.5 * h)
            amp = rng.uniform(0.5, 1.0) * (1 if rng.random() < 0.5 else -1)
            for d in range(3):
                c = rng.uniform(0.35, 0.65) * ext[d]
                g.append(torch.exp(-((xs[d] - c) / sig) ** 2) if n[d] > 1 else torch.ones_like(xs[d]))
            out[i] += amp * g[2][:, None, None] * g[1][None, :, None] * g[0][None, None, :]
    if node:
        for d, b in enumerate(_bcs(case)):
            if b == "PP":  # the last node is the first one's image
                out.select(3 - d, n[d] - 1).copy_(out.select(3 - d, 0))
    return out


# ------------------------------------------------------------------ the call
def prepare(case, seed):
    n, h = _dims(case), _h(case)
    node = case["center"] == "node"
    lda = 3 if case["rot"] else 1
    topo = pf.Topology(0, lda, n)
    length = [h * (m - 1 if node and m > 1 else m) for m in n]
    center = pf.CenterType.NODE_CENTER if node else pf.CenterType.CELL_CENTER
    solver = pf.Solver(topo, [[_BC[b[0]], _BC[b[1]]] for b in _bcs(case)], [h] * 3, length,
                       order_diff=pf.DiffType.SPE if case["rot"] else pf.DiffType.NOD, center_type=[center] * 3)
    solver.set_green_type(pf.GreenType[case["green"]])
    if case["bits"] == 32:
        solver.set_precision(32)
    solver.set_stream(torch.cuda.current_stream())
    solver.setup()
    rhs = _rhs(case, seed, "cuda")
    if case["kind"] == "host":
        rhs = rhs.cpu().pin_memory()
        field = torch.zeros(rhs.shape, dtype=torch.float64).pin_memory()
    else:
        field = torch.zeros_like(rhs)
        solver.set_async(True)  # a GPU program's calls: queued on its stream
    return {"case": case, "topo": topo, "solver": solver, "rhs": rhs, "field": field}


def run(state):
    case, solver = state["case"], state["solver"]
    kind = pf.SolverType.ROT if case["rot"] else pf.SolverType.STD
    if case["kind"] == "batch":
        return solver.solve_batch(state["field"], state["rhs"], case["batch"], kind)
    return solver.solve(state["field"], state["rhs"], kind)


# ------------------------------------------------------------------ sizes and tolerances
def _line(n, b, node):
    """Points of one direction's transform line as a real sequence of the given period."""
    m = n - 1 if node else n
    if b == "--":
        return 1
    if b == "PP":
        return m
    if b in ("UU", "EE", "OO"):
        return 2 * m
    return 4 * m  # even/odd walls, or one wall and one open end


def work(case):
    n, node, bcs = _dims(case), case["center"] == "node", _bcs(case)
    comps = case["batch"] * (3 if case["rot"] else 1)
    es = case["bits"] // 8
    # the real spectrum of the kernel, one value per distinct wave number
    green = 1
    for m, b in zip(n, bcs):
        ln = _line(m, b, node)
        green *= 1 if b == "--" else ln // 2 + 1
    flops, ext = 0.0, list(n)
    for d in range(3):
        ln = _line(n[d], bcs[d], node)
        if ln == 1:
            continue
        lines = 1
        for e in range(3):
            if e != d:
                lines *= ext[e]
        # forward and inverse real transforms of the line (2.5 L log2 L each)
        flops += 2 * 2.5 * lines * ln * math.log2(max(ln, 2)) * comps
        if "U" in bcs[d]:
            ext[d] = 2 * n[d]
    return {"bytes": 16 * n[0] * n[1] * n[2] * comps + es * green, "flops": int(flops)}


def tolerance(case):
    # four times the largest error against exact() over the ranges above: 2.0e-7 (FP32), 6.0e-16 (FP64)
    return {"rel": 8e-7} if case["bits"] == 32 else {"rel": 2.5e-15}


# ------------------------------------------------------------------ 64-bit values
def _extend(f, d, b, node):
    """The line of direction d (tensor axis 3 - d) as one period of the sequence it stands for."""
    ax = 3 - d
    n = f.shape[ax]
    if b == "--":
        return f
    if node:
        n1 = n - 1
        if b == "PP":
            return f.narrow(ax, 0, n1)
        if b == "UU":
            z = list(f.shape)
            z[ax] = n1 - 1
            return torch.cat([f, torch.zeros(z, dtype=f.dtype, device=f.device)], ax)
        f = f.clone()
        if b[0] == "O":
            f.narrow(ax, 0, 1).zero_()
        if b[1] == "O":
            f.narrow(ax, n1, 1).zero_()
        inner = f.narrow(ax, 1, n1 - 1).flip(ax)  # nodes n1 - 1 .. 1
        if "U" not in b:
            if b[0] == b[1]:
                return torch.cat([f, inner if b[0] == "E" else -inner], ax)
            s = -1.0 if b == "EO" else 1.0
            half = torch.cat([f.narrow(ax, 0, n1), s * f.narrow(ax, 1, n1).flip(ax)], ax)
            return torch.cat([half, -half], ax)
        # one symmetric face, one open face: the image about the symmetric face, zeros to 4 n1 points
        s = 1.0 if "E" in b else -1.0
        z = list(f.shape)
        z[ax] = 2 * n1 - 1
        pad = torch.zeros(z, dtype=f.dtype, device=f.device)
        img = s * f.narrow(ax, 1, n1).flip(ax)  # nodes n1 .. 1 reflected: positions -n1 .. -1
        if b[1] == "U":
            return torch.cat([f, pad, img], ax)
        img = s * f.narrow(ax, 0, n1).flip(ax)  # positions n1 + 1 .. 2 n1
        return torch.cat([f, img, pad], ax)
    if b == "PP":
        return f
    if b == "UU":
        return torch.cat([f, torch.zeros_like(f)], ax)
    r = f.flip(ax)
    if "U" not in b:
        if b == "EE":
            return torch.cat([f, r], ax)
        if b == "OO":
            return torch.cat([f, -r], ax)
        if b == "EO":
            return torch.cat([f, -r, -f, r], ax)
        return torch.cat([f, r, -f, -r], ax)
    s = 1.0 if "E" in b else -1.0
    z = torch.zeros_like(f)
    if b[1] == "U":
        return torch.cat([f, z, z, s * r], ax)
    return torch.cat([f, s * r, z, z], ax)


def _length_axis(shape, d):
    s = [1, 1, 1, 1]
    s[3 - d] = shape
    return s


def _kernel_regular(green, r, sig, hprod):
    """Free-space kernels of the three-dimensional Laplacian (Gaussian-regularised HEJ, or -1 / 4 pi r)."""
    rho = r / sig
    safe = torch.where(r > 0, r, torch.ones_like(r))
    s2 = math.sqrt(2.0)
    if green == "CHAT_2":
        g = -1.0 / (4 * math.pi * safe)
        g0 = -0.5 * (1.5 * hprod / (2 * math.pi)) ** (2.0 / 3.0) / hprod
    elif green == "HEJ_2":
        g = -torch.erf(rho / s2) / (4 * math.pi * safe)
        g0 = -s2 / (4.0 * sig * math.pi ** 1.5)
    else:
        g = -(torch.erf(rho / s2) + rho * torch.exp(-0.5 * rho * rho) / math.sqrt(2 * math.pi)) / (4 * math.pi * safe)
        g0 = -3.0 * s2 / (8.0 * sig * math.pi ** 1.5)
    return torch.where(r > 0, g, torch.full_like(g, g0))


def _one_minus_erf(x):
    """1 - erf(x) as the library states it: erf rounded to the nearest double first."""
    return torch.where(x >= 2.0, 1.0 - (1.0 - torch.special.erfc(x)), 1.0 - torch.erf(x))


def _kernel_line(green, k, r, sig, k_cut):
    """Kernels of (d^2/dx^2 - k^2) on an open line at distance r; wave numbers up to k_cut count as zero
    (the library's rule: a fifth of the sum of the closed directions' base wave numbers)."""
    s2 = math.sqrt(2.0)
    pos = k > k_cut
    ks = torch.where(pos, k, torch.ones_like(k))
    if green == "CHAT_2":
        return torch.where(pos, -0.5 * torch.exp(-ks * r) / ks, 0.5 * r + 0 * k)
    s, rho = ks * sig, r / sig
    near = s * rho <= 100.0
    a = _one_minus_erf((s - rho) / s2) * torch.exp(-s * rho)
    b = _one_minus_erf((s + rho) / s2) * torch.exp(torch.where(near, s * rho, torch.zeros_like(s * rho)))
    gk = -0.25 * sig / s * torch.where(near, a + b, torch.zeros_like(a))
    g0 = 0.5 * r * torch.erf(rho / s2)
    er = torch.exp(-0.5 * rho * rho)
    q = sig / math.sqrt(2 * math.pi)
    if green == "HEJ_2":
        g0 = g0 - (1.0 - er) * q
    else:
        gk = gk - 0.25 * sig * math.sqrt(2 / math.pi) * torch.exp(-0.5 * (s * s + rho * rho))
        g0 = g0 - 0.5 * (1.0 - er) * q
    return torch.where(pos, gk, g0 + 0 * k)


def exact(case, seed):
    """The same solve with plain 64-bit FFTs of the extended problem, the kernel written out from its
    definition.  The regularisation length is two spacings, the library's default."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, h, node, bcs = _dims(case), _h(case), case["center"] == "node", _bcs(case)
    sig = 2.0 * h
    rhs = _rhs(case, seed, dev)
    lda = 3 if case["rot"] else 1
    per = [_line(n[d], bcs[d], node) for d in range(3)]
    unb = [("U" in b) for b in bcs]
    nunb = sum(unb)
    if nunb == 2:
        return None  # no case has two open directions and a third one that is not
    # distances along the open directions, wave numbers along the others (last axis: the half spectrum of rfft)
    dist, wave = [], []
    for d in range(3):
        i = torch.arange(per[d], dtype=torch.float64, device=dev)
        i = torch.minimum(i, per[d] - i) if per[d] > 1 else i
        dist.append((i * h).reshape(_length_axis(per[d], d)))
        wave.append((i * (2 * math.pi / (per[d] * h))).reshape(_length_axis(per[d], d)))
    half = per[0] // 2 + 1
    if nunb == 3:
        r = torch.sqrt(dist[0] ** 2 + dist[1] ** 2 + dist[2] ** 2)
        g = torch.fft.rfftn(_kernel_regular(case["green"], r, sig, h ** 3) * h ** 3, dim=(1, 2, 3)).real
        del r
    elif nunb == 1:
        du = unb.index(True)
        k2 = sum(wave[d] ** 2 for d in range(3) if d != du and per[d] > 1)
        base = [2 * math.pi / (h * (per[d] if bcs[d] == "PP" else 2 * (n[d] - 1 if node else n[d])))
                for d in range(3) if d != du and per[d] > 1]
        g = _kernel_line(case["green"], torch.sqrt(k2), dist[du], sig, 0.2 * sum(base)) * h
        g = torch.fft.fft(g, dim=3 - du).real.narrow(3, 0, half)
    else:
        k2 = sum(wave[d] ** 2 for d in range(3) if per[d] > 1)
        g = torch.where(k2 > 0, -1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
        # only the wave numbers of the line's own sequence carry energy; the mean is set to zero
        g = g.narrow(3, 0, half)
    out = torch.empty_like(rhs)
    for b in range(case["batch"]):
        spec = []
        for c in range(lda):
            f = rhs[b * lda + c:b * lda + c + 1]
            for d in range(3):
                f = _extend(f, d, bcs[d], node)
            spec.append(torch.fft.rfftn(f, dim=(1, 2, 3)))
            del f
        if case["rot"]:
            k = []
            for d in range(3):
                s = torch.fft.fftfreq(per[d], d=h, dtype=torch.float64, device=dev) * (2 * math.pi)
                s = s.reshape(_length_axis(per[d], d))
                if per[d] % 2 == 0:  # the Nyquist wave number counts as positive
                    s.view(-1)[per[d] // 2] *= -1
                k.append(s.narrow(3, 0, half) if d == 0 else s)
            for c in range(3):
                p, q = (c + 1) % 3, (c + 2) % 3
                u = 1j * (k[p] * spec[q] - k[q] * spec[p]) * g
                _put(out, b * lda + c, torch.fft.irfftn(u, s=per[::-1], dim=(1, 2, 3)), case)
                del u
        else:
            _put(out, b, torch.fft.irfftn(spec[0] * g, s=per[::-1], dim=(1, 2, 3)), case)
        del spec
    return out


def _put(out, i, u, case):
    """The grid's own points of the periodic result; node-centred odd faces hold zero, the last periodic
    node repeats the first."""
    n, node, bcs = _dims(case), case["center"] == "node", _bcs(case)
    for d in range(3):
        ax = 3 - d
        if node and bcs[d] == "PP":
            u = torch.cat([u, u.narrow(ax, 0, 1)], ax)
        else:
            u = u.narrow(ax, 0, n[d])
    u = u.clone()
    if node:
        for d in range(3):
            if bcs[d][0] == "O":
                u.select(3 - d, 0).zero_()
            if bcs[d][1] == "O":
                u.select(3 - d, n[d] - 1).zero_()
    out[i] = u[0]
