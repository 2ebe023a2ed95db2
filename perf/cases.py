"""Performance cases of the evolution engine: what its users have it do, through its public
entry points, from lattices of a few thousand cells to the 8192^2 precision workload.

A case is a dict of plain values; `kind` says which entry point it goes through:

  solver   the drop-in Solver: a State is filled, evolved and read back on the host
  tile     one lattice tile that stays on the GPU (Kernel): state in, evolve, state out
  batch    many tiles of uneven sizes in one launch per step (Batch)
  pair     two species with a Rabi coupling (Pair)
  trap     a potential that changes with every step (Kernel.evolve_potentials)
  adjoint  a differentiable evolution, forward and backward (adjoint.evolve)

Lattice sizes, couplings and time steps are those of the benchmark workloads and the tests,
or fractions of them.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "trotter-suzuki-mpi_b200"))


def _case(name, kind, nx, ny, length, dt, steps, **more):
    c = {"kind": kind, "nx": nx, "ny": ny, "length": length, "dt": dt, "steps": steps,
         "fp32": False, "imag": False, "px": False, "py": False, "g": 0.0, "lhy": 0.0,
         "omega": 0.0, "cyl": False, "l": 0, "wy": 1.5, "checkpoint": 0, "count": 0}
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a quick look at a small lattice: few steps, so launches and latency are what it costs
        _case("small_real_64", "tile", 64, 64, 10.0, 1e-3, 20),
        # the plain method: the whole program of a first user, host arrays in and out
        _case("solver_real_256", "solver", 256, 256, 20.0, 1e-4, 1000, wy=1.0),
        # relaxation to a GPE ground state, the headline workload, a stretch of its steps
        _case("gpe_imag_2048", "tile", 2048, 2048, 24.0, 1e-4, 100, imag=True, g=100.0),
        # the same with single-precision storage
        _case("gpe_imag_2048_fp32", "tile", 2048, 2048, 24.0, 1e-4, 100, imag=True, g=100.0,
              fp32=True),
        # real-time dynamics on an odd, unequal, periodic lattice with the Lee-Huang-Yang term
        _case("gpe_lhy_periodic_1013x770", "tile", 1013, 770, 20.0, 1e-4, 100, px=True, py=True,
              g=50.0, lhy=1.0),
        # vortices in a rotating frame in double precision
        _case("vortex_periodic_2048", "tile", 2048, 2048, 20.0, 5e-5, 40, px=True, py=True,
              g=500.0, omega=0.7, wy=1.0),
        # the precision workload: the largest lattice, single-precision storage
        _case("vortex_periodic_8192_fp32", "tile", 8192, 8192, 40.0, 5e-5, 20, px=True, py=True,
              g=500.0, omega=0.7, wy=1.0, fp32=True),
        # a parameter scan: many instances of uneven sizes at once
        _case("batch_32_uneven", "batch", 1024, 128, 20.0, 1e-4, 50, g=200.0, wy=1.0, count=32),
        # gradients of a nonlinear evolution by checkpoints
        _case("adjoint_gpe_512", "adjoint", 512, 512, 20.0, 1e-4, 300, g=50.0, checkpoint=100,
              wy=1.0),
        # two species with a Rabi coupling, real time
        _case("pair_rabi_1024", "pair", 1024, 1024, 24.0, 1e-4, 60, g=100.0),
        # a cylindrical lattice with angular momentum, imaginary time
        _case("cylindrical_imag_1024", "tile", 1024, 1024, 12.0, 1e-4, 100, imag=True, g=100.0,
              cyl=True, l=1),
        # a moving trap: V(x, y, t) evaluated and applied on the GPU, 16 steps per call
        _case("moving_trap_1024", "trap", 1024, 1024, 24.0, 1e-4, 64, g=100.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes over the logarithm of the range, odd ones among them."""
    kind = rng.choice(["tile", "tile", "tile", "tile", "tile", "solver", "batch", "pair", "trap",
                       "adjoint"])
    length, dt = rng.choice([10.0, 20.0, 24.0]), rng.choice([5e-5, 1e-4, 2e-4])
    g = round(rng.uniform(1.0, 200.0), 3)
    if kind == "solver":
        n = _log_int(rng, 48, 512)
        return _case(None, kind, n, n + rng.randint(-8, 8), length, dt, rng.randint(100, 1000),
                     wy=1.0, g=rng.choice([0.0, g]), imag=rng.random() < 0.3,
                     fp32=rng.random() < 0.3)
    if kind == "batch":
        return _case(None, kind, _log_int(rng, 256, 1024), _log_int(rng, 48, 200), length, dt,
                     rng.randint(20, 60), g=g, wy=1.0, count=rng.randint(4, 32),
                     fp32=rng.random() < 0.5)
    if kind == "adjoint":
        n = _log_int(rng, 96, 512)
        if rng.random() < 0.5:
            return _case(None, kind, n, n + rng.randint(-9, 9), length, dt, rng.randint(50, 300),
                         wy=1.0)
        return _case(None, kind, n, n + rng.randint(-9, 9), length, dt, rng.randint(50, 300),
                     g=g, wy=1.0, checkpoint=rng.choice([20, 50, 100]))
    nx = _log_int(rng, 64, 3000)
    ny = max(48, int(nx * rng.uniform(0.6, 1.4)))
    steps = rng.randint(10, 100)
    if kind == "pair":
        return _case(None, kind, min(nx, 1500), min(ny, 1500), 24.0, dt, steps, g=g,
                     fp32=rng.random() < 0.4)
    if kind == "trap":
        return _case(None, kind, min(nx, 1500), min(ny, 1500), 24.0, dt, steps, g=g)
    c = _case(None, kind, nx, ny, length, dt, steps, fp32=rng.random() < 0.4,
              imag=rng.random() < 0.4, g=rng.choice([0.0, g, g]),
              lhy=rng.choice([0.0, 0.0, 1.0]))
    form = rng.random()
    if form < 0.25:
        c.update(omega=0.7, imag=False, px=True, py=True)
    elif form < 0.45:
        c.update(cyl=True, l=rng.randint(0, 2), lhy=0.0)
    else:
        c.update(px=rng.random() < 0.5)
        c.update(py=c["px"])
    return c


# ------------------------------------------------------------------ geometry and inputs


def _geometry(c, nx=None, ny=None):
    """The tile of a lattice: its halo, spacings and the coordinates of its columns and rows."""
    nx, ny = nx or c["nx"], ny or c["ny"]
    h = 8 if c["omega"] else 4
    cols = nx + 1 if c["cyl"] else nx
    length_y = 2 * c["length"] if c["cyl"] else c["length"]
    dx = c["length"] / (cols - 0.5) if c["cyl"] else c["length"] / cols
    dy = length_y / ny
    hx, hy = (h if c["px"] else 0), (h if c["py"] else 0)
    ix = np.arange(-hx, cols + hx)
    iy = np.arange(-hy, ny + hy)
    y = (np.mod(iy, ny) + 0.5) * dy - 0.5 * length_y
    x = ix * dx - 0.5 * dx if c["cyl"] else (np.mod(ix, cols) + 0.5) * dx - 0.5 * c["length"]
    return {"h": h, "hx": hx, "hy": hy, "cols": cols, "ny": ny, "dx": dx, "dy": dy,
            "ix": np.mod(ix, cols), "iy": np.mod(iy, ny), "x": x, "y": y,
            "shape": (len(iy), len(ix)), "inner": (slice(hy, hy + ny),
                                                   slice(hx + int(c["cyl"]), hx + cols))}


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _trap(c, geo, wx=1.0, wy=None, shift=0.0):
    x, y = _dev(geo["x"])[None, :], _dev(geo["y"])[:, None]
    v = 0.5 * (wx * wx * (x - shift) ** 2 + (wy or c["wy"]) ** 2 * y * y)
    if c["cyl"]:
        v = v + c["l"] ** 2 / (2.0 * x * x)
    return v.contiguous()


def _psi(c, geo, seed, centre=(0.0, 0.0), width=2.0, kick=0.0):
    """A normalised Gaussian (a Thomas-Fermi profile with windings in a rotating frame) with 1 %
    of seeded noise, over the whole tile: halo cells repeat the lattice's."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    x, y = _dev(geo["x"])[None, :], _dev(geo["y"])[:, None]
    r = random.Random(int(seed))
    cx, cy = centre[0] + r.uniform(-0.3, 0.3), centre[1] + r.uniform(-0.3, 0.3)
    noise = torch.rand((geo["ny"], geo["cols"]), generator=gen, device="cuda",
                       dtype=torch.float64)
    noise = noise[torch.tensor(geo["iy"], device="cuda")][:, torch.tensor(geo["ix"],
                                                                         device="cuda")]
    if c["omega"]:
        mu = math.sqrt(c["g"] / math.pi) if c["g"] else 5.0
        amp = torch.sqrt(torch.clamp(mu - 0.5 * (x * x + y * y), min=0.0)) + 1e-3
        theta = torch.zeros_like(amp)
        for _ in range(8):
            theta += torch.atan2(y - r.uniform(-5, 5), x - r.uniform(-5, 5))
        psi = torch.polar(amp * (1 + 0.01 * noise), theta)
    else:
        amp = torch.exp(-((x - (0 if c["cyl"] else cx)) ** 2 + (y - cy) ** 2) / (2 * width ** 2))
        if c["cyl"]:
            amp = amp * torch.abs(x) ** c["l"] * torch.sign(x) ** c["l"]
        psi = torch.polar(torch.ones_like(amp), kick * x + 0 * y) * (amp * (1 + 0.01 * noise))
        if c["cyl"]:  # the axis column mirrors its neighbour
            psi[:, 0] = (-1.0) ** c["l"] * psi[:, 1]
    inner = psi[geo["inner"]]
    psi = psi / torch.sqrt((inner.abs() ** 2).sum() * geo["dx"] * geo["dy"])
    return psi.to(torch.complex64 if c["fp32"] else torch.complex128).contiguous()


def _norm(geo, psi):
    return float((psi[geo["inner"]].to(torch.complex128).abs() ** 2).sum()) * geo["dx"] * geo["dy"]


def _instances(c):
    """The uneven batch: side, trap frequency, coupling, centre and width of each instance."""
    r = random.Random(c["nx"] * 1009 + c["count"])
    return [{"side": r.randint(c["ny"] // 8, c["nx"] // 8) * 8, "w": r.uniform(0.5, 2.0),
             "g": r.uniform(1.0, c["g"]), "centre": (r.uniform(-2, 2), r.uniform(-2, 2)),
             "width": r.uniform(0.5, 2.0)} for _ in range(c["count"])]


def _sites(c):
    if c["kind"] == "batch":
        return sum(i["side"] ** 2 for i in _instances(c))
    geo = _geometry(c)
    return geo["shape"][0] * geo["shape"][1] * (2 if c["kind"] == "pair" else 1)


# ------------------------------------------------------------------ what a program holds


def _lattice(ts, c, nx=None, ny=None):
    nx, ny = nx or c["nx"], ny or c["ny"]
    if c["cyl"]:
        return ts.Lattice2D(nx, c["length"], ny, 2 * c["length"], coordinate_system="cylindrical")
    return ts.Lattice2D(nx, c["length"], ny, c["length"], c["px"], c["py"], c["omega"])


def _tile(ts, c, grid, geo, v, norm, g=None, mass=1.0):
    """A Kernel with its table, and what keeps it alive."""
    ham = ts.Hamiltonian(grid, ts.Potential(grid), mass, c["g"] if g is None else g, c["lhy"],
                         c["omega"])
    desc = ts.make_desc(grid, ham, c["dt"], c["imag"], norm, 1 if c["fp32"] else 0)
    if c["cyl"]:
        desc.angular_momentum = c["l"]
    k = ts.Kernel(desc)
    assert k.shape == geo["shape"]
    k.set_potential_device(v.data_ptr(), v.shape[1], c["dt"])
    return k


def prepare(case, seed):
    import trottersuzuki_b200 as ts
    c = case
    kind = c["kind"]
    geo = _geometry(c)
    if kind == "solver":
        grid = _lattice(ts, c)
        pot = ts.HarmonicPotential(grid, 1.0, c["wy"])
        psi = _psi(dict(c, fp32=False), geo, seed, (1.0, 0.0), 1.0).cpu().numpy()
        return {"c": c, "ts": ts, "grid": grid, "pot": pot,
                "ham": ts.Hamiltonian(grid, pot, 1.0, c["g"]), "re": psi.real.copy(),
                "im": psi.imag.copy()}
    if kind == "batch":
        tiles = []
        for n, i in enumerate(_instances(c)):
            gi = _geometry(c, i["side"], i["side"])
            v = _trap(c, gi, i["w"], i["w"])
            psi = _psi(c, gi, seed * 64 + n, i["centre"], i["width"])
            k = _tile(ts, c, _lattice(ts, c, i["side"], i["side"]), gi, v, 0.0, i["g"])
            tiles.append((k, psi, torch.empty_like(psi)))
        torch.cuda.synchronize()
        return {"c": c, "tiles": tiles, "batch": ts.Batch([t[0] for t in tiles])}
    if kind == "adjoint":
        from trottersuzuki_b200 import adjoint
        grid = _lattice(ts, c)
        desc = ts.make_desc(grid, ts.Hamiltonian(grid, ts.Potential(grid), 1.0, c["g"]), c["dt"])
        v, psi, mask = _adjoint_inputs(c, geo, seed)
        return {"c": c, "evolve": adjoint.evolve, "v": v.requires_grad_(),
                "psi": psi.requires_grad_(), "mask": mask, "da": geo["dx"] * geo["dy"],
                "engine": adjoint.AdjointEngine(desc, c["dt"], c["steps"], c["checkpoint"])}
    v = _trap(c, geo)
    psi = _psi(c, geo, seed)
    if kind == "pair":
        grid = _lattice(ts, c)
        vb = _trap(c, geo, 1.2, 1.0)
        psib = _psi(c, geo, seed + 1, (1.5, 0.0))
        a = _tile(ts, c, grid, geo, v, 0.0)
        b = _tile(ts, c, grid, geo, vb, 0.0, 0.8 * c["g"], 1.2)
        torch.cuda.synchronize()
        return {"c": c, "a": a, "b": b, "psi": psi, "psib": psib,
                "pair": ts.Pair(a, b, 0.6 * c["g"], 5.0, 2.0, c["dt"]),
                "out": torch.empty_like(psi), "outb": torch.empty_like(psib)}
    k = _tile(ts, c, _lattice(ts, c), geo, v, _norm(geo, psi) if c["imag"] else 0.0)
    torch.cuda.synchronize()
    s = {"c": c, "k": k, "psi": psi, "out": torch.empty_like(psi), "geo": geo}
    if kind == "trap":
        s["x"], s["y"], s["stream"] = _dev(geo["x"])[None, :], _dev(geo["y"])[:, None], \
            torch.cuda.Stream()
        torch.cuda.synchronize()
    return s


def _moving(x, y, t, wy):
    return 0.5 * ((x - torch.sin(5.0 * t)) ** 2 + (wy * y) ** 2)


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "solver":
        ts = state["ts"]
        psi = ts.State(state["grid"])
        psi.init_state_matrix(state["re"], state["im"])
        solver = ts.Solver(state["grid"], psi, state["ham"], c["dt"],
                           kernel_type="gpu_fp32" if c["fp32"] else "gpu")
        solver.evolve(c["steps"], c["imag"])
        return {"psi": psi.get_state(), "norm": psi.get_squared_norm(),
                "energy": solver.get_total_energy()}
    if kind == "batch":
        for k, psi, _ in state["tiles"]:
            k.set_state_device(psi.data_ptr(), psi.shape[1])
        state["batch"].evolve(c["steps"])
        for k, _, out in state["tiles"]:
            k.get_state_device(out.data_ptr(), out.shape[1])
        return [t[2] for t in state["tiles"]]
    if kind == "adjoint":
        state["v"].grad = state["psi"].grad = None
        psi = state["evolve"](state["v"], state["psi"], state["engine"])
        loss = (state["mask"] * (psi.real ** 2 + psi.imag ** 2)).sum() * state["da"]
        loss.backward()
        return {"psi": psi.detach(), "loss": loss.detach(), "grad_v": state["v"].grad,
                "grad_psi": state["psi"].grad}
    if kind == "pair":
        for k, psi in ((state["a"], state["psi"]), (state["b"], state["psib"])):
            k.set_state_device(psi.data_ptr(), psi.shape[1])
        state["pair"].rabi(0.5)
        state["pair"].evolve(c["steps"])
        for k, out in ((state["a"], state["out"]), (state["b"], state["outb"])):
            k.get_state_device(out.data_ptr(), out.shape[1])
        return [state["out"], state["outb"]]
    k, psi, out = state["k"], state["psi"], state["out"]
    if kind == "trap":
        st = state["stream"]
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            k.set_stream(st.cuda_stream)
            k.set_state_device(psi.data_ptr(), psi.shape[1])
            h, w = k.shape
            for n in range(0, c["steps"], 16):
                m = min(16, c["steps"] - n)
                t = (torch.arange(n, n + m, device="cuda", dtype=torch.float64) * c["dt"])
                v = _moving(state["x"], state["y"], t.view(-1, 1, 1), c["wy"]).contiguous()
                k.evolve_potentials(v.data_ptr(), w, w * h, m, c["dt"])
            k.get_state_device(out.data_ptr(), out.shape[1])
        torch.cuda.current_stream().wait_stream(st)
        return out
    k.set_state_device(psi.data_ptr(), psi.shape[1])
    k.evolve(c["steps"])
    k.get_state_device(out.data_ptr(), out.shape[1])
    return out[state["geo"]["inner"]]


def work(case):
    """The state in and out and the potential in, once each; the arithmetic of every step (real
    operations per cell: 8 pair sweeps, the phase, and the sweeps that a form adds)."""
    c = case
    sites = _sites(c)
    cell = 8 if c["fp32"] else 16
    per = 8 * 6 + 8 + (20 if c["g"] else 0) + (10 if c["lhy"] else 0) + (36 if c["omega"] else 0) \
        + (24 if c["cyl"] else 0) + (14 if c["kind"] == "pair" else 0)
    flops, data = sites * c["steps"] * per, sites * (2 * cell + 8)
    if c["kind"] == "trap":
        data += sites * 8 * (c["steps"] - 1)
        flops += sites * c["steps"] * 20
    if c["kind"] == "adjoint":
        flops, data = 3 * flops, sites * (16 + 8 + 16 + 8 + 16)
    return {"bytes": data, "flops": flops}


# ------------------------------------------------------------------ the same in plain 64 bits


def _sweep_v(p, s, a, b):
    rows, cols = p.shape
    for x in (0, 1):
        y = (s + x) % 2
        n = (rows - y) // 2
        if n <= 0 or x >= cols:
            continue
        up, lo = p[y:y + 2 * n:2, x::2], p[y + 1:y + 2 * n:2, x::2]
        u = up.clone()
        up.mul_(a).add_(lo, alpha=b)
        lo.mul_(a).add_(u, alpha=b)


def _sweep_h(p, s, a, b):
    _sweep_v(p.transpose(0, 1), s, a, b)


def _half(c, geo, p, sign=1, mass=1.0):
    """V0 H0 V1 H1 of one step (sign -1: the inverse sweeps), or with `sign` None reversed."""
    kx, ky = (c["dt"] / (4 * mass * d * d) for d in (geo["dx"], geo["dy"]))
    if c["imag"]:
        h, v = (math.cosh(kx), math.sinh(kx)), (math.cosh(ky), math.sinh(ky))
    else:
        h, v = (math.cos(kx), 1j * math.sin(kx)), (math.cos(ky), 1j * math.sin(ky))
    order = [(_sweep_v, 0, v), (_sweep_h, 0, h), (_sweep_v, 1, v), (_sweep_h, 1, h)]
    for f, s, (a, b) in order if sign else order[::-1]:
        f(p, s, a, b if sign != -1 else -b)


def _rotate(p, first, count, a, b, dim):
    """Pairs (i, i + 1) along `dim` from `first`: (f, s) -> (a f + b s, a s - b f)."""
    f = p.narrow(dim, first, count * 2 - 1)
    s = p.narrow(dim, first + 1, count * 2 - 1)
    f, s = (f[::2], s[::2]) if dim == 0 else (f[:, ::2], s[:, ::2])
    u = f.clone()
    f.mul_(a).add_(b * s)
    s.mul_(a).sub_(b * u)


def _rotation(c, geo, p):
    rows, cols = p.shape
    ax = c["omega"] * c["dt"] * geo["dx"] / (2 * geo["dy"])
    ay = c["omega"] * c["dt"] * geo["dy"] / (2 * geo["dx"])
    ox, oy = int(-geo["hx"] - geo["cols"] * 0.5), int(-geo["hy"] - geo["ny"] * 0.5)
    ry = _dev(-0.5 * ay * (np.arange(rows) + oy))[:, None]
    rx = _dev(ax * (np.arange(cols) + ox))[None, :]
    for axis, ang, n in ((1, ry, cols), (0, rx, rows), (1, ry, cols)):
        for par in (0, 1):
            if (n - par) // 2 > 0:
                _rotate(p, par, (n - par) // 2, torch.cos(ang), torch.sin(ang), axis)


def _radial(c, geo, p, par):
    """The radial pairs (i, i + 1) with i = par (mod 2)."""
    n = p.shape[1]
    kr = c["dt"] / (8 * geo["dx"] ** 2)
    i = np.arange(par, n - 1, 2).astype(np.float64)
    x = np.where(i == 0, 1.0, i)
    ang, ratio = kr / np.sqrt(x * x - 0.25), np.sqrt((2 * x + 1) / (2 * x - 1))
    sk, ck = (np.sin(ang), np.cos(ang)) if c["imag"] else (np.sinh(ang), np.cosh(ang))
    a, b, d = ck, sk * ratio, -sk / ratio
    if par == 0:
        a[0] = math.cosh(2 * kr) if c["imag"] else math.cos(2 * kr)
        b[0] = d[0] = -math.sinh(2 * kr) if c["imag"] else -math.sin(2 * kr)
    a, b, d = (_dev(t)[None, :] * (1 if c["imag"] else 1) for t in (a, b, d))
    if not c["imag"]:
        b, d = 1j * b, 1j * d
    m = len(i)
    f, s = p[:, par:par + 2 * m:2], p[:, par + 1:par + 2 * m:2]
    u = f.clone()
    f.mul_(a).add_(b * s)
    s.mul_(a).add_(d * u)


def _phase(c, p, table, g, other=None, gb=0.0):
    n2 = p.real ** 2 + p.imag ** 2
    th = g * c["dt"] * n2
    if c["lhy"]:
        th += c["lhy"] * c["dt"] * n2 * torch.sqrt(n2)
    if other is not None:
        th += gb * c["dt"] * (other.real ** 2 + other.imag ** 2)
    p.mul_(table)
    p.mul_(torch.exp(-th) if c["imag"] else torch.exp(-1j * th))


def _step(c, geo, p, table, g, other=None, gb=0.0, mass=1.0):
    _half(c, geo, p, 1, mass)
    if c["cyl"]:
        _radial(c, geo, p, 0)
        _radial(c, geo, p, 1)
    _phase(c, p, table, g, other, gb)
    if c["omega"]:
        _rotation(c, geo, p)
    if c["cyl"]:
        _radial(c, geo, p, 1)
        _radial(c, geo, p, 0)
    _half(c, geo, p, None, mass)


def _halo(geo, p):
    if geo["hx"]:
        n = geo["cols"]
        p[:, :geo["hx"]] = p[:, n:n + geo["hx"]].clone()
        p[:, -geo["hx"]:] = p[:, geo["hx"]:2 * geo["hx"]].clone()
    if geo["hy"]:
        n = geo["ny"]
        p[:geo["hy"]] = p[n:n + geo["hy"]].clone()
        p[-geo["hy"]:] = p[geo["hy"]:2 * geo["hy"]].clone()


def _table(c, v):
    return torch.exp(-c["dt"] * v) if c["imag"] else torch.exp(-1j * c["dt"] * v)


def _exact_tile(c, geo, psi, v, g, potential=None):
    p = psi.to(torch.complex128).clone()
    table = _table(c, v)
    n0 = _norm(geo, p)
    for i in range(c["steps"]):
        if potential is not None:
            table = _table(c, potential(i))
        _step(c, geo, p, table, g)
        if potential is None and i < c["steps"] - 1:
            _halo(geo, p)
        if c["imag"]:
            p /= math.sqrt(_norm(geo, p) / n0)
            if c["cyl"]:
                p[:, 0] = (-1.0) ** c["l"] * p[:, 1]
    return p


def _rabi(c, a, b, var):
    """exp(-i (omega sigma / 2) var dt) on the pair of species."""
    w = math.hypot(2.5, 1.0)
    cs, sn = math.cos(-c["dt"] * var * w), math.sin(-c["dt"] * var * w)
    sr, si = 2.5 / w * sn, 1.0 / w * sn
    u = a.clone()
    a.mul_(cs).add_(b, alpha=complex(-si, sr))
    b.mul_(cs).add_(u, alpha=complex(si, sr))


def _adjoint_inputs(c, geo, seed):
    r = random.Random(int(seed) + 5)
    x, y = _dev(geo["x"])[None, :], _dev(geo["y"])[:, None]
    v = _trap(c, geo)
    for _ in range(16):
        w = r.uniform(1.0, 3.0)
        cx, cy = (r.uniform(-0.5, 0.5) * c["length"] for _ in range(2))
        v += r.uniform(-0.5, 0.5) * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * w * w))
    mask = (x > 0).to(torch.float64).expand(geo["shape"]).contiguous()
    return v, _psi(c, geo, seed, (-0.15 * c["length"], 0.0), 1.0, 2.0), mask


def _exact_adjoint(c, geo, seed):
    v, psi, mask = _adjoint_inputs(c, geo, seed)
    table, da = _table(c, v), geo["dx"] * geo["dy"]
    states, p = [], psi.clone()
    for _ in range(c["steps"]):
        states.append(p.clone())
        _step(c, geo, p, table, c["g"])
    lam, grad = 2 * da * mask * p, torch.zeros_like(v)
    g = c["g"] * c["dt"]
    for x in reversed(states):
        _half(c, geo, x)
        _half(c, geo, lam, -1)
        rot = table * torch.exp(-1j * g * (x.real ** 2 + x.imag ** 2))
        q = (lam.conj() * rot * x).imag
        grad += c["dt"] * q
        lam = rot.conj() * lam + 2 * g * q * x
        # H1 V1 H0 V0 backwards
        kx, ky = (c["dt"] / (4 * d * d) for d in (geo["dx"], geo["dy"]))
        for f, s, k in ((_sweep_h, 1, kx), (_sweep_v, 1, ky), (_sweep_h, 0, kx),
                        (_sweep_v, 0, ky)):
            f(lam, s, math.cos(k), -1j * math.sin(k))
    return {"psi": p, "loss": (mask * p.abs() ** 2).sum() * da, "grad_v": grad, "grad_psi": lam}


def exact(case, seed):
    c = case
    kind = c["kind"]
    geo = _geometry(c)
    if kind == "solver":
        psi = _psi(dict(c, fp32=False), geo, seed, (1.0, 0.0), 1.0)
        p = _exact_tile(c, geo, psi, _trap(c, geo), c["g"])
        return {"psi": p.cpu().numpy(), "norm": _norm(geo, p), "energy": None}
    if kind == "batch":
        outs = []
        for n, i in enumerate(_instances(c)):
            gi = _geometry(c, i["side"], i["side"])
            psi = _psi(c, gi, seed * 64 + n, i["centre"], i["width"])
            outs.append(_exact_tile(c, gi, psi, _trap(c, gi, i["w"], i["w"]), i["g"]))
        return outs
    if kind == "adjoint":
        return _exact_adjoint(c, geo, seed)
    psi = _psi(c, geo, seed)
    if kind == "pair":
        ta, tb = _table(c, _trap(c, geo)), _table(c, _trap(c, geo, 1.2, 1.0))
        a = psi.to(torch.complex128).clone()
        b = _psi(c, geo, seed + 1, (1.5, 0.0)).to(torch.complex128)
        _rabi(c, a, b, 0.5)
        for i in range(c["steps"]):
            old = a.clone()
            _step(c, geo, a, ta, c["g"], b, 0.6 * c["g"])
            _step(c, geo, b, tb, 0.8 * c["g"], old, 0.6 * c["g"], 1.2)
            _rabi(c, a, b, 0.5 if i == c["steps"] - 1 else 1.0)
        return [a, b]
    if kind == "trap":
        x, y = _dev(geo["x"])[None, :], _dev(geo["y"])[:, None]
        return _exact_tile(c, geo, psi, _trap(c, geo), c["g"],
                           lambda i: _moving(x, y, torch.tensor(i * c["dt"],
                                                                dtype=torch.float64,
                                                                device="cuda"), c["wy"]))
    return _exact_tile(c, geo, psi, _trap(c, geo), c["g"])[geo["inner"]]
