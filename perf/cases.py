"""The measured cases of the MHD time step.

A pass is what a program that uses the library does with one grid: it hands in
the state of its host arrays (cState records, pinned memory), advances it by
some steps through the fused entry points (or, for one case, through the
per-routine calls in ComputeSolution's order), and reads the new state back.
The precision of the host arrays follows the run's (float64, or float32 as in a
SINGLE_PRECISION build).

``exact`` restates the time step on whole arrays in float64 (torch): stages,
sources, Tcheck, the three TVD sweeps, with periodic or mirrored x.
"""
import math
import os
import tempfile

import numpy as np
import torch

from muram_main_gb300 import eos_table, gpumhd

FIELDS = ("rho", "mx", "my", "mz", "e", "bx", "by", "bz")
GH = 2
B_UNIT = math.sqrt(4.0 * math.pi)
DX = {"periodic": 3.2e6, "stratified": 1.6e6}
GRAV = 2.74e4


def _case(name, kind, setup, nx, ny, nz, precision, steps, **kw):
    c = dict(name=name, kind=kind, setup=setup, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps, eos=1000)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one step of a box of the size the smoke check uses
        _case("smallest_fp32_16x12x8", "steps", "periodic", 16, 12, 8, 32, 1),
        # an odd box whose rows are no multiple of 16 bytes, in both dimensions ragged against every tile
        _case("ragged_fp32_50x37x43", "steps", "periodic", 50, 37, 43, 32, 10),
        # the plain FP64 run: 64^3 periodic at 32 km, 100 G, 1 km/s
        _case("periodic_fp64_64x64x64", "steps", "periodic", 64, 64, 64, 64, 10),
        # the stratified convection box in FP64, at a quarter of its horizontal extent
        _case("stratified_fp64_128x192x192", "steps", "stratified", 128, 192, 192, 64, 2),
        # the stratified convection box in FP32, the run the benchmark quotes
        _case("stratified_fp32_128x384x384", "steps", "stratified", 128, 384, 384, 32, 10),
        # a large periodic box: a seeded block tiled over 192 x 512 x 512 cells
        _case("large_fp32_192x512x512", "tiled", "periodic", 192, 512, 512, 32, 4, tile=4),
        # FP32 with compensated sums, the mode for long stratified runs
        _case("compensated_fp32_128x256x256", "steps", "stratified", 128, 256, 256, 32, 5, compensated=1),
        # the full physics of a production box: open bottom, divB cleaning, Spitzer conduction
        _case("open_bottom_fp32_128x256x256", "physics", "stratified", 128, 256, 256, 32, 5),
        # the routines one by one, as MURaM calls them through the shim
        _case("routines_fp32_128x256x256", "routines", "stratified", 128, 256, 256, 32, 2),
        # a host program that owns the state: every step goes in and comes out
        _case("host_steps_fp32_128x256x256", "host", "stratified", 128, 256, 256, 32, 4),
        # an ensemble of independent boxes of uneven size in one launch
        _case("ensemble_fp32_16_boxes", "ensemble", "periodic", 0, 0, 0, 32, 20, boxes=16, eos=400),
        # the gradient of an objective with respect to the initial state
        _case("adjoint_fp64_48x32x32", "adjoint", "periodic", 48, 32, 32, 64, 4),
    ]


def draw(rng):
    """Fused FP32 runs of either set-up, FP64 and compensated runs, and the routines, on boxes from the
    smallest to the benchmark's, odd sizes among them."""
    what = rng.choice(["fp32", "fp32", "fp32", "fp64", "compensated", "routines", "routines64"])
    fp64 = what.endswith("64")
    most = 1.2e6 if fp64 else 1.6e7
    cells = math.exp(rng.uniform(math.log(1.5e3), math.log(most)))
    setup = rng.choice(["periodic", "stratified"])
    side = cells ** (1.0 / 3.0)
    f, g = (math.exp(rng.uniform(-0.5, 0.5)) for _ in range(2))
    nx, ny = max(7, round(side * f)), max(7, round(side * g))
    nz = max(7, round(cells / (nx * ny)))
    if rng.random() < 0.5:  # rows of whole 16 bytes, as most runs choose them
        nx = max(8, nx // 4 * 4)
    steps = rng.randint(1, 2) if what.startswith("routines") else rng.randint(1, 6)
    c = dict(kind="routines" if what.startswith("routines") else "steps", setup=setup, nx=nx, ny=ny, nz=nz,
             precision=64 if fp64 else 32, steps=steps, eos=1000)
    if what == "compensated":
        c["compensated"] = 1
    return c


# ------------------------------------------------------------------ inputs
def _eos_path(n):
    path = os.path.join(tempfile.gettempdir(), "gpumhd_eos_%d_%d.dat" % (n, os.getuid()))
    if not os.path.exists(path):
        eos_table.write_table(path, n_eps=n, n_lr=n, n_lp3=200, n_s3=160)
    return path


class _Eos:
    """ln p and ln T tables of an EOS file (axes ln eps, ln rho), bilinear in float64."""

    def __init__(self, path, device):
        with open(path, "rb") as fh:
            h = np.frombuffer(fh.read(56), dtype="<f4").astype(np.float64)
            self.ne, self.nr = int(h[0]), int(h[1])
            t = np.frombuffer(fh.read(8 * self.ne * self.nr), dtype="<f4").astype(np.float64)
        self.eps0, self.lr0, self.eps_off = float(h[4]), float(h[6]), float(h[12])
        self.de = (float(h[5]) - self.eps0) / (self.ne - 1)
        self.dr = (float(h[7]) - self.lr0) / (self.nr - 1)
        # the values the library holds: divided by the cell's area, in float32
        t = (t / (self.de * self.dr)).astype(np.float32).astype(np.float64)
        self.tabs = torch.from_numpy(t.reshape(2, self.nr * self.ne)).to(device)

    def look(self, which, ei, rho):
        """exp of table `which` (0: p, 1: T) at internal energy per mass ei and density rho."""
        le, lr = torch.log(ei + self.eps_off), torch.log(rho)
        i = ((le - self.eps0) * (1.0 / self.de)).long().clamp(0, self.ne - 2)
        j = ((lr - self.lr0) * (1.0 / self.dr)).long().clamp(0, self.nr - 2)
        at = j * self.ne + i
        i, j = i.double(), j.double()
        a, b = le - (self.eps0 + self.de * i), (self.eps0 + self.de * (i + 1)) - le
        c, d = lr - (self.lr0 + self.dr * j), (self.lr0 + self.dr * (j + 1)) - lr
        del i, j, le, lr
        T = self.tabs[which]
        s = a * c * T[at + self.ne + 1]
        s += a * d * T[at + 1]
        s += b * c * T[at + self.ne]
        s += b * d * T[at]
        return torch.exp(s)

    def energy_for(self, T, rho):
        """Internal energy per mass with temperature T at density rho (1-D tensors), by bisection."""
        lo, hi = torch.full_like(rho, math.log(2e11)), torch.full_like(rho, math.log(1e14))
        for _ in range(50):
            mid = 0.5 * (lo + hi)
            low = self.look(1, torch.exp(mid), rho) < T
            lo, hi = torch.where(low, mid, lo), torch.where(low, hi, mid)
        return torch.exp(0.5 * (lo + hi))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _field(shape, gen, device):
    """Real random field, random phases on the wavenumbers 1 to 8 (as far as the box resolves them)."""
    nz, ny, nx = shape
    kz = torch.fft.fftfreq(nz, 1.0 / nz, dtype=torch.float64, device=device)[:, None, None]
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device=device)[None, :, None]
    kx = torch.fft.rfftfreq(nx, 1.0 / nx, dtype=torch.float64, device=device)[None, None, :]
    kk = (kx * kx + ky * ky + kz * kz).sqrt()
    keep = (kk >= 1) & (kk <= max(1.0, min(8.0, min(shape) / 3.0)))
    n = int(keep.sum())
    amp = torch.randn(n, generator=gen, dtype=torch.float64).square() + 0.5
    ph = torch.rand(n, generator=gen, dtype=torch.float64) * (2 * math.pi)
    spec = torch.zeros(kk.shape, dtype=torch.complex128, device=device)
    spec[keep] = torch.polar(amp, ph).to(device)
    return torch.fft.irfftn(spec, s=shape)


def _state(setup, nx, ny, nz, seed, eos_n, v_rms=None, b_gauss=None):
    """Interior state (8, nz, ny, nx) in float64 on the device."""
    dev = _device()
    eos = _Eos(_eos_path(eos_n), dev)
    gen = torch.Generator().manual_seed(int(seed))
    shape, dx = (nz, ny, nx), DX[setup]
    U = torch.empty((8,) + shape, dtype=torch.float64, device=dev)
    x = torch.arange(nx, dtype=torch.float64, device=dev)
    if setup == "periodic":
        T, v_rms, b_gauss = 6000.0, v_rms or 1e5, b_gauss or 100.0
        rho = torch.full_like(x, 3e-7)
        ei = eos.energy_for(T, rho)
    else:
        T, v_rms, b_gauss = 1e4, v_rms or 5e4, b_gauss or 20.0
        rho0 = torch.full((1,), 3e-7, dtype=torch.float64, device=dev)
        H = float(eos.look(0, eos.energy_for(T, rho0), rho0) / (rho0 * GRAV))
        rho = 3e-7 * torch.exp(-x * dx / H)
        ei = eos.energy_for(T, rho)
    U[0] = rho
    v = torch.stack([_field(shape, gen, dev) for _ in range(3)])
    if setup == "stratified":
        v[0] *= torch.sin(math.pi * (x + 0.5) / nx)
    v *= v_rms / v.square().sum(0).mean().sqrt()
    U[1:4] = rho * v
    U[4] = rho * ei + 0.5 * rho * v.square().sum(0)
    del v
    A = [_field(shape, gen, dev) for _ in range(3)]  # x, y, z components

    def d(f, axis):
        return (8.0 * (f.roll(-1, axis) - f.roll(1, axis)) - (f.roll(-2, axis) - f.roll(2, axis))) / (12.0 * dx)

    U[5] = d(A[2], 1) - d(A[1], 0)
    U[6] = d(A[0], 0) - d(A[2], 2)
    U[7] = d(A[1], 2) - d(A[0], 1)
    U[5:] *= (b_gauss / B_UNIT) / U[5:].square().sum(0).mean().sqrt()
    if setup == "stratified":
        U[5] += 50.0 / B_UNIT
    return U


MIRROR = (1.0, -1.0, 1.0, 1.0, 1.0, 1.0, -1.0, -1.0)  # signs across a closed x boundary


def _pad(f, axis, wrap=True, sign=1.0):
    """f with two ghost cells at both ends of the axis: periodic, or mirrored."""
    n = f.shape[axis]
    a, b = f.narrow(axis, 0, 2), f.narrow(axis, n - 2, 2)
    if wrap:
        return torch.cat([b, f, a], axis)
    return torch.cat([sign * a.flip(axis), f, sign * b.flip(axis)], axis)


def _with_ghosts(U, setup):
    out = []
    for v in range(8):
        f = _pad(U[v], 2, setup == "periodic", MIRROR[v])
        out.append(_pad(_pad(f, 1), 0))
    return out


def _host(U, setup, dtype):
    """The cState records of a state: pinned host memory, 8 values per node."""
    rec = torch.stack(_with_ghosts(U, setup), -1).to(dtype)
    return rec.cpu().pin_memory() if torch.cuda.is_available() else rec.cpu()


def _params(case, nx, ny, nz, **kw):
    setup = case["setup"]
    if setup == "stratified":
        kw.update(periodic_x=0, grav=GRAV)
    if case.get("compensated"):
        kw.update(compensated=1)
    if case["kind"] == "physics":
        kw.update(xbnd=1, bnd_top=0, bnd_bcrit=2.5e30, divB_switch=1, divB_itmax=5, divB_err=0.2, spitzer=1e-6)
    return gpumhd.default_params(nx, ny, nz, DX[setup], precision=case["precision"], **kw)


def _context(case, nx, ny, nz, **kw):
    return gpumhd.MuramGPU(_params(case, nx, ny, nz, **kw), eos_path=_eos_path(case["eos"]))


def _box_list(case):
    """Sizes, velocity and field strengths of an ensemble's boxes: the same boxes for every seed."""
    rng = np.random.default_rng(2024)
    out = []
    for _ in range(case["boxes"]):
        nx, ny, nz = (int(s) for s in rng.choice([32, 48, 64, 96], 3))
        out.append((nx, ny, nz, float(np.exp(rng.uniform(np.log(0.2e5), np.log(2e5)))),
                    float(np.exp(rng.uniform(np.log(10.0), np.log(500.0))))))
    return out


ADJOINT_DT = 0.4


def _adjoint_seed(case, seed):
    """dJ/dU_T on the interior: independent normal weights."""
    gen = torch.Generator().manual_seed(int(seed) + 77)
    return torch.randn((8, case["nz"], case["ny"], case["nx"]), generator=gen, dtype=torch.float64)


def prepare(case, seed):
    nx, ny, nz, kind, setup = case["nx"], case["ny"], case["nz"], case["kind"], case["setup"]
    dtype = torch.float64 if case["precision"] == 64 else torch.float32
    s = {"case": case, "np": np.float64 if dtype == torch.float64 else np.float32}

    def pinned(n):
        return torch.empty((n, 8), dtype=dtype).pin_memory()

    if kind == "ensemble":
        boxes, s["in"], total = [], [], 0
        for b, (bx, by, bz, v, g) in enumerate(_box_list(case)):
            s["in"].append(_host(_state(setup, bx, by, bz, seed * 1000 + b, case["eos"], v, g), setup, dtype))
            boxes.append(_context(case, bx, by, bz))
            total += (bx + 4) * (by + 4) * (bz + 4)
            boxes[-1].upload_ptr(gpumhd.FIELD_U, s["in"][-1].data_ptr(), s["np"])
        s["out"] = pinned(total)
        s["ens"] = gpumhd.MuramEnsemble(boxes)
        s["ens"].autotune(2)
        return s
    if kind == "tiled":
        t = case["tile"]
        seedbox = _context(case, nx, ny // t, nz // t)
        U = _host(_state(setup, nx, ny // t, nz // t, seed, case["eos"]), setup, dtype)
        seedbox.upload_ptr(gpumhd.FIELD_U, U.data_ptr(), s["np"])
        seedbox.synchronize()
        s["seedbox"] = seedbox
        s["box"] = _context(case, nx, ny, nz)
        s["out"] = pinned((nx + 4) * (ny + 4) * (nz + 4))
        return s
    U = _state(setup, nx, ny, nz, seed, case["eos"])
    if kind == "adjoint":
        s["box"] = _context(case, nx, ny, nz, autostep=0, dt=ADJOINT_DT)
        s["in"] = torch.stack(_with_ghosts(U, setup)).cpu().numpy()
        lam = torch.zeros((8, nz + 4, ny + 4, nx + 4), dtype=torch.float64)
        lam[:, 2:-2, 2:-2, 2:-2] = _adjoint_seed(case, seed)
        s["lam"] = lam.numpy()
        return s
    s["in"] = _host(U, setup, dtype)
    s["box"] = _context(case, nx, ny, nz)
    s["out"] = pinned((nx + 4) * (ny + 4) * (nz + 4))
    if kind == "host":
        s["out2"] = pinned((nx + 4) * (ny + 4) * (nz + 4))
    if kind == "physics":
        s["zero"] = torch.zeros((nx + 4) * (ny + 4) * (nz + 4), dtype=dtype).pin_memory()
    return s


def _named(out, n):
    return {f: out[:n, v] for v, f in enumerate(FIELDS)}


def run(s):
    case, t = s["case"], s["np"]
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        ens, at = s["ens"], 0
        for box, u in zip(ens.boxes, s["in"]):
            box.upload_ptr_async(gpumhd.FIELD_U, u.data_ptr(), t)
        ens.run_steps(steps)
        for box in ens.boxes:
            n = int(np.prod(box.shape))
            box.download_ptr_async(gpumhd.FIELD_U, s["out"][at].data_ptr(), t)
            at += n
        for box in ens.boxes:
            box.synchronize()
        return _named(s["out"], at)
    g = s["box"]
    if kind == "adjoint":
        g.upload_state(s["in"])
        grad = g.adjoint(steps, s["lam"], checkpoint_every=2)
        return {f: grad[v] for v, f in enumerate(FIELDS)}
    n = s["out"].shape[0]
    if kind == "host":
        outs = (s["out"], s["out2"])
        for k in range(steps):
            g.upload_ptr_async(gpumhd.FIELD_U, s["in"].data_ptr(), t)
            g.enqueue_steps(1)
            g.download_ptr_async(gpumhd.FIELD_U, outs[k & 1].data_ptr(), t)
        g.synchronize()
        return _named(outs[(steps - 1) & 1], n)
    if kind == "tiled":
        g.tile_from(s["seedbox"])
    else:
        g.upload_ptr(gpumhd.FIELD_U, s["in"].data_ptr(), t)
    if kind == "physics":  # a restart: the cleaning's potential and count and the heat flux start afresh
        g.upload_ptr(gpumhd.FIELD_PHI, s["zero"].data_ptr(), t)
        g.upload_ptr(gpumhd.FIELD_SFLX, s["zero"].data_ptr(), t)
        g.set_divb_iters(3)
    if kind == "routines":
        g.exchange_grid(True)
        for _ in range(steps):
            g.step_reference_order()
    else:
        g.run_steps(steps)
    g.download_ptr(gpumhd.FIELD_U, s["out"].data_ptr(), t)
    return _named(s["out"], n)


def work(case):
    """A step reads and writes the state once per RK stage (with the step's first state from stage 2 on and the
    pressure) and once per TVD sweep: 140 words and about 4000 operations a cell.  The adjoint goes forward
    twice and back once at about four times a step's cost.  The host's records go in and out once a pass."""
    size = case["precision"] // 8
    if case["kind"] == "ensemble":
        cells = sum(x * y * z for x, y, z, _, _ in _box_list(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    n = cells * case["steps"] * (6 if case["kind"] == "adjoint" else 1)
    host = 16 * cells * size * (case["steps"] if case["kind"] == "host" else 1)
    return {"bytes": 140.0 * size * n + host, "flops": 4000.0 * n}


# ------------------------------------------------------------------- exact
VA_MAX, V_LIM, E_MAX, EPS_MIN, RHO_MIN = 1e7, 1e7, 4e15, 1e11, 1e-16


class _Exact:
    """The time step in float64 on the interior cells (default TVD and Tcheck settings)."""

    def __init__(self, setup, shape, eos_n, device):
        self.wrap = setup == "periodic"
        self.dx = DX[setup]
        self.grav = 0.0 if self.wrap else GRAV
        self.shape = shape
        self.eos = _Eos(_eos_path(eos_n), device)
        self.inv_va2 = 1.0 / VA_MAX ** 2
        nx = shape[2]
        h = (0.5 + torch.arange(-2, nx + 2, dtype=torch.float64, device=device)) / nx
        self.ht = (1.0 - 0.5 * (1.0 - h) / 1e-6).clamp(0.0).square().clamp(max=1.0)
        self.hb = (1.0 - 0.5 * h / 1e-6).clamp(0.0).square().clamp(max=1.0)

    def pad(self, f, axis, sign=1.0):
        return _pad(f, axis, self.wrap or axis != 2, sign)

    def prim(self, U):
        r = U[0]
        v = [U[q] / r for q in (1, 2, 3)]
        vv = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
        ei = U[4] - 0.5 * vv * r
        return [r] + v + [ei] + [U[5], U[6], U[7]], vv

    def pressure(self, U):
        W, _ = self.prim(U)
        return self.eos.look(0, W[4] / W[0], W[0])

    def boris(self, W):
        bb = W[5] ** 2 + W[6] ** 2 + W[7] ** 2
        x2 = bb / W[0] * self.inv_va2
        return bb, x2, (1.0 + x2) / (1.0 + x2 + x2 * x2)

    def cfl_speed(self, W, P):
        bb, _, lf = self.boris(W)
        c2, va2 = 5.0 / 3.0 * P / W[0], bb / W[0]
        v = (W[1] ** 2 + W[2] ** 2 + W[3] ** 2).sqrt()
        return float((v + torch.maximum(c2, lf * (c2 + va2)).sqrt()).max())

    def residual(self, U, P):
        W, vv = self.prim(U)
        r, v, ei, B = W[0], W[1:4], W[4], W[5:8]
        bb, x2, lf = self.boris(W)
        ent, pm = ei + 0.5 * r * vv + P, 0.5 * bb
        R = [torch.zeros_like(r) for _ in range(8)]
        for d in range(3):
            axis, n = 2 - d, r.shape[2 - d]

            def D(f, s):
                f = self.pad(f, axis, s)
                a = f.narrow(axis, 3, n) - f.narrow(axis, 1, n)
                b = f.narrow(axis, 4, n) - f.narrow(axis, 0, n)
                return (8.0 * a - b) / (12.0 * self.dx)

            m, bs = MIRROR[1:4], MIRROR[5:8]
            fl = v[d] * r
            R[0] -= D(fl, m[d])
            lor = []
            o = [q for q in range(3) if q != d]
            dB = {q: D(B[q], bs[q]) for q in o}
            cbb = [None, None, None]
            cbb[d] = -B[o[0]] * dB[o[0]] - B[o[1]] * dB[o[1]]
            for q in o:
                cbb[q] = B[d] * dB[q]
            for q in range(3):
                f, ms = fl * v[q], B[d] * B[q]
                if q == d:
                    f, ms = f + P, ms - pm
                lor.append(lf * D(ms, bs[d] * bs[q]) + (1.0 - lf) * cbb[q])
                R[1 + q] -= D(f, m[d] * m[q])
                R[1 + q] += lor[q]
                if q != d:
                    R[5 + q] -= D(v[d] * B[q] - v[q] * B[d], m[d] * bs[q])
            R[4] -= D(v[d] * ent, m[d])
            R[4] += v[0] * lor[0] + v[1] * lor[1] + v[2] * lor[2]
        # gravity and the Boris correction
        R[1] -= self.grav * r
        R[4] -= self.grav * r * v[0]
        bf = x2 * x2 / (1.0 + x2 + x2 * x2)
        F = [R[1 + q] - v[q] * R[0] for q in range(3)]
        q0 = (F[0] * B[0] + F[1] * B[1] + F[2] * B[2]) / bb.clamp(min=1e-100)
        for q in range(3):
            c = -bf * (F[q] - q0 * B[q])
            R[1 + q] += c
            R[4] += c * v[q]
        return R

    def tcheck(self, U):
        r = U[0].clamp(min=RHO_MIN)
        v = (U[1] ** 2 + U[2] ** 2 + U[3] ** 2).sqrt() / r
        s = V_LIM / v.clamp(min=V_LIM)
        k = 0.5 * r * v * v * s * s
        e = torch.minimum(torch.maximum(U[4], EPS_MIN * r + k), E_MAX * r + k)
        return [r, U[1] * s, U[2] * s, U[3] * s, e, U[5], U[6], U[7]]

    def tvd(self, U, P, d, dt):
        """One directional sweep; P: the pressure of the last stage's input."""
        axis, n = 2 - d, U[0].shape[2 - d]
        cmax, fac0 = 0.975 * self.dx / dt, 0.5 / self.dx
        q = [self.pad(U[v], axis, MIRROR[v]) for v in range(8)]
        p = self.pad(P, axis)
        shape = [1, 1, 1]
        hb = ht = 0.0
        if d == 0:  # the profiles are 1 in the ghost cells next to either end
            shape[2] = n + 4
            hb, ht = self.hb.view(shape), self.ht.view(shape)
        r = q[0].clamp(min=RHO_MIN)
        q[0] = r
        for c in (1, 2, 3):
            q[c] = q[c] / r
        vv = q[1] ** 2 + q[2] ** 2 + q[3] ** 2
        bb = q[5] ** 2 + q[6] ** 2 + q[7] ** 2
        q[4] = q[4] / r - 0.5 * vv
        x2 = bb / r * self.inv_va2
        lf = (1.0 + x2) / (1.0 + x2 + x2 * x2)
        c2 = 5.0 / 3.0 * p / r
        rf = torch.minimum(lf, r * r / (r * r + 1e-22))
        hh = 1.0 - hb - ht
        cf = 0.2 * hb + (rf * 0.2 + (1.0 - rf) * 0.2) * hh + 0.2 * ht
        c2 = c2 * cf * cf
        v1 = vv.sqrt()
        cm = v1 + torch.maximum(c2, lf * (c2 + bb / r)).sqrt()
        hyp = hb * 2.0 + (rf * 2.0 + (1.0 - rf) * 2.0) * hh + ht * 2.0
        bc = 1.0 - lf
        hd = fac0 * torch.minimum(v1, cmax - cm).clamp(min=0.0) if d == 0 else None
        q[0], q[4] = q[0].log(), q[4].log()
        del r, x2, lf, c2, rf, cf, v1, p

        def at(f, i, m):  # cells i .. i+m-1 along the axis
            return f.narrow(axis, i, m)

        fast = at(vv, 1, n + 2) > (0.75 * V_LIM) ** 2
        jump = (at(q[0], 1, n + 2) - at(q[0], 2, n + 2)).abs() > math.log(10.0)
        m = n + 1  # interfaces 1 .. n+1, between cells i and i+1
        fac = fac0 * torch.maximum(at(cm, 1, m), at(cm, 2, m)).clamp(max=cmax)
        h = at(hyp, 1, m)
        F, S = [], []
        for v in range(8):
            sl, sr = at(q[v], 1, n + 2) - at(q[v], 0, n + 2), at(q[v], 2, n + 2) - at(q[v], 1, n + 2)
            sm = 0.25 * (sl + sr)
            s = torch.minimum(torch.minimum(sl, sr), sm).clamp(min=0.0) + \
                torch.maximum(torch.maximum(sl, sr), sm).clamp(max=0.0)
            if v == 0:
                s = torch.where(jump, torch.zeros_like(s), s)
            if 1 <= v <= 3:
                s = torch.where(fast, torch.zeros_like(s), s)
            S.append(s if v < 5 else None)
            sa, sb = s.narrow(axis, 0, m), s.narrow(axis, 1, m)
            dq = at(q[v], 2, m) - at(q[v], 1, m)
            lim = dq - (sa + sb)
            ratio = lim.abs() / dq.abs().clamp(min=1e-100)
            c = torch.minimum(lim, dq).clamp(min=0.0) + torch.maximum(lim, dq).clamp(max=0.0)
            F.append((1.0 + h * (ratio - 1.0)).clamp(min=0.0) * c * fac)
        F[5 + d] = F[5 + d] * 0.2
        if d == 0:
            first = 0 if self.wrap else 2  # a closed x skips the interfaces next to its bottom
            for v in (0, 1, 4):
                w = torch.maximum(at(hd, 1, m), at(hd, 2, m))
                g = w * (0.125 * (at(q[v], 3, m) - at(q[v], 0, m)) - 0.375 * (at(q[v], 2, m) - at(q[v], 1, m)))
                g[..., :first] = 0.0
                F[v] = F[v] - g
        u = [0.5 * (at(q[v], 1, m) + S[v].narrow(axis, 0, m) + at(q[v], 2, m) - S[v].narrow(axis, 1, m))
             for v in range(5)]
        u[0], u[4] = u[0].exp(), u[4].exp()
        F[0] = F[0] * u[0]
        for c in (1, 2, 3):
            F[c] = F[c] * u[0] + u[c] * F[0]
        F[4] = F[4] * u[4] * u[0] + u[4] * F[0] + (u[1] * F[1] + u[2] * F[2] + u[3] * F[3])
        if d == 0 and not self.wrap:
            F[5][..., 0] = 0.0
            F[5][..., n] = 0.0
        heat = sum((at(q[v], 2, m) - at(q[v], 1, m)) * F[v] for v in (5, 6, 7))
        res = [dt * (F[v].narrow(axis, 1, n) - F[v].narrow(axis, 0, n)) for v in range(8)]
        B, vel, bcc = [at(q[v], 2, n) for v in (5, 6, 7)], [at(q[v], 2, n) for v in (1, 2, 3)], at(bc, 2, n)
        q0 = (res[1] * B[0] + res[2] * B[1] + res[3] * B[2]) / at(bb, 2, n).clamp(min=1e-100)
        b = [-bcc * (res[1 + c] - q0 * B[c]) for c in range(3)]
        for c in range(3):
            res[1 + c] = res[1 + c] + b[c]
            res[4] = res[4] + b[c] * vel[c]
        res[4] = res[4] + dt * 0.5 * (heat.narrow(axis, 1, n) + heat.narrow(axis, 0, n))
        out = [U[v] + res[v] for v in range(8)]
        out[0] = out[0].clamp(min=RHO_MIN)
        out[4] = torch.maximum(out[4], EPS_MIN * out[0] + 0.5 * (out[1] ** 2 + out[2] ** 2 + out[3] ** 2) / out[0])
        return out

    def step(self, U):
        U0 = [f.clone() for f in U]
        dt = None
        for stage in range(1, 5):
            P = self.pressure(U)
            if dt is None:
                dt = 0.8 * self.dx / self.cfl_speed(self.prim(U)[0], P)
            R = self.residual(U, P)
            w = dt / (5 - stage)
            U = self.tcheck([U0[v] + w * R[v] for v in range(8)])
            del R
        for d in range(3):
            U = self.tvd(U, P, d, dt)
        return self.tcheck(U)


def _exact_state(case, nx, ny, nz, seed, steps, **kw):
    """The state after `steps` steps from the records that prepare() hands in (rounded as they are there)."""
    setup = case["setup"]
    U = _state(setup, nx, ny, nz, seed, case["eos"], **kw)
    if case["precision"] == 32:
        U = U.float().double()
    ex = _Exact(setup, (nz, ny, nx), case["eos"], U.device)
    U = [U[v] for v in range(8)]
    for _ in range(steps):
        U = ex.step(U)
    return U


def exact(case, seed):
    kind, setup = case["kind"], case["setup"]
    if kind in ("physics", "adjoint"):
        return None
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "ensemble":
        parts = []
        for b, (bx, by, bz, v, g) in enumerate(_box_list(case)):
            U = _exact_state(case, bx, by, bz, seed * 1000 + b, case["steps"], v_rms=v, b_gauss=g)
            parts.append(torch.stack([f.reshape(-1) for f in _with_ghosts(U, setup)]).cpu())
        full = torch.cat(parts, 1)
        return {f: full[v] for v, f in enumerate(FIELDS)}
    if kind == "tiled":
        t = case["tile"]
        U = [f.repeat(t, t, 1) for f in _exact_state(case, nx, ny // t, nz // t, seed, case["steps"])]
    else:
        U = _exact_state(case, nx, ny, nz, seed, 1 if kind == "host" else case["steps"])
    return {f: x.reshape(-1).cpu() for f, x in zip(FIELDS, _with_ghosts(U, setup))}
