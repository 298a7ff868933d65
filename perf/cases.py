"""The work that users of libdft_gb300 have it do, as measurable cases.

A case is a dict: `kind` (the calls made), the grid (`nx`, `ny`, `nz`, `step` in
bohr), `prec` (the grids' precision, "f64" or "f32"), `model` (the OT
functional: 0 plain, 1 kinetic correlation, 2 high density, 8 backflow, added),
`state` (the helium the call meets), `dt` (fs) in imaginary or real time, and
`steps` of one call.  Kinds:

  run        dftgpu_run: predict-correct steps between two outputs of a relaxation or a dynamics run
  loop       the same steps by libdft's separate calls, as its example drivers write them
  potential  dft_ot_potential alone
  propagate  one split-operator step in a given potential (FFT or Crank-Nicolson, moving frame or not)
  report     the energies, the chemical potential and the energy density written between steps
  adjoint    the gradient of an end-of-trajectory objective with respect to the external potential and psi_0

`exact` evaluates the same mathematics in FP64 with torch alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import libdft_gb300 as G

AUTOANG, AUTOK, AUTOFS, AUTOAMU = 0.529177210903, 3.1577502480407e5, 0.024188843265857, 1.0 / 1822.888486209
HELIUM_MASS = 4.002602 / AUTOAMU          # of the wave function
RHO0 = 0.0218360 * AUTOANG ** 3           # bulk liquid at zero pressure (bohr^-3)
MU0 = -7.149933 / AUTOK                   # its chemical potential
PREC = {"f64": G.FP64, "f32": G.FP32}


def _case(name, kind, shape, step, prec, model, state, dt, imag, steps=1, cn=False, k0=0.0):
    c = dict(kind=kind, nx=shape[0], ny=shape[1], nz=shape[2], step=step, prec=prec, model=model, state=state, dt=dt,
             imag=imag, steps=steps, cn=cn, k0=k0)
    return dict(c, name=name) if name else c


def listed():
    return [
        # libdft's imag_time driver as it stands: one step of its loop on its 64^3 grid, FP64 (the default)
        _case("loop_64_f64_plain", "loop", (64, 64, 64), 1.0, "f64", 0, "bubble", 10.0, True),
        # the same relaxation by the run call in FP32, twenty steps between two looks at it
        _case("run_64_f32_plain", "run", (64, 64, 64), 1.0, "f32", 0, "bubble", 10.0, True, 20),
        # a sound wave in the bulk liquid: real-time dynamics with the full functional, an ordinary grid
        _case("run_128_f32_full", "run", (128, 128, 128), 0.8, "f32", 9, "wave", 1.0, False, 10),
        # a nanodroplet's relaxation at the size that the benchmark is quoted on
        _case("run_256_f32_full", "run", (256, 256, 256), 0.8, "f32", 9, "droplet", 20.0, True, 4),
        # a vortex ring in a large box, short along its axis: the largest grid
        _case("run_512_f32_full", "run", (512, 512, 256), 0.6, "f32", 9, "ring", 0.5, False),
        # the droplet in FP64, the precision that results are checked in
        _case("run_256_f64_full", "run", (256, 256, 256), 0.8, "f64", 9, "droplet", 20.0, True),
        # a box that is no power of two, as a droplet's diameter asks for it
        _case("run_240_f32_full", "run", (240, 240, 240), 0.8, "f32", 9, "droplet", 20.0, True, 2),
        # the potential alone on a ragged grid with odd sides, FP64
        _case("pot_135_125_90_f64_full", "potential", (135, 125, 90), 0.8, "f64", 9, "ring", 0.0, False),
        # the 1-D bubble driver's grid, real time: the smallest work per launch
        _case("run_1d_4096_f64_full", "run", (1, 1, 4096), 0.2, "f64", 9, "wave", 1.0, False, 20),
        # the energies printed between steps, FP64
        _case("report_128_f64_kc", "report", (128, 128, 128), 0.8, "f64", 1, "bubble", 0.0, True),
        # one gradient of an optimal-control loop, FP64 (the precision that meets its accuracy target)
        _case("adjoint_64_f64_full", "adjoint", (64, 64, 64), 0.8, "f64", 9, "wave", 2.0, False, 4),
        # an impurity's or the liquid's step in a known potential
        _case("prop_256_f32", "propagate", (256, 256, 256), 0.8, "f32", 0, "droplet", 5.0, False),
    ]


USUAL = (16, 32, 48, 64, 96, 128, 160, 192, 240, 256)
SMOOTH = sorted(a * b * c for a in (1, 2, 4, 8, 16, 32, 64, 128, 256) for b in (1, 3, 9, 27, 81, 243) for c in (1, 5, 25, 125)
                if 8 <= a * b * c <= 400)


def _length(rng, want, even):
    """A grid length near `want`: half the time a usual one, else any 2^a 3^b 5^c (z is even)."""
    if rng.random() < 0.5:
        return min(USUAL, key=lambda n: abs(math.log(n / want)))
    near = [n for n in SMOOTH if 0.8 < n / want < 1.25 and not (even and n % 2)]
    return rng.choice(near) if near else min((n for n in SMOOTH if n % 2 == 0), key=lambda n: abs(n - want))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "loop", "potential", "propagate", "report", "adjoint"))
    prec = rng.choice(("f64", "f32")) if kind != "adjoint" else "f64"
    model = rng.choice((0, 1, 9, 9)) if kind != "loop" else rng.choice((0, 1, 3, 9))
    imag = rng.random() < 0.5
    if kind != "adjoint" and rng.random() < 0.1:                       # a 1-D effective grid
        nz = rng.choice([n for n in (256, 320, 384, 500, 512, 600, 768, 1000, 1024, 1250, 1536, 2000, 2048, 2160, 3000,
                                     3072, 3600, 4000, 4096)])
        shape, step, state = (1, 1, nz), rng.choice((0.2, 0.25, 0.5)), "wave"
    else:
        most = {"adjoint": 72, "report": 200}.get(kind, 256 if prec == "f32" else 192)
        side = math.exp(rng.uniform(math.log(20), math.log(most)))
        skew = [rng.uniform(-0.35, 0.35) for _ in range(2)]
        want = (side * math.exp(skew[0]), side * math.exp(skew[1]), side * math.exp(-skew[0] - skew[1]))
        shape = tuple(_length(rng, min(max(w, 12), 400), a == 2) for a, w in enumerate(want))
        step, state = rng.choice((0.6, 0.8, 1.0)), rng.choice(("droplet", "bubble") if imag else ("wave", "ring"))
    n = shape[0] * shape[1] * shape[2]
    steps = 1
    if kind == "run":
        steps = max(1, min(20, int(4e7 / n * (1.0 if prec == "f32" else 0.1))))
    elif kind == "adjoint":
        steps = rng.choice((2, 3, 4))
    dt = rng.choice((5.0, 10.0, 20.0)) if imag else rng.choice((0.5, 1.0, 2.0))
    cn, k0 = False, 0.0
    if kind == "propagate":
        cn, k0 = rng.random() < 0.3, rng.choice((0.0, 0.0, 0.05))
    return _case(None, kind, shape, step, prec, model, state, dt, imag, steps, cn, k0)


# ---------------------------------------------------------------------- inputs
def _axes(case, device, centre=(0.0, 0.0, 0.0)):
    ax = []
    for a, n in enumerate((case["nx"], case["ny"], case["nz"])):
        v = (torch.arange(n, dtype=torch.float64, device=device) - n // 2) * case["step"] - centre[a]
        ax.append(v.reshape([-1 if b == a else 1 for b in range(3)]))
    return ax


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _inputs(case, seed):
    """psi, the external potential (or None) and the adjoint's target density, in the grids' precision."""
    dev = _device()
    rng = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 17)
    u = torch.rand(8, dtype=torch.float64, device="cpu", generator=torch.Generator().manual_seed(int(seed) * 104729 + 3)).tolist()
    shape, h = (case["nx"], case["ny"], case["nz"]), case["step"]
    box = [n * h for n in shape if n > 1]
    X, Y, Z = _axes(case, dev, [(u[a] - 0.5) * h if shape[a] > 1 else 0.0 for a in range(3)])
    noise = 1.0 + 1e-3 * torch.randn(shape, dtype=torch.float64, device=dev, generator=rng)
    vext = None
    if case["state"] == "droplet":      # a free droplet with a 1.5 bohr surface
        r = torch.sqrt(X * X + Y * Y + Z * Z)
        psi = torch.sqrt(0.5 * RHO0 * (1.0 - torch.tanh((r - (0.25 + 0.02 * u[3]) * min(box)) / 1.5))) * noise
        psi = psi.to(torch.complex128)
    elif case["state"] == "bubble":     # the liquid around a repulsive Gaussian impurity
        r2 = X * X + Y * Y + Z * Z
        psi = (math.sqrt(RHO0) * (1.0 - torch.exp(-r2 / 50.0)) * noise).to(torch.complex128)
        vext = (8.0 + 4.0 * u[3]) / AUTOK * torch.exp(-r2 / 18.0)
    elif case["state"] == "wave":       # a 1 % density wave along the longest axis
        a = max(range(3), key=lambda i: shape[i])
        k = 2.0 * math.pi * max(1, shape[a] // 32) / (shape[a] * h)
        psi = torch.sqrt(RHO0 * (1.0 + 0.01 * torch.cos(k * (X, Y, Z)[a] + 6.0 * u[3]))) * noise
        psi = psi.to(torch.complex128)
    else:                               # a vortex ring about the z axis
        rc = torch.sqrt(X * X + Y * Y)
        R = (0.12 + 0.02 * u[3]) * min(box)
        d = torch.sqrt((rc - R) ** 2 + Z * Z)
        psi = math.sqrt(RHO0) * torch.tanh(d) * noise * torch.exp(1j * torch.atan2(Z.expand(shape), (rc - R).expand(shape)))
    if case["kind"] == "adjoint" and vext is None:
        vext = 2.0 / AUTOK * torch.exp(-((X / box[0]) ** 2 + (Y / box[1]) ** 2 + (Z / box[2]) ** 2) * 40.0)
    pot = None
    if case["kind"] == "propagate":     # a potential of the liquid's size, with the small imaginary part that backflow has
        w = torch.cos(2 * math.pi * X / box[0] + 6 * u[4]) * torch.cos(2 * math.pi * Z / box[-1] + 6 * u[5])
        pot = torch.complex((w * noise) * 10.0 / AUTOK, (w * w).expand(shape) * 0.1 / AUTOK)
    target = (psi.abs() ** 2 * 1.01).expand(shape) if case["kind"] == "adjoint" else None
    real, cplx = (torch.float64, torch.complex128) if case["prec"] == "f64" else (torch.float32, torch.complex64)

    def put(x, t):
        return None if x is None else x.expand(shape).to(t).contiguous()

    return put(psi, cplx), put(vext, real), put(pot, cplx), put(target, real)


class _Handles:
    """The library's objects of one program, freed with it."""

    def __init__(self):
        self.all = []

    def keep(self, x):
        self.all.append(x)
        return x

    def __del__(self):
        for x in reversed(self.all):
            x.free()


class _Memory:
    """A grid's device memory for torch; keeps the grid alive."""

    def __init__(self, handles, address, shape, kind):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (address, False), "version": 3, "strides": None}


def _tensor(handles, case, grid, cplx):
    """The values of a cgrid / rgrid (its struct starts with their device address) as a tensor on the same memory."""
    address = C.cast(grid, C.POINTER(C.c_void_p))[0]
    size = (8 if case["prec"] == "f64" else 4) * (2 if cplx else 1)
    return torch.as_tensor(_Memory(handles, address, (case["nx"], case["ny"], case["nz"]), "<%s%d" % ("c" if cplx else "f", size)),
                           device="cuda")


def prepare(case, seed):
    torch.cuda.init()
    G.check(G.lib().dftgpu_init(0), "dftgpu_init")
    psi, vext, pot, target = _inputs(case, seed)
    shape, h, kind = (case["nx"], case["ny"], case["nz"]), case["step"], case["kind"]
    H = _Handles()
    S = {"case": case, "handles": H}
    G.set_precision(PREC[case["prec"]])
    w = S["wf"] = H.keep(G.Wf(shape, h, propagator=G.WF_2ND_ORDER_CN if case["cn"] else G.WF_2ND_ORDER_FFT))
    S["psi"] = _tensor(H, case, w.grid_ptr, True)
    S["psi"].copy_(psi)
    w.norm_target = float((psi.abs().to(torch.float64) ** 2).sum()) * h ** 3
    S["vext"] = S["P"] = S["ot"] = None
    if vext is not None:
        S["vext"] = H.keep(G.RGrid(shape, h))
        _tensor(H, case, S["vext"].ptr, False).copy_(vext)
    if kind != "propagate":
        S["ot"] = H.keep(G.OT(case["model"], w))
    if kind in ("run", "loop", "potential", "propagate"):
        S["P"] = H.keep(G.CGrid(shape, h))
        S["pot"] = _tensor(H, case, S["P"].ptr, True)
    if kind in ("run", "loop"):
        S["wfp"] = H.keep(G.Wf(shape, h))
    if kind == "propagate":
        S["pot"].copy_(pot)
        if case["k0"]:
            w.set_momentum(case["k0"], -case["k0"], 0.5 * case["k0"])
    if kind == "report":
        S["ed"] = H.keep(G.RGrid(shape, h))
        S["edv"] = _tensor(H, case, S["ed"].ptr, False)
    if kind == "adjoint":
        S["psi0"], S["gpsi"] = H.keep(G.CGrid(shape, h)), H.keep(G.CGrid(shape, h))
        S["target"], S["gvext"] = H.keep(G.RGrid(shape, h)), H.keep(G.RGrid(shape, h))
        _tensor(H, case, S["psi0"].ptr, True).copy_(psi)
        _tensor(H, case, S["target"].ptr, False).copy_(target)
        S["gpsiv"], S["gvextv"] = _tensor(H, case, S["gpsi"].ptr, True), _tensor(H, case, S["gvext"].ptr, False)
    G.set_precision(G.FP64)
    torch.cuda.synchronize()
    return S


def _dt(case):
    return (-1j if case["imag"] else 1.0 + 0j) * case["dt"] / AUTOFS


def run(S):
    case, w, ot, P, vext, L = S["case"], S["wf"], S["ot"], S["P"], S["vext"], G.lib()
    kind, dt = case["kind"], _dt(case)
    if kind == "run":
        ot.run(w, S["wfp"], P, vext, MU0, dt, case["steps"], case["imag"])
        return [S["psi"]]
    if kind == "loop":        # examples/imag_time/imag_time.c:229-240 of libdft
        for _ in range(case["steps"]):
            if vext:
                L.grid_real_to_complex_re(P.ptr, vext.ptr)
            else:
                P.zero()
            ot.potential(P, w)
            L.cgrid_add(P.ptr, -MU0, 0.0)
            w.predict(S["wfp"], P, dt)
            if vext:
                L.grid_add_real_to_complex_re(P.ptr, vext.ptr)
            ot.potential(P, S["wfp"])
            L.cgrid_add(P.ptr, -MU0, 0.0)
            L.cgrid_multiply(P.ptr, 0.5, 0.0)
            w.correct(P, dt)
            if case["imag"]:
                w.normalize()
        return [S["psi"]]
    if kind == "potential":
        P.zero()
        ot.potential(P, w)
        return [S["pot"]]
    if kind == "propagate":
        w.propagate(P, dt)
        return [S["psi"]]
    if kind == "report":
        ot.energy_density(S["ed"], w)
        e, n, mu = ot.energy_report(w, vext)
        return [S["edv"], np.array([e, n, mu], np.float64 if case["prec"] == "f64" else np.float32)]
    L.cgrid_copy(w.grid_ptr, S["psi0"].ptr)
    J = ot.adjoint_run(w, vext, MU0, dt, case["steps"], case["imag"], S["target"], S["gvext"], S["gpsi"])
    return [S["gvextv"], S["gpsiv"], S["psi"], np.array([J], np.float64 if case["prec"] == "f64" else np.float32)]


# ---------------------------------------------------------------------- work
def _transforms(model):
    """Real 3-D transforms of one potential: forward and inverse, one per field that has to cross."""
    return 4 + (8 if model & 1 else 0) + (8 if model & 8 else 0)


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    size = 8 if case["prec"] == "f64" else 4
    log = math.log2(max(2, n))
    real, cplx = 2.5 * n * log, 5.0 * n * log          # operations of a transform
    pot = _transforms(case["model"]) * real + n * (40 + (60 if case["model"] & 1 else 0) + (90 if case["model"] & 8 else 0))
    prop = 2 * cplx + 40 * n
    psi = 2 * n * size
    fields = n * size if case["state"] == "bubble" else 0
    step = 2 * (pot + prop)
    if case["kind"] in ("run", "loop"):
        return {"bytes": 2 * psi + fields, "flops": case["steps"] * step}
    if case["kind"] == "potential":
        return {"bytes": 2 * psi, "flops": pot}
    if case["kind"] == "propagate":
        return {"bytes": 3 * psi, "flops": prop}
    if case["kind"] == "report":                       # energy density, potential, kinetic energy
        return {"bytes": psi + n * size + fields, "flops": 2 * pot + cplx}
    # adjoint: forward, recomputed and reverse steps; psi_0, the target and Vext in, both gradients and psi_T out
    return {"bytes": 3 * psi + 3 * n * size, "flops": 4 * case["steps"] * step}


# ---------------------------------------------------------------------- the same in 64 bits
class _OT:
    """The Orsay-Trento functional's parameters (atomic units) and its kernels' spectra on a case's grid."""

    def __init__(self, case):
        a3 = AUTOANG ** 3
        self.case, self.model, self.h = case, case["model"], case["step"]
        self.shape = (case["nx"], case["ny"], case["nz"])
        self.dev = _device()
        self.dv = self.h ** 3
        self.b, self.c2, self.c3 = -718.99 / (AUTOK * a3), -2.411857e4 / (AUTOK * a3 ** 2), 1.858496e6 / (AUTOK * a3 ** 3)
        self.mass, self.rho_0s, self.alpha_s = 4.0026 / AUTOAMU, 0.04 * a3, 54.31 / a3
        self.eps = 1e-4
        self.beta, self.rhom, self.C = 40.0 / a3, 0.37 * a3, 0.1
        if case["kind"] != "propagate":
            self._kernels()

    def _average(self, f, x, y, z, ns):
        """Averages of f over the cells about the points, ns^3 sub-points each."""
        off = ((torch.arange(ns, dtype=torch.float64, device=self.dev) + 0.5) / ns - 0.5) * self.h
        out, per = [], max(1, int(3e7 // ns ** 3))
        for i in range(0, x.numel(), per):
            xs = (x[i:i + per, None] + off)[:, :, None, None]
            ys = (y[i:i + per, None] + off)[:, None, :, None]
            zs = (z[i:i + per, None] + off)[:, None, None, :]
            out.append(f(xs, ys, zs).expand(-1, ns, ns, ns).sum(dim=(1, 2, 3)) / ns ** 3)
        return torch.cat(out)

    def _spectrum(self, f):
        """Cell averages about the grid points, sub-points doubled from 4 to at most 32 until they change by less than
        0.01 K; sampled on the octant of distances from the centre, which all the kernels are even about."""
        half = [torch.arange(n // 2 + 1, dtype=torch.float64, device=self.dev) * self.h for n in self.shape]
        x, y, z = (g.reshape(-1) for g in torch.meshgrid(*half, indexing="ij"))
        v = self._average(f, x, y, z, 4)
        open_, ns = torch.arange(x.numel(), device=self.dev), 4
        while 2 * ns <= 32 and open_.numel():
            ns *= 2
            v2 = self._average(f, x[open_], y[open_], z[open_], ns)
            more = (v2 - v[open_]).abs() >= 0.01 / AUTOK
            v[open_] = v2
            open_ = open_[more]
        v = v.reshape([n // 2 + 1 for n in self.shape])
        for a, n in enumerate(self.shape):               # about index 0, periodic
            i = torch.arange(n, device=self.dev)
            v = v.index_select(a, torch.minimum(i, n - i))
        return torch.fft.rfftn(v).real.contiguous()

    def _kernels(self):
        sig, lj_e, core = 2.556 / AUTOANG, 10.22 / AUTOK, 2.1903 / AUTOANG
        iw = AUTOANG                                      # 1 / l_g, l_g = 1 Angstrom
        g11, g12, a1 = -19.7544, 12.5616 * AUTOANG ** 2, 1.023 * AUTOANG ** 2
        g21, g22, a2 = -0.2395, 0.0312 * AUTOANG ** 2, 0.14912 * AUTOANG ** 2
        one_d = self.shape[0] == self.shape[1] == 1

        def lj(x, y, z):
            if one_d:
                a = z.abs().clamp(min=core)
                return 2 * math.pi * lj_e * sig ** 6 * (2 * sig ** 6 - 5 * a ** 6) / (5 * a ** 10)
            r2 = x * x + y * y + z * z
            s6 = (sig * sig / r2) ** 3
            return torch.where(r2 <= core * core, torch.zeros_like(r2), 4 * lj_e * s6 * (s6 - 1.0))

        def ball(x, y, z):
            if one_d:
                return torch.where(z.abs() > core, torch.zeros_like(z), 3 * (core ** 2 - z * z) / (4 * core ** 3))
            r2 = x * x + y * y + z * z
            return torch.where(r2 <= core * core, 3 / (4 * math.pi * core ** 3), 0.0).to(torch.float64)

        def gauss(x, y, z):
            if one_d:
                return iw / math.sqrt(math.pi) * torch.exp(-z * z * iw * iw)
            return iw ** 3 / math.pi ** 1.5 * torch.exp(-(x * x + y * y + z * z) * iw * iw)

        def flow(x, y, z):
            if one_d:
                z2 = z * z
                return math.pi * ((g11 + g12 * (1 + a1 * z2) / a1) * torch.exp(-a1 * z2) / a1
                                  + (g21 + g22 * (1 + a2 * z2) / a2) * torch.exp(-a2 * z2) / a2)
            r2 = x * x + y * y + z * z
            return (g11 + g12 * r2) * torch.exp(-a1 * r2) + (g21 + g22 * r2) * torch.exp(-a2 * r2)

        dv = self.h if one_d else self.dv
        self.lj, self.sa = self._spectrum(lj), self._spectrum(ball)
        self.lj = self.lj * (dv if one_d else self.b / self.lj.flatten()[0])   # 3-D: integrals b and 1
        self.sa = self.sa * (dv if one_d else 1.0 / self.sa.flatten()[0])
        self.f = self._spectrum(gauss) * dv if self.model & 1 else None
        self.vj = self._spectrum(flow) * dv if self.model & 8 else None

    def conv(self, k, f):
        return torch.fft.irfftn(k * torch.fft.rfftn(f), s=self.shape)

    def d(self, f, a):
        return (torch.roll(f, -1, a) - torch.roll(f, 1, a)) / (2 * self.h)

    def velocity(self, psi, eps):
        rho = (psi.real ** 2 + psi.imag ** 2).clamp(min=eps)
        return [(psi.conj() * self.d(psi, a)).imag / (HELIUM_MASS * rho) for a in range(3)]

    def potential(self, psi):
        rho = psi.real ** 2 + psi.imag ** 2
        rb = self.conv(self.sa, rho)
        v = self.conv(self.lj, rho) + self.c2 / 2 * rb ** 2 + self.c3 / 3 * rb ** 3
        v = v + self.conv(self.sa, (self.c2 * rb + self.c3 * rb ** 2) * rho)
        im = torch.zeros_like(v)
        if self.model & 2:
            t = self.beta * (rho - self.rhom)
            v = v + self.C * (1 + torch.tanh(t)) + self.C * self.beta * rho / torch.cosh(t) ** 2
        if self.model & 1:
            c = self.alpha_s / (2 * self.mass)
            rt = self.conv(self.f, rho)
            st, h = 1 - rt / self.rho_0s, 0.0
            for a in range(3):
                g = self.d(rho, a)
                j = self.conv(self.f, g * st)
                v = v + c * (st * self.d(j, a) - j * self.d(rt, a))
                h = h + g * j
            v = v + c * self.conv(self.f, h)
        if self.model & 8:
            vel = self.velocity(psi, self.eps)
            A, v2 = self.conv(self.vj, rho), sum(u * u for u in vel)
            B = [self.conv(self.vj, rho * u) for u in vel]
            v = v - 0.5 * self.mass * (A * v2 - 2 * sum(u * b for u, b in zip(vel, B)) + self.conv(self.vj, rho * v2))
            for a in range(3):
                w = vel[a] * A - B[a]
                im = im + 0.5 * (self.d(rho, a) / rho.clamp(min=self.eps) * w + self.d(w, a))
        return torch.complex(v, im)

    def energy_density(self, psi):
        rho = psi.real ** 2 + psi.imag ** 2
        rb = self.conv(self.sa, rho)
        e = 0.5 * rho * self.conv(self.lj, rho) + self.c2 / 2 * rb ** 2 * rho + self.c3 / 3 * rb ** 3 * rho
        if self.model & 2:
            e = e + self.C * rho * (1 + torch.tanh(self.beta * (rho - self.rhom)))
        if self.model & 1:
            st = 1 - self.conv(self.f, rho) / self.rho_0s
            for a in range(3):
                g = self.d(rho, a)
                e = e - self.alpha_s / (4 * self.mass) * self.conv(self.f, g * st) * g * st
        if self.model & 8:
            vel = self.velocity(psi, self.eps)
            v2 = sum(u * u for u in vel)
            e = e - self.mass / 4 * rho * (self.conv(self.vj, rho) * v2 + self.conv(self.vj, rho * v2))
            e = e + self.mass / 2 * rho * sum(u * self.conv(self.vj, rho * u) for u in vel)
        return e

    def _k(self, a):
        n = self.shape[a]
        k0 = (self.case["k0"], -self.case["k0"], 0.5 * self.case["k0"])[a]
        k = 2 * math.pi * torch.fft.fftfreq(n, self.h, dtype=torch.float64, device=self.dev) - k0
        return k.reshape([-1 if b == a else 1 for b in range(3)])

    def propagate(self, psi, pot, dt):
        half = torch.exp(-0.5j * dt * pot)
        f = torch.fft.fftn(half * psi)
        for a in range(3):
            if self.case["cn"]:
                q = -0.5j * dt / HELIUM_MASS * (2 * torch.sin(0.5 * self.h * self._k(a)) / self.h) ** 2
                f = f * ((1 + 0.5 * q) / (1 - 0.5 * q))
            else:
                f = f * torch.exp(-0.5j * dt / HELIUM_MASS * self._k(a) ** 2)
        return half * torch.fft.ifftn(f)

    def step(self, psi, vext, norm):
        dt = _dt(self.case)
        v1 = self.potential(psi) + vext - MU0
        v2 = 0.5 * (v1 + self.potential(self.propagate(psi, v1, dt)) + vext - MU0)
        psi = self.propagate(psi, v2, dt)
        if norm is not None:
            psi = psi * torch.sqrt(norm / ((psi.real ** 2 + psi.imag ** 2).sum() * self.dv))
        return psi

    def kinetic(self, psi):
        s = torch.fft.fftn(psi)
        k2 = sum(self._k(a) ** 2 for a in range(3))
        return (k2 * (s.real ** 2 + s.imag ** 2)).sum() / (2 * HELIUM_MASS) * self.dv / psi.numel()


def exact(case, seed):
    n, kind = case["nx"] * case["ny"] * case["nz"], case["kind"]
    if n * (1 if kind == "propagate" else case["steps"]) > 8e7:
        return None
    psi, vext, pot, target = _inputs(case, seed)
    psi = psi.to(torch.complex128)
    norm = float((psi.abs() ** 2).sum()) * case["step"] ** 3 if case["imag"] else None
    vext = vext.to(torch.float64) if vext is not None else torch.zeros((), dtype=torch.float64, device=psi.device)
    ot = _OT(case)
    if kind == "propagate":
        return [ot.propagate(psi, pot.to(torch.complex128), _dt(case))]
    if kind == "potential":
        return [ot.potential(psi)]
    if kind == "report":
        rho, ed = psi.real ** 2 + psi.imag ** 2, ot.energy_density(psi)
        ekin, evx, atoms = ot.kinetic(psi), (rho * vext).sum() * ot.dv, rho.sum() * ot.dv
        mu = (ekin + (rho * ot.potential(psi).real).sum() * ot.dv + evx) / atoms
        return [ed, np.array([float(ekin + ed.sum() * ot.dv + evx), float(atoms), float(mu)])]
    if kind in ("run", "loop"):
        for _ in range(case["steps"]):
            psi = ot.step(psi, vext, norm)
        return [psi]
    psi0, vext = psi.clone().requires_grad_(True), vext.clone().requires_grad_(True)
    end = psi0
    for _ in range(case["steps"]):
        end = ot.step(end, vext, norm)
    J = ((end.real ** 2 + end.imag ** 2 - target.to(torch.float64)) ** 2).sum() * ot.dv
    J.backward()
    return [vext.grad, psi0.grad, end.detach(), np.array([J.item()])]
