"""The work that users of this library have it do, as measurable cases.

Four kinds of call, each through the public Python binding of the C ABI:

* ``deriv``: one constant-Q derivative field of a device array through the
  allocation-free entry point (q_derivative_noalloc): forward and inverse 3D
  transforms of one field.  The smallest calls of the library, bound by
  launches and latency.
* ``steps``: a wavefield kept on the device (an in-HBM consumer writes and
  reads the fields where they are): the state is cleared, an initial particle
  velocity that fills the grid (as a wavefield in the middle of a shot does) is
  put in, and ``nt`` time steps of an iso or VTI medium follow.
* ``shot``: one shot of a shot loop from host arrays: model upload, receivers,
  source, clear, ``nt`` steps, seismograms back on the host.
* ``rtm``: one reverse-time-migrated shot from host arrays: two propagations,
  the records injected, two images back.

Sizes are those of the workloads in models.py, the tests and bench.py: the
96^3 cube with a 20-cell C-PML, the 256^3 and 512x512x256 VTI models with a
30-cell one, the batch grids (128^3 .. 256x256x192), the serving range (96..384
in x and y, 96..256 in z, iso and VTI alike), and the tests' small and odd
grids, whose lengths have factors 2, 3, 5 and 7.  ``exact`` restates the scheme in FP64 with
torch.fft, on full grids and with every transform of the formulation.
"""
import ctypes
import importlib.util
import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PI = 3.1415926  # the scheme's pi (viscoelas_3D.cpp:14)


def _load(name, file):
    spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "q-vti_b200", file))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


qvti = _load("qvti_b200", "qvti.py")
models = _load("qvti_models", "models.py")


# ------------------------------------------------------------------- cases --
def _case(kind, n, **kw):
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], **kw)


def listed():
    return [
        # one small field on a latency-critical path: five dependent passes
        dict(_case("deriv", (32, 48, 40), axis=1, fwd=True, power=1), name="deriv_32x48x40"),
        # the largest cube the fixed scratch admits
        dict(_case("deriv", (96, 96, 96), axis=0, fwd=True, power=-1), name="deriv_96"),
        # the tests' 32^3 cube: a whole short run of tiny steps
        dict(_case("steps", (32, 32, 32), pml=8, nt=120, vti=False, src=0), name="steps_iso_32"),
        # the small workload's cube, explosive source at the centre's depth
        dict(_case("steps", (96, 96, 96), pml=20, nt=60, vti=False, src=1), name="steps_iso_96"),
        # lengths with factors of 7, which have no compiled transform
        dict(_case("steps", (84, 112, 98), pml=12, nt=48, vti=True, src=0), name="steps_vti_84x112x98"),
        # odd smooth lengths of the serving range, every tile ragged
        dict(_case("steps", (150, 108, 120), pml=15, nt=32, vti=False, src=0), name="steps_iso_150x108x120"),
        # the smallest and most frequent batch grid
        dict(_case("steps", (128, 128, 128), pml=20, nt=32, vti=True, src=0), name="steps_vti_128"),
        # the headline model
        dict(_case("steps", (256, 256, 256), pml=30, nt=16, vti=True, src=0), name="steps_vti_256"),
        # the largest grid of the serving range
        dict(_case("steps", (384, 384, 256), pml=30, nt=8, vti=False, src=0), name="steps_iso_384x384x256"),
        # the precision workload's grid, the largest of all
        dict(_case("steps", (512, 512, 256), pml=30, nt=6, vti=True, src=0), name="steps_vti_512x512x256"),
        # one shot of a shot loop, host arrays in and out
        dict(_case("shot", (160, 160, 128), pml=20, nt=60, vti=True, src=0), name="shot_vti_160x160x128"),
        # one migrated shot, Q compensated
        dict(_case("rtm", (64, 80, 72), pml=10, nt=60, vti=False, src=0, media=4, every=5), name="rtm_64x80x72"),
    ]


def _smooth_lengths(lo, hi, primes):
    out = []
    for m in range(lo, hi + 1, 2):
        r = m
        for p in primes:
            while r % p == 0:
                r //= p
        if r == 1:
            out.append(m)
    return out


def _length(rng, lo, hi, primes=(2, 3, 5)):
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_smooth_lengths(lo, hi, primes), key=lambda m: abs(m - x))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choices(("deriv", "steps_small", "steps_serve", "shot", "rtm"), (2, 3, 4, 2, 1))[0]
    if kind == "deriv":
        while True:
            n = tuple(_length(rng, 16, 160, (2, 3, 5, 7)) for _ in range(3))
            if (n[2] // 2 + 1) * n[0] * n[1] <= 1 << 19:
                break
        return _case("deriv", n, axis=rng.randrange(3), fwd=rng.random() < 0.5, power=rng.choice((-1, 0, 1)))
    if kind == "steps_small":  # test sizes up to the small workload's, any supported length
        n = tuple(_length(rng, 32, 128, (2, 3, 5, 7)) for _ in range(3))
        return _case("steps", n, pml=rng.randint(6, 12), nt=rng.randint(24, 64), vti=rng.random() < 0.5,
                     src=rng.randrange(2))
    if kind == "steps_serve":
        n = (_length(rng, 96, 384), _length(rng, 96, 384), _length(rng, 96, 256))
        cells = n[0] * n[1] * n[2]
        return _case("steps", n, pml=rng.randint(16, 30), nt=max(6, min(32, int(2.5e8 / cells))),
                     vti=rng.random() < 0.5, src=rng.randrange(2))
    if kind == "shot":
        n = (_length(rng, 96, 224), _length(rng, 96, 224), _length(rng, 96, 192))
        cells = n[0] * n[1] * n[2]
        return _case("shot", n, pml=rng.randint(16, 24), nt=max(24, min(80, int(2.5e8 / cells))),
                     vti=rng.random() < 0.5, src=rng.randrange(2))
    n = tuple(_length(rng, 48, 96) for _ in range(3))
    return _case("rtm", n, pml=rng.randint(8, 12), nt=rng.randint(40, 80), vti=rng.random() < 0.5, src=0,
                 media=rng.choice((1, 2, 3, 4)), every=rng.randint(4, 8))


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _smooth_noise(n, corr_cells, gen):
    """Unit Gaussian random field of a Gaussian correlation length, clipped to
    three standard deviations."""
    w = torch.fft.rfftn(torch.randn(n, generator=gen, device="cuda"))
    s = corr_cells / 2.0
    k = [torch.fft.fftfreq(m, device="cuda") for m in n[:2]] + [torch.fft.rfftfreq(n[2], device="cuda")]
    f = [torch.exp(-2.0 * (math.pi * s) ** 2 * kk ** 2) for kk in k]
    w = w * f[0][:, None, None] * f[1][None, :, None] * f[2][None, None, :]
    g = torch.fft.irfftn(w, s=n)
    return ((g - g.mean()) / g.std()).clamp_(-3.0, 3.0)


FIELDS = ("velp", "vels", "rho", "gama_p", "gama_s", "eps", "delta")


def _model(case, seed):
    """Six layers, 5 % perturbations of 80 m correlation length, Q 30..200
    (models.layered_vti), as device arrays."""
    n = (case["nx"], case["ny"], case["nz"])
    prof = models.layered_profiles(n[2], seed)
    gen = _gen(seed)
    out = {}
    for name in ("velp", "vels", "rho", "qp", "qs") + (("eps", "delta") if case["vti"] else ()):
        p = torch.from_numpy(prof[name]).cuda()
        out[name] = (p[None, None, :] * (1.0 + 0.05 * _smooth_noise(n, 8.0, gen))).contiguous()
    for a, b in (("gama_p", "qp"), ("gama_s", "qs")):
        out[a] = (torch.atan(1.0 / out.pop(b).double()) / PI).float()
    return {k: out[k] for k in FIELDS if k in out}


def _shot(case, seed):
    """Spacing, time step, wavelet, source and receivers of a case."""
    rng = np.random.default_rng([int(seed), 7])
    n = (case["nx"], case["ny"], case["nz"])
    pml, nt, f0, d = case["pml"], case["nt"], 20.0, (10.0, 10.0, 10.0)
    prof = models.layered_profiles(n[2], seed)
    # the perturbed model's extremes bound the time step
    ext = {k: prof[k] * 1.15 for k in ("velp", "eps", "delta")}
    ext["gama_p"] = models.gamma_of_q(prof["qp"] * 0.85)
    dt, _, _ = models.choose_dt(ext, d, f0, 0.8e-3, vti=True)
    t = np.arange(nt) * dt - min(1.0 / f0, 0.5 * nt * dt)
    tau = (PI * f0 * t) ** 2
    wavelet = ((1.0 - 2.0 * tau) * np.exp(-tau)).astype(np.float32)
    src = (int(rng.integers(n[0] // 3, 2 * n[0] // 3)), int(rng.integers(n[1] // 3, 2 * n[1] // 3)),
           int(rng.integers(pml, max(pml + 1, n[2] // 2))))
    rx = np.arange(n[0], dtype=np.int32)
    if case["kind"] == "shot":  # every fourth surface point
        gx, gy = np.meshgrid(np.arange(0, n[0], 4), np.arange(0, n[1], 4), indexing="ij")
        rx, ry = gx.ravel().astype(np.int32), gy.ravel().astype(np.int32)
    else:  # a line
        ry = np.full(n[0], n[1] // 2, np.int32)
    return dict(n=n, pml=pml, nt=nt, f0=f0, d=d, dt=dt, wavelet=wavelet, src=src, r_iz=pml + 2, r_ix=rx, r_iy=ry)


def _observed(s, seed):
    """Records to migrate: a direct and a reflected arrival with moveout."""
    rng = np.random.default_rng([int(seed), 9])
    t = (np.arange(s["nt"]) * s["dt"])[:, None]
    off = 10.0 * np.abs(s["r_ix"] - s["src"][0])[None, :].astype(np.float64)
    obs = np.zeros((3, s["nt"], len(s["r_ix"])), np.float32)
    for c in range(3):
        for depth in (30.0, 120.0):
            at = 0.012 + np.sqrt(off ** 2 + depth ** 2) / 2500.0
            tau = (PI * 40.0 * (t - at)) ** 2
            obs[c] += (rng.uniform(0.2, 1.0) * (1.0 - 2.0 * tau) * np.exp(-tau)).astype(np.float32)
    return obs


def _initial(case, seed):
    """Three unit particle-velocity fields of 40 m correlation length."""
    gen = _gen(seed + 2)
    return [_smooth_noise((case["nx"], case["ny"], case["nz"]), 4.0, gen) for _ in range(3)]


class _Field:
    """A wavefield of a simulation where it lies, for torch; keeps the simulation."""

    def __init__(self, sim, which):
        self.sim = sim
        self.__cuda_array_interface__ = dict(shape=sim.shape, typestr="<f4", data=(sim.device_field(which), False),
                                             strides=None, version=2)


def _simulation(case, s):
    return qvti.Simulation(*s["n"], s["pml"], *s["d"], s["dt"], s["f0"], vti=case["vti"])


def prepare(case, seed):
    if case["kind"] == "deriv":
        n = (case["nx"], case["ny"], case["nz"])
        f = _smooth_noise(n, 3.0, _gen(seed)) + 0.05 * torch.randn(n, generator=_gen(seed + 1), device="cuda")
        return dict(case=case, f=f.contiguous(), out=torch.empty_like(f), n=n)
    s = _shot(case, seed)
    m = _model(case, seed)
    if case["kind"] == "steps":
        sim = _simulation(case, s)
        torch.cuda.synchronize()  # the model arrays are read on the simulation's stream
        sim.set_model_device([a.data_ptr() for a in m.values()])
        sim.set_receivers(s["r_iz"], s["r_ix"], s["r_iy"])
        sim.set_source(*s["src"], s["wavelet"], kind=case["src"])
        st = ctypes.c_void_p()
        if qvti.lib().qvti_get_stream(sim._h, ctypes.byref(st)):
            raise RuntimeError("qvti_get_stream")
        return dict(case=case, sim=sim, init=_initial(case, seed), stream=torch.cuda.ExternalStream(st.value),
                    fields=[torch.as_tensor(_Field(sim, i), device="cuda") for i in range(9)])
    host = {k: a.cpu().numpy() for k, a in m.items()}
    if case["kind"] == "shot":
        return dict(case=case, s=s, host=host, sim=_simulation(case, s))
    c = dict(host, ntx=s["n"][0], nty=s["n"][1], ntz=s["n"][2], pml=s["pml"], dx=s["d"][0], dy=s["d"][1],
             dz=s["d"][2], dt=s["dt"], f0=s["f0"], rik=s["wavelet"], s_ix=s["src"][0], s_iy=s["src"][1],
             s_iz=s["src"][2], r_iz=s["r_iz"], r_ix=s["r_ix"], r_iy=s["r_iy"])
    return dict(case=case, c=c, obs=_observed(s, seed))


def run(state):
    case = state["case"]
    if case["kind"] == "deriv":
        qvti.q_derivative_noalloc(state["f"].data_ptr(), state["out"].data_ptr(), state["n"], (10.0, 10.0, 10.0),
                                  case["axis"], case["fwd"], case["power"],
                                  stream=torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if case["kind"] == "steps":
        sim = state["sim"]
        sim.reset()
        with torch.cuda.stream(state["stream"]):
            for v, v0 in zip(state["fields"], state["init"]):
                v.copy_(v0)
        sim.step(case["nt"])
        return state["fields"]
    if case["kind"] == "shot":
        sim, s, h = state["sim"], state["s"], state["host"]
        sim.set_model(h["velp"], h["vels"], h["rho"], h["gama_p"], h["gama_s"], h.get("eps"), h.get("delta"))
        sim.set_receivers(s["r_iz"], s["r_ix"], s["r_iy"])
        sim.set_source(*s["src"], s["wavelet"], kind=case["src"])
        sim.reset()
        sim.step(s["nt"])
        return sim.records()
    return list(qvti.rtm_shot(state["c"], state["obs"], media=case["media"], snap_every=case["every"],
                              illum_eps=1e-2, vti=case["vti"], src_type=case["src"], ref_offset=False))


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes: each input and state array read once, each result written once,
    per step; flops: 5 N log2 N per complex transform (half for a real one)."""
    nx, ny, nz = n = (case["nx"], case["ny"], case["nz"])
    cells = nx * ny * nz
    lg = [math.log2(m) for m in n]
    fft3 = 2.5 * cells * sum(lg)
    if case["kind"] == "deriv":
        return dict(bytes=8.0 * cells, flops=2 * fft3 + 10.0 * cells)
    pml, nt = case["pml"], case["nt"]
    slab = [2.0 * pml * cells / m for m in n]  # C-PML cells per axis; 13, 13 and 11 variables
    state = 4.0 * (15 * cells + 13 * slab[0] + 13 * slab[1] + 11 * slab[2])
    model = 4.0 * cells * (7 if case["vti"] else 5)
    step_bytes = 2 * state + model
    # 3 forward and 27 inverse 3D transforms, 9 derivatives along one axis, updates
    step_flops = 30 * fft3 + 6 * 2.5 * cells * sum(lg) + 250.0 * cells
    if case["kind"] == "rtm":
        keep = nt // case["every"]
        return dict(bytes=2 * nt * step_bytes + keep * 12.0 * cells * 4, flops=2 * nt * step_flops)
    return dict(bytes=nt * step_bytes + state, flops=nt * step_flops)


# ------------------------------------------------------------------- FP64 --
def _axis_tables(n, d):
    """|k| and the staggered-shift multipliers i k e^{+-i k d/2} of one axis,
    the Nyquist bin reduced to its real part."""
    i = torch.arange(n, device="cuda")
    m = torch.where(i <= n // 2, i, n - i).double()
    sign = torch.where(i <= n // 2, 1.0, -1.0).double()
    sign[n // 2] = 0.0
    c = 2.0 * PI / n / d
    sn, cs = torch.sin(m * PI / n), torch.cos(m * PI / n)
    return c * m, torch.complex(-c * m * sn, sign * c * m * cs), torch.complex(c * m * sn, sign * c * m * cs)


def _along(v, axis):
    shape = [1, 1, 1]
    shape[axis] = -1
    return v.reshape(shape)


def _profiles(n, pml, d, f0):
    """C-PML a, b and their half-point averages."""
    amax = PI * f0
    om = 4.0 * 5000.0 * math.log(1.0 / float(np.float32(1e-2))) / (2.0 * pml * d)
    i = torch.arange(n, device="cuda")
    j = torch.minimum(i, n - 1 - i).double()
    inside = j < pml
    b = torch.where(inside, om * ((pml - 1 - j).clamp(min=0) / pml) ** 3, 0.0)
    a = torch.where(inside, amax * (j / (pml - 1)) ** 2, amax) + b
    half = lambda v: 0.5 * (v + torch.cat([v[1:], v[-1:]]))  # noqa: E731
    return a, b, half(a), half(b)


class _Exact:
    """The scheme in FP64: full grids, every derivative by its own transform."""

    def __init__(self, case, s, model, media=1):
        self.n, self.case, self.s = s["n"], case, s
        f32 = lambda v: float(np.float32(v))  # noqa: E731
        self.dt = f32(s["dt"])
        d, f0 = [f32(v) for v in s["d"]], f32(s["f0"])
        w0 = f32(2 * PI * f0)
        self.loss = {1: 1.0, 2: 0.0, 3: 0.0, 4: -1.0}[media]
        tab = [_axis_tables(self.n[a], d[a]) for a in range(3)]
        half = self.n[2] // 2 + 1
        self.full = [(t[1], t[2]) for t in tab]  # forward, backward, whole axes
        self.sh = [(_along(t[1][:half] if a == 2 else t[1], a), _along(t[2][:half] if a == 2 else t[2], a))
                   for a, t in enumerate(tab)]
        k2 = (_along(tab[0][0], 0) ** 2 + _along(tab[1][0], 1) ** 2 + _along(tab[2][0][:half], 2) ** 2)
        k2[0, 0, 0] = 1e-10
        self.k = k2.sqrt()
        self.prof = [[_along(v, a) for v in _profiles(self.n[a], s["pml"], d[a], f0)] for a in range(3)]
        m = {k: v.double() for k, v in model.items()}
        r, vp, vs = m["rho"], m["velp"], m["vels"]
        gp, gs = (torch.zeros_like(r), torch.zeros_like(r)) if media == 3 else (m["gama_p"], m["gama_s"])

        def qset(v, g):
            c = v * torch.cos(g * PI / 2.0)
            return [-r * c * g * w0, r * c * c, r * c ** 3 * g / w0, r * c * g * PI, r * c * c * g * g * PI / w0]

        sset, p33 = qset(vs, gs), qset(vp, gp)
        p11, p13 = p33, p33
        if case["vti"]:
            c33, c44 = r * vp * vp, r * vs * vs
            c13 = torch.sqrt((c33 - c44) * (c33 * (1 + 2 * m["delta"]) - c44)) - c44
            p11, p13 = qset(vp * torch.sqrt(1 + 2 * m["eps"]), gp), qset(torch.sqrt((c13 + 2 * c44) / r), gp)
        self.k11, self.k33 = p11, p33
        self.k12 = [a - 2 * b for a, b in zip(p11, sset)]
        self.k13 = [a - 2 * b for a, b in zip(p13, sset)]

        def corner(v):
            out = torch.zeros_like(v)
            acc = 0
            for x in (0, 1):
                for y in (0, 1):
                    for z in (0, 1):
                        acc = acc + v[x:self.n[0] - 1 + x, y:self.n[1] - 1 + y, z:self.n[2] - 1 + z]
            out[:-1, :-1, :-1] = 0.125 * acc
            return out

        self.mu = [corner(v) for v in sset]
        self.rinv = [2.0 / (r + r.roll(-1, a)) for a in range(3)]
        self.inside = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        self.inside[:-1, :-1, :-1] = 1.0
        zero = lambda: torch.zeros(self.n, dtype=torch.float64, device="cuda")  # noqa: E731
        self.v, self.p = [zero() for _ in range(3)], {k: zero() for k in ("xx", "yy", "zz", "xy", "xz", "yz")}
        self.phv, self.phs, self.prev = {}, {}, {}
        self.zero = zero

    def _mem(self, store, key, axis, half, term):
        """One C-PML memory variable advanced by its term."""
        a, b = self.prof[axis][2:] if half else self.prof[axis][:2]
        q = store.get(key)
        new = -self.dt * b * term if q is None else q + self.dt * (-a * q - b * term)
        store[key] = new * self.inside
        return store[key]

    def _d1(self, f, axis, fwd):
        T = _along(self.full[axis][0 if fwd else 1], axis)
        return torch.fft.ifft(torch.fft.fft(f, dim=axis) * T, dim=axis).real

    def step(self, w, inject=None):
        p, dt = self.p, self.dt
        # per velocity: (stress, axis, forward shift), averaged profile on the diagonal
        for c, terms in enumerate(((("xx", 0, 0), ("xy", 1, 1), ("xz", 2, 1)), (("xy", 0, 1), ("yy", 1, 0), ("yz", 2, 1)),
                                   (("xz", 0, 1), ("yz", 1, 1), ("zz", 2, 0)))):
            rhs = 0
            for st, ax, fw in terms:
                d = self._d1(p[st], ax, fw)
                rhs = rhs + d + self._mem(self.phv, (c, ax), ax, st in ("xx", "yy", "zz"), d)
            self.v[c] += dt * self.rinv[c] * rhs * self.inside
        spec = [torch.fft.rfftn(f) for f in self.v]

        def fields(name, c, axis, fwd):
            """The five fields of one derivative: |k|^-1, 1, |k| and the time
            derivatives of the first two."""
            X = spec[c] * self.sh[axis][0 if fwd else 1]
            S = [torch.fft.irfftn(X / self.k, s=self.n), torch.fft.irfftn(X, s=self.n),
                 torch.fft.irfftn(X * self.k, s=self.n)]
            old = self.prev.get(name)
            self.prev[name] = S[:2]
            rate = [self.loss / dt * (a if old is None else a - b) for a, b in zip(S, old or S)]
            return S + rate

        dot = lambda q, S: q[0] * S[0] + q[1] * S[1] + q[2] * S[2] + q[3] * S[3] + q[4] * S[4]  # noqa: E731
        X, Y, Z = fields("xx", 0, 0, 1), fields("yy", 1, 1, 1), fields("zz", 2, 2, 1)
        zx = dot(self.k13, Z)
        zx = zx + self._mem(self.phs, "zx", 2, False, zx)
        rows = {"xx": (self.k11, self.k12, zx), "yy": (self.k12, self.k11, zx), "zz": (self.k13, self.k13, None)}
        for st, (kx, ky, z) in rows.items():
            a, b = dot(kx, X), dot(ky, Y)
            if z is None:
                z = dot(self.k33, Z)
                z = z + self._mem(self.phs, "zz", 2, False, z)
            tot = a + self._mem(self.phs, ("x", st), 0, False, a) + b + self._mem(self.phs, ("y", st), 1, False, b) + z
            p[st] += dt * tot * self.inside
        del X, Y, Z, zx, rows
        for st, pair in (("xz", ((0, 2), (2, 0))), ("xy", ((0, 1), (1, 0))), ("yz", ((1, 2), (2, 1)))):
            tot = 0
            for c, ax in pair:
                d = dot(self.mu, fields((c, ax), c, ax, 0))
                tot = tot + d + self._mem(self.phs, (c, ax), ax, True, d)
            p[st] += dt * tot * self.inside
        if w is not None:
            at = tuple(self.s["src"])
            for f in ((p["xx"], p["yy"], p["zz"]) if self.case["src"] == 1 else (self.v[0],)):
                f[at] += w
        if inject is not None:
            rx, ry = (torch.from_numpy(self.s[k].astype(np.int64)).cuda() for k in ("r_ix", "r_iy"))
            for c in range(3):
                self.v[c][rx, ry, self.s["r_iz"]] += inject[c]

    def record(self):
        rx, ry = (torch.from_numpy(self.s[k].astype(np.int64)).cuda() for k in ("r_ix", "r_iy"))
        return torch.stack([v[rx, ry, self.s["r_iz"]] for v in self.v])


def exact(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "deriv":
        f = prepare(case, seed)["f"].double()
        tab = [_axis_tables(m, 10.0) for m in n]
        half = n[2] // 2 + 1
        k2 = _along(tab[0][0], 0) ** 2 + _along(tab[1][0], 1) ** 2 + _along(tab[2][0][:half], 2) ** 2
        k2[0, 0, 0] = 1e-10
        T = tab[case["axis"]][1 if case["fwd"] else 2]
        T = _along(T[:half] if case["axis"] == 2 else T, case["axis"])
        return torch.fft.irfftn(torch.fft.rfftn(f) * T * k2 ** (0.5 * case["power"]), s=n)
    s, m = _shot(case, seed), _model(case, seed)
    w = [float(v) for v in s["wavelet"]]
    if case["kind"] in ("steps", "shot"):
        e = _Exact(case, s, m)
        if case["kind"] == "steps":
            e.v = [f.double() for f in _initial(case, seed)]
        recs = []
        for v in w:
            e.step(v)
            if case["kind"] == "shot":
                recs.append(e.record())
        if case["kind"] == "shot":
            return torch.stack(recs, 1)
        return e.v + [e.p[k] for k in ("xx", "yy", "zz", "xy", "xz", "yz")]
    every, nt = case["every"], case["nt"]
    e, kept = _Exact(case, s, m, case["media"]), {}
    for t, v in enumerate(w):
        e.step(v)
        if (t + 1) % every == 0:
            kept[t] = [f.clone() for f in e.v]
    obs = torch.from_numpy(_observed(s, seed)).cuda().double()
    e = _Exact(case, s, m, case["media"])
    image, illum = e.zero(), e.zero()
    for j in range(nt):
        t = nt - 1 - j
        e.step(None, obs[:, t])
        if t in kept:
            for a, b in zip(kept[t], e.v):
                image += a * b
                illum += a * a
        if t <= min(kept):
            break
    return [image, image / (illum + float(np.float32(1e-2)) * illum.max())]
