"""Performance cases: the work a program has the engine do, through its public API.

A propagation program keeps one handle per shot (grid, model, sources and
receivers resident on the GPU) and drives it in three ways, all measured here:

  modelling  advance a running shot by `steps` time steps, recording the
             receivers (Propagator.modelling, then the traces on the host);
  rtm        one whole reverse-time-migration shot (Propagator.rtm_shot):
             forward pass storing snapshots, backward pass injecting the
             recorded gather with the imaging condition, image on the host;
  batch      many small shots stepped together (Batch.modelling);

and `codec` encodes and decodes one wavefield snapshot with the learned
compressor (AutoEncoder's library calls on device memory).

`exact` is the same propagation in 64 bits in plain torch: finite differences,
compact-FD lines as dense banded solves, transform engines as dense line
matrices, the PML recursion, the acoustic VTI / TTI scaling, the
visco-acoustic memory variables, separable injection / extraction and the
zero-lag image.
"""
import ctypes as C
import math

import numpy as np
import torch

from konglong_b200 import compressor as AE
from konglong_b200 import spec as S
from konglong_b200 import workloads as W
from konglong_b200.propagator import Batch, Propagator, spread_coeffs

ENGINE = {"fd8": S.ENGINE_FD8, "cfd": S.ENGINE_CFD, "r2c": S.ENGINE_R2C, "r2r": S.ENGINE_R2R}
MODEL = {"iso": S.ISO, "vti": S.VTI, "tti": S.TTI}
SNAP = {"fp32": S.SNAP_FP32, "c16": S.SNAP_C16, "fp16s": S.SNAP_FP16S}
DEV = "cuda" if torch.cuda.is_available() else "cpu"
VMIN, VMAX, EPS_MAX, DEL_MAX = 1500.0, 4500.0, 0.25, 0.10


# --- the cases ------------------------------------------------------------------
def _shot(kind, engine, model, nx, ny, nz, pml, steps, nrec, **more):
    return dict(kind=kind, engine=engine, model=model, nx=nx, ny=ny, nz=nz, pml=pml, steps=steps, nrec=nrec,
                q=False, q_bf16=False, **more)


def listed():
    cases = []

    def add(name, case, **kw):
        cases.append(dict(case, name=name, **kw))

    # a 2-D line shot: the smallest grid the engine is used on, all launch latency
    add("iso_2d_line", _shot("modelling", "fd8", "iso", 601, 1, 300, 20, 50, 60))
    # the 128^3 isotropic shot (64 x 64 receivers, PML 20): every array fits in L2
    add("iso_128", _shot("modelling", "fd8", "iso", 128, 128, 128, 20, 100, 64))
    # isotropic production grid
    add("iso_512", _shot("modelling", "fd8", "iso", 512, 512, 400, 32, 24, 64))
    # VTI on the FD8 engine, a mid-size aperture with uneven extents
    add("vti_fd8", _shot("modelling", "fd8", "vti", 330, 283, 260, 24, 20, 48))
    # the headline workload: VTI, compact FD, 512 x 512 x 400, 256 x 256 receivers
    add("vti_cfd_512", _shot("modelling", "cfd", "vti", 512, 512, 400, 32, 10, 256))
    # a whole compact-FD RTM shot on a small odd grid (nz not a multiple of 4), COMPRESS_16 snapshots
    add("vti_cfd_rtm_odd", _shot("rtm", "cfd", "vti", 199, 163, 150, 16, 40, 48, snap="c16", interval=4))
    # visco-acoustic TTI, FP32 memory variables
    add("tti_q", dict(_shot("modelling", "fd8", "tti", 400, 400, 320, 32, 10, 64), q=True))
    # a whole mixed-precision TTI + Q RTM shot: BF16 memory variables, FP16 snapshots
    add("tti_q_rtm_mixed", dict(_shot("rtm", "fd8", "tti", 232, 220, 200, 20, 32, 48, snap="fp16s", interval=8),
                                q=True, q_bf16=True))
    # pseudo-spectral engines: cosine / sine lines and Fourier lines
    add("vti_r2r", _shot("modelling", "r2r", "vti", 256, 256, 200, 16, 16, 48))
    add("vti_r2c", _shot("modelling", "r2c", "vti", 300, 260, 220, 20, 12, 48))
    # many small isotropic shots of uneven aperture in one batch
    cases.append(dict(name="batch_iso", kind="batch", shots=12, lo=96, hi=160, steps=60, nrec=16, pml=16))
    # one snapshot through the learned compressor, encode and decode
    cases.append(dict(name="ae_codec", kind="codec", nx=400, ny=400, nz=320))
    return cases


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, cells, z4, even=False, top=512):
    """Extents of about `cells` cells with uneven aspect; z4: nz a multiple of 4."""
    e = cells ** (1 / 3)
    n = [min(top, max(48, int(e * _log(rng, 0.8, 1.25)))) for _ in range(3)]
    if even:  # the Fourier engine's gradient grows on lines of odd length
        return [n[0] // 2 * 2, n[1] // 2 * 2, n[2] // 4 * 4 - (0 if z4 else 2)]
    return [n[0], n[1], n[2] // 4 * 4 - (0 if z4 else 1)]


def draw(rng):
    what = rng.choice(["line", "iso", "iso", "vti_fd8", "vti_cfd", "vti_cfd", "tti_q", "spectral", "cfd_rtm", "q_rtm",
                       "batch", "codec"])
    z4 = rng.random() < 0.7
    if what == "line":
        return _shot("modelling", "fd8", "iso", int(_log(rng, 200, 1500)), 1,
                     int(_log(rng, 60, 250)) * 4, rng.randint(12, 24), rng.randint(20, 60), 60)
    if what == "batch":
        lo = rng.randint(64, 110)
        return dict(kind="batch", shots=rng.randint(4, 14), lo=lo, hi=lo + rng.randint(16, 60), steps=rng.randint(24, 60),
                    nrec=16, pml=rng.randint(10, 18))
    if what == "codec":
        nx, ny, nz = _grid(rng, _log(rng, 1e6, 4.5e7), False)
        return dict(kind="codec", nx=nx, ny=ny, nz=nz)
    top = {"iso": 9e7, "vti_fd8": 5e7, "vti_cfd": 8e7, "tti_q": 4e7, "spectral": 2.5e7, "cfd_rtm": 8e6, "q_rtm": 1.2e7}
    nx, ny, nz = _grid(rng, _log(rng, 4e5, top[what]), z4, even=what == "spectral")
    cells = nx * ny * nz
    pml = max(8, min(32, min(nx, ny, nz) // rng.randint(7, 14)))
    steps = int(max(8, min(60, 8e8 / cells)))
    nrec = rng.randint(16, 64)
    if what == "iso":
        return _shot("modelling", "fd8", "iso", nx, ny, nz, pml, steps, nrec)
    if what == "vti_fd8":
        return _shot("modelling", "fd8", "vti", nx, ny, nz, pml, steps, nrec)
    if what == "vti_cfd":
        return _shot("modelling", "cfd", "vti", nx, ny, nz, pml, max(4, steps // 2), nrec)
    if what == "tti_q":
        return dict(_shot("modelling", "fd8", "tti", nx, ny, nz, pml, steps, nrec), q=True, q_bf16=rng.random() < 0.3)
    if what == "spectral":
        return _shot("modelling", rng.choice(["r2r", "r2c"]), "vti", nx, ny, nz, pml, max(4, steps // 2), nrec)
    if what == "cfd_rtm":
        return _shot("rtm", "cfd", "vti", nx, ny, nz, pml, rng.randint(16, 40), nrec, snap=rng.choice(["c16", "fp32"]),
                     interval=rng.choice([4, 8]))
    return dict(_shot("rtm", "fd8", "tti", nx, ny, nz, pml, rng.randint(16, 32), nrec,
                      snap=rng.choice(["fp16s", "c16", "fp32"]), interval=rng.choice([4, 8])), q=True,
                q_bf16=rng.random() < 0.6)


# --- inputs ---------------------------------------------------------------------
def _smooth(gen, shape, cell):
    """Smooth noise in [-1, 1]: a coarse normal field (one node per `cell` cells), interpolated."""
    ny, nx, nz = shape
    c = [max(2, -(-n // cell) + 1) for n in (ny, nx, nz)]
    g = torch.randn(1, 1, *c, generator=gen, device=DEV)
    v = torch.nn.functional.interpolate(g, size=(ny, nx, nz), mode="trilinear", align_corners=True)[0, 0]
    return v / v.abs().max()


def _ramp(v, lo, hi):
    a, b = v.min(), v.max()
    return lo + (v - a) * ((hi - lo) / (b - a))


def _spec(c):
    engine, model = ENGINE[c["engine"]], MODEL[c["model"]]
    p, py = c["pml"], c["pml"] if c["ny"] > 1 else 0
    spec = S.PropSpec(nx=c["nx"], ny=c["ny"], nz=c["nz"], engine=engine, model_type=model, use_q=c["q"],
                      q_bf16=c["q_bf16"], nbnd=(p, p, py, py, p, p), vmax=VMAX)
    # the stability rule at the model's fastest, most anisotropic cell, with a margin for the tilt and for Q
    one = [np.array([v]) for v in (VMAX, EPS_MAX, 0.0)]
    dt = W.cfl_dt(spec, *one) if model == S.ISO else \
        W.cfl_dt(S.PropSpec(nx=9, ny=c["ny"], nz=9, engine=engine, model_type=S.VTI), *one)
    spec.dt = float(np.float32(min(0.001, dt * (0.7 if model == S.TTI else 0.95))))
    return spec


def _axis_kernels(n, pos, k):
    """Spread kernels of positions along one axis: first index, length, taps padded to 20."""
    off, ln, taps = np.zeros(len(pos), np.int32), np.zeros(len(pos), np.int32), np.zeros((len(pos), 20), np.float32)
    for i, x in enumerate(pos):
        o, t = spread_coeffs(n, x, k[0], k[1], 20, False, 10)
        off[i], ln[i], taps[i, :len(t)] = o, len(t), t
    return off, ln, taps


def _traceset(spec, xs, ys, z):
    """Traces at every (x, y) of two position lists, depth z (fractional grid indices)."""
    k = W.spread_band(spec)
    ox, lx, tx = _axis_kernels(spec.nx, xs, k)
    oz, lz, tz = _axis_kernels(spec.nz, [z], k)
    if spec.ny > 1:
        oy, ly, ty = _axis_kernels(spec.ny, ys, k)
    else:
        oy, ly, ty = np.zeros(1, np.int32), np.ones(1, np.int32), np.ones((1, 1), np.float32)
    iy, ix = [a.ravel() for a in np.meshgrid(np.arange(len(oy)), np.arange(len(ox)), indexing="ij")]
    n = len(ix)
    off = np.stack([ox[ix], oy[iy], np.full(n, oz[0], np.int32)], 1)
    ln = np.stack([lx[ix], ly[iy], np.full(n, lz[0], np.int32)], 1)
    return S.TraceSet(n, tx.shape[1], ty.shape[1], tz.shape[1], off, ln, tx[ix], ty[iy], np.repeat(tz, n, 0))


def _spread_out(n, count):
    return [float(v) for v in np.linspace(1.3, n - 2.7, min(count, n - 2))] if n > 1 else [0.0]


def _wavelets(gen, spec, count, nt):
    """Band-limited trace samples: Ricker wavelets of 10-25 Hz with peaks spread around the window."""
    t = torch.arange(nt, device=DEV) * spec.dt
    f = 10 + 15 * torch.rand(count, 1, generator=gen, device=DEV)
    t0 = nt * spec.dt * torch.rand(count, 1, generator=gen, device=DEV)
    a = (math.pi * f * (t - t0)) ** 2
    return ((1 - 2 * a) * torch.exp(-a) * 1e5).float().cpu().numpy()


def _inputs(c, seed):
    """Everything a shot program holds before its loop, on the host: spec, model, traces, first wavefield."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    spec = _spec(c)
    shape = spec.shape
    depth = torch.linspace(0, 1, spec.nz, device=DEV)
    layers = (depth * 6 + 0.8 * float(torch.rand(1, generator=gen, device=DEV))).floor().clamp(0, 6) / 6
    vel = (VMIN + (VMAX - VMIN) * layers) * (1 + 0.05 * _smooth(gen, shape, 16))
    m = {"vel": vel.clamp(VMIN, VMAX)}
    if spec.model_type != S.ISO:
        m["eps"] = _ramp(_smooth(gen, shape, 20), 0.0, EPS_MAX)
        m["dl"] = _ramp(_smooth(gen, shape, 20), 0.0, DEL_MAX)
    if spec.model_type == S.TTI:
        th = torch.deg2rad(_ramp(_smooth(gen, shape, 24), 0.0, 45.0))
        ph = torch.deg2rad(_ramp(_smooth(gen, shape, 24), 0.0, 360.0))
        m["pjx"], m["pjy"] = -torch.sin(th) * torch.cos(ph), -torch.sin(th) * torch.sin(ph)
    if spec.use_q:
        m["invq"] = 1.0 / _ramp(_smooth(gen, shape, 24), 30.0, 200.0)
    m = {k: v.float().cpu().numpy() for k, v in m.items()}
    p = c["pml"]
    jit = [float(v) for v in torch.rand(3, generator=gen, device=DEV).cpu()]
    src = _traceset(spec, [spec.nx / 2 + jit[0]], [spec.ny / 2 + jit[1]], p + 11 + jit[2])
    rcv = _traceset(spec, _spread_out(spec.nx, c["nrec"]), _spread_out(spec.ny, c["nrec"]), p + 2.0)
    d = dict(spec=spec, model=m, src=src, rcv=rcv, src_tr=_wavelets(gen, spec, src.ntr, c["steps"]),
             q=W.q_coefficients(spec.dt, 20.0) if spec.use_q else None)
    if c["kind"] == "rtm":
        d["rcv_tr"] = 1e-2 * _wavelets(gen, spec, rcv.ntr, c["steps"])
    else:  # a shot on its way: a wavefield of about 8-cell half wavelengths everywhere
        d["field"] = (100 * _smooth(gen, shape, 8)).float().cpu().numpy()
    return d


def _propagator(d):
    p = Propagator(d["spec"])
    if d["q"]:
        p.set_q_coeffs(*d["q"])
    p.set_model(**d["model"])
    return p


def _running_shot(d, steps):
    """A handle in mid-shot: sources, receivers and the wavefields of the last two steps set."""
    p = _propagator(d)
    p.set_injection(d["src"], d["src_tr"], d["spec"].dt_dxyz)
    p.set_extraction(d["rcv"], steps)
    p.reset()
    p.put(S.FIELD_W0, d["field"])
    p.put(S.FIELD_W1, d["field"])
    return p


def _batch_cases(c, seed):
    r = np.random.default_rng(int(seed) + 7 * c["lo"])
    out = []
    for _ in range(c["shots"]):
        nx, ny, nz = (int(v) for v in r.integers(c["lo"], c["hi"] + 1, 3))
        out.append(_shot("modelling", "fd8", "iso", nx, ny, nz, c["pml"], int(r.integers(c["steps"] // 2, c["steps"] + 1)),
                         c["nrec"]))
    return out


def _batch_layout(c):
    """Grids and step counts of a batch: of the case, not of the seed, so that every seed is the same work."""
    return _batch_cases(c, 0)


def _codec_params(seed):
    """The average code's weights, perturbed: a code that carries the field, with every weight in use."""
    p = AE.init_params_average()
    return (p + 0.01 * np.random.default_rng(int(seed)).standard_normal(p.size)).astype(np.float32)


def _codec_volume(c, seed):
    """A wavefield as a snapshot meets it: strong in one region, weak far away, zero where it has not arrived."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (c["ny"], c["nx"], c["nz"])
    v = _smooth(gen, shape, 6)
    r2 = sum(((torch.arange(n, device=DEV) / n - 0.5) ** 2).reshape([-1 if i == a else 1 for i in range(3)])
             for a, n in enumerate(shape))
    return (v * 1e3 * torch.exp(-12 * r2) * (r2 < 0.5)).float().contiguous()


def prepare(case, seed):
    if case["kind"] == "codec":
        v = _codec_volume(case, seed)
        nb = math.prod(-(-n // 8) for n in v.shape)
        return dict(kind="codec", ae=AE.AutoEncoder(_codec_params(seed)), v=v,
                    lat=torch.empty(nb, AE.LATENT, dtype=torch.bfloat16, device=DEV),
                    sc=torch.empty(nb, device=DEV), out=torch.empty_like(v))
    if case["kind"] == "batch":
        subs = _batch_layout(case)
        shots = [_running_shot(_inputs(c, seed + k), c["steps"]) for k, c in enumerate(subs)]
        return dict(kind="batch", shots=shots, batch=Batch(shots), nts=[c["steps"] for c in subs])
    d = _inputs(case, seed)
    if case["kind"] == "rtm":
        return dict(kind="rtm", p=_propagator(d), d=d, case=case)
    return dict(kind="modelling", p=_running_shot(d, case["steps"]), steps=case["steps"])


def run(state):
    if state["kind"] == "modelling":
        state["p"].modelling(state["steps"])
        return state["p"].traces()
    if state["kind"] == "rtm":
        c, d = state["case"], state["d"]
        image, _, _ = state["p"].rtm_shot(d["src"], d["src_tr"], d["rcv"], d["rcv_tr"], c["steps"], c["steps"],
                                          c["interval"], snap_fmt=SNAP[c["snap"]])
        return image
    if state["kind"] == "batch":
        state["batch"].modelling(state["nts"])
        return [p.traces() for p in state["shots"]]
    ae, v = state["ae"], state["v"]
    ny, nx, nz = v.shape
    ptr = [C.c_void_p(t.data_ptr()) for t in (v, state["lat"], state["sc"], state["out"])]
    rc = ae.L.rtm_ae_compress_volume(ae.a, ptr[0], nx, ny, nz, ptr[1], ptr[2], None) or \
        ae.L.rtm_ae_decompress_volume(ae.a, ptr[1], ptr[2], nx, ny, nz, ptr[3], None)
    if rc:
        raise RuntimeError("codec call failed: %d" % rc)
    return {"latent": state["lat"], "scales": state["sc"], "volume": state["out"]}


# --- what a pass cannot do without ------------------------------------------------
def work(case):
    if case["kind"] == "codec":
        n, nb = case["nx"] * case["ny"] * case["nz"], math.prod(-(-case[k] // 8) for k in ("nx", "ny", "nz"))
        macs = sum(k * n_ * r for k, n_, r, _ in AE.LAYERS)
        return {"bytes": 8 * n + 2 * nb * (2 * AE.LATENT + 4), "flops": 2 * macs * nb}
    if case["kind"] == "batch":
        w = [work(c) for c in _batch_layout(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    dims = [case[k] for k in ("nx", "ny", "nz") if case[k] > 1]
    n, m = math.prod(dims), sum(2 * case["pml"] / d for d in dims)
    iso = case["engine"] == "fd8" and case["model"] == "iso"
    # each step: both wavefields read, one written, the velocity (and eps / delta, tilts, 1/Q and the memory
    # variables of both time levels) read, every PML memory value read and written
    per = 16 + 16 * m if iso else 24 + 48 * m
    per += 8 if case["model"] == "tti" else 0
    per += 4 + 12 * (2 if case["q_bf16"] else 4) if case["q"] else 0
    flops = 60 if iso else 150
    steps = case["steps"] * (2 if case["kind"] == "rtm" else 1)
    total = n * per * steps
    recs = math.prod(min(case["nrec"], case[k] - 2) for k in ("nx", "ny") if case[k] > 1)
    if case["kind"] == "rtm":
        snaps = (case["steps"] - 1) // case["interval"] + 1
        total += snaps * n * (2 * (4 if case["snap"] == "fp32" else 2) + 16) + 4 * n + 4 * recs * case["steps"]
    else:
        total += 4 * recs * case["steps"]
    return {"bytes": total, "flops": n * flops * steps}


# --- the same in 64 bits ------------------------------------------------------------
def _cfd_matrix(n, d, second):
    """Compact first derivative B^-1 A of n points (dense), with the mirrored boundary rows of the
    gradient pass (even field, odd derivative) or the divergence pass (`second`)."""
    ca = [0.861085998189822, 0.753782983214427, 0.257072513289755, 0.031326722562826, 0.000410456919800]
    cb = [1.0, 0.753205475977546, 0.312203852849021, 0.063580085296350, 0.004597763362256]
    A, B = np.zeros((n, n)), np.zeros((n, n))
    sb, sa = (1.0, -1.0) if second else (-1.0, 1.0)

    def put(M, i, j, v, sign):
        if j < 0:
            M[i, -j] += sign * v
        elif j > n - 1:
            M[i, 2 * (n - 1) - j] += sign * v
        else:
            M[i, j] += v

    for i in range(n):
        for k in range(-4, 5):
            put(B, i, i + k, cb[abs(k)], sb)
        for k in range(1, 6):
            put(A, i, i + k, ca[k - 1] / d / 2, sa)
            put(A, i, i - k, -ca[k - 1] / d / 2, sa)
    return np.linalg.solve(B, A)


def _r2r_matrix(n, d, second):
    """Cosine-transform derivative (sine back) of the gradient pass, or sine-transform derivative."""
    dk = np.float32(math.pi / float(np.float32(d) * np.float32(n)) * 0.5 * float(np.float32(1) / np.float32(n)))
    k = (-(np.arange(n) + 1).astype(np.float32) * dk).astype(np.float64)
    j, h = np.arange(n), np.arange(n) + 0.5
    if not second:
        X = 2 * np.cos(np.pi * np.outer(j, h) / n)
        Y = np.zeros((n, n))
        Y[:-1] = -k[:-1, None] * X[1:]
        T = 2 * np.sin(np.pi * np.outer(h, j + 1) / n)
        T[:, -1] = (-1.0) ** j
        return T @ Y
    X = 2 * np.sin(np.pi * np.outer(j + 1, h) / n)
    Y = np.zeros((n, n))
    Y[1:] = k[:-1, None] * X[:-1]
    T = 2 * np.cos(np.pi * np.outer(h, j) / n)
    T[:, 0] = 1.0
    return T @ Y


def _r2c_matrix(n, d, second):
    """Fourier derivative: bins below Nyquist times i k (the top bin of an odd line times the pass's sign)."""
    dk = np.float32(2 * float(np.float32(math.pi)) / float(np.float32(d) * np.float32(n)) * float(np.float32(1) / np.float32(n)))
    c = np.zeros(n)
    m = np.arange(n)
    for j in range(1, n // 2 if n % 2 == 0 else (n - 1) // 2 + 1):
        c -= 2 * float(np.float32(-j) * dk) * (-1.0 if second and j == n // 2 else 1.0) * np.sin(2 * np.pi * ((j * m) % n) / n)
    return c[(m[:, None] - m[None, :]) % n]


class _Exact:
    """One shot in 64 bits; volumes [ny][nx][nz], axes 1, 0, 2 = x, y, z."""
    AX = {"x": 1, "y": 0, "z": 2}

    def __init__(self, d):
        self.d, s = d, d["spec"]
        self.s = s
        self.f = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV).double()
        self.axes = [a for a in "xyz" if s.shape[self.AX[a]] > 1]
        self.three = s.ny > 1
        m = {k: self.f(v).reshape(s.shape) for k, v in d["model"].items()}
        dt = float(np.float32(s.dt))
        self.vel = m["vel"] ** 2 * dt ** 2
        if s.use_q:
            self.cq0, self.cq, self.wq = d["q"][0], [float(v) for v in d["q"][1]], [float(v) for v in d["q"][2]]
            corr = 1 / (1 - self.cq0 * m["invq"])
            q2 = m["invq"] ** 2
            self.vel = self.vel * (1 - 0.25 * q2 + q2 * q2 / 48) * corr
            self.invq = m["invq"] * corr
        self.m = m
        self.iso = s.engine == S.ENGINE_FD8 and s.model_type == S.ISO
        self.pml3d = bool(s.pml3d) and s.engine in (S.ENGINE_FD8, S.ENGINE_CFD)
        self.h = {"x": s.dx, "y": s.dy, "z": s.dz}
        if s.engine != S.ENGINE_FD8:
            make = {S.ENGINE_CFD: _cfd_matrix, S.ENGINE_R2R: _r2r_matrix, S.ENGINE_R2C: _r2c_matrix}[s.engine]
            self.D = {a: [self.f(make(s.shape[self.AX[a]], self.h[a], r)) for r in (False, True)] for a in self.axes}
        self.g = {}
        for i, a in enumerate("xyz"):
            for side in (0, 1):
                w = s.nbnd[2 * i + side]
                if w > 1 and a in self.axes:
                    beta = self.h[a] / (dt * s.vmax)
                    p = 0.75 * (np.arange(w, 0, -1) / w) ** 2 * math.log(1 / float(np.float32(s.pml_eps))) / (w * beta)
                    self.g[a, side] = self.f(p if side == 0 else p[::-1])
        self.reset()

    def reset(self):
        z = torch.zeros(self.s.shape, dtype=torch.float64, device=DEV)
        self.w0, self.w1 = z, z.clone()
        self.mem = {}
        if self.s.use_q:
            self.q = [[z.clone() for _ in self.cq] for _ in range(2)]

    def damp(self, v, axis, scale, key):
        """One round of the PML recursion along `axis`, its memory under `key`."""
        ax = self.AX[axis]
        n = v.shape[ax]
        for side in (0, 1):
            g = self.g.get((axis, side))
            if g is None:
                continue
            w = g.numel()
            g = (g * scale).reshape([-1 if i == ax else 1 for i in range(3)])
            p = v.narrow(ax, 0 if side == 0 else n - w, w)
            q = self.mem.get((axis, side) + key, 0.0)
            q = (1 - g) / (1 + g) * q - 2 * g / (1 - g * g) * p
            self.mem[(axis, side) + key] = q
            p.copy_(q + p / (1 - g))

    def tap(self, v, axis, k):
        """v shifted by k cells along axis: value at i + k, zero outside."""
        ax, n = self.AX[axis], v.shape[self.AX[axis]]
        out = torch.zeros_like(v)
        if abs(k) < n:
            out.narrow(ax, max(0, -k), n - abs(k)).copy_(v.narrow(ax, max(0, k), n - abs(k)))
        return out

    def deriv(self, v, axis, rnd):
        if self.s.engine == S.ENGINE_FD8:
            out = torch.zeros_like(v)
            for k, c in enumerate((4 / 5, -1 / 5, 4 / 105, -1 / 280), 1):
                out += c / self.h[axis] * (self.tap(v, axis, k) - self.tap(v, axis, -k))
        else:
            M = self.D[axis][rnd]
            if axis == "z":
                out = v @ M.T
            elif axis == "x":
                out = torch.matmul(M, v)
            else:
                out = (M @ v.reshape(v.shape[0], -1)).reshape(v.shape)
        self.damp(out, axis, 1.0, (rnd, 0))
        if self.pml3d:
            sc = float(np.float32(self.s.pml3d_scaler))
            for other in {"z": "xy", "x": "zy", "y": "zx"}[axis]:
                if other in self.axes:
                    self.damp(out, other, sc, (rnd, axis))
        return out

    def laplacian(self, v):
        out = torch.zeros_like(v)
        for axis in ("z", "x") + (("y",) if self.three else ()):
            h2 = self.h[axis] ** 2
            out += -205 / 72 / h2 * v
            for k, c in enumerate((8 / 5, -1 / 5, 8 / 315, -1 / 560), 1):
                out += c / h2 * (self.tap(v, axis, k) + self.tap(v, axis, -k))
        for axis in ("z", "x") + (("y",) if self.three else ()):
            for rnd in (0, 1):
                self.damp(out, axis, 1.0, (rnd, 0))
        return out

    def operator(self):
        if self.iso:
            return self.vel * self.laplacian(self.w1)
        g = {a: self.deriv(self.w1, a, 0) for a in self.axes}
        vx, vy, vz = g["x"], g.get("y", 0.0), g["z"]
        if self.s.model_type != S.ISO:
            e = 1 + 2 * self.m["eps"]
            dl = self.m["eps"] - self.m["dl"]
            if self.s.model_type == S.TTI:
                ax, ay = self.m["pjx"], self.m["pjy"] if self.three else 0.0
                az = torch.sqrt(1 - (ax * ax + ay * ay))
                along = vx * ax + vy * ay + vz * az
                vz2 = along ** 2
                vh2 = vx * vx + vy * vy + vz * vz - vz2
            else:
                vh2, vz2 = vx * vx + vy * vy, vz * vz
            ecl = e * vh2 + vz2
            sc = torch.clamp(0.5 * (1 + torch.sqrt(1 - 8 * dl * vh2 * vz2 / (ecl * ecl + 1e-32))), max=1.0)
            if self.s.model_type == S.TTI:
                for a, u in (("x", ax), ("y", ay), ("z", az)):
                    if a in g:
                        g[a] = (along * u + (g[a] - along * u) * e) * sc
            else:
                for a in "xy":
                    if a in g:
                        g[a] = g[a] * (e * sc)
        return self.vel * sum(self.deriv(g[a], a, 1) for a in self.axes)

    def step(self):
        out = self.w0 - self.operator()
        if not self.s.use_q:
            self.w0 = 2 * self.w1 - out
            return
        v = self.w1 * (2 + self.invq * sum(self.cq)) - out
        for l, (c, w) in enumerate(zip(self.cq, self.wq)):
            d0, d1 = self.q[0][l], self.q[1][l]
            v += self.invq * ((1 + w) * d0 - 2 * d1)
            self.q[0][l] = c * self.w1 + w * d0
        self.w0 = v

    def swap(self):
        self.w0, self.w1 = self.w1, self.w0
        if self.s.use_q:
            self.q.reverse()

    def dense(self, ts):
        """Trace set as dense x / y kernel matrices and its one z kernel."""
        key = id(ts)
        if getattr(self, "_dense", (None,))[0] != key:
            r = np.arange(ts.ntr)[:, None]
            mats = []
            for k, n, a in ((ts.kx, self.s.nx, 0), (ts.ky, self.s.ny, 1)):
                M = np.zeros((ts.ntr, n + k.shape[1]))
                j = np.arange(k.shape[1])[None, :]
                M[r, ts.off[:, a:a + 1] + j] = np.where(j < ts.len[:, a:a + 1], k, 0)
                mats.append(self.f(M[:, :n]))
            z0, lz = int(ts.off[0, 2]), int(ts.len[0, 2])
            self._dense = (key, mats[0], mats[1], slice(z0, z0 + lz), self.f(ts.kz[0, :lz]))
        return self._dense[1:]

    def inject(self, ts, traces, it):
        if 0 <= it < traces.shape[1]:
            kx, ky, z, kz = self.dense(ts)
            val = self.f(traces[:, it]) * float(self.s.dt_dxyz)
            self.w0[:, :, z] += ((ky * val[:, None]).T @ kx)[:, :, None] * kz * self.vel[:, :, z]

    def extract(self, ts):
        kx, ky, z, kz = self.dense(ts)
        return ((ky @ (self.w0[:, :, z] @ kz)) * kx).sum(1)

    def modelling(self, steps):
        self.w0, self.w1 = (self.f(self.d["field"]).reshape(self.s.shape) for _ in range(2))
        src, rcv, out = self.d["src"], self.d["rcv"], []
        both = {}
        for it in range(steps):
            self.step()
            self._dense = both.get("s", (None,))
            self.inject(src, self.d["src_tr"], it - 1)
            both["s"] = self._dense
            self._dense = both.get("r", (None,))
            out.append(self.extract(rcv))
            both["r"] = self._dense
            self.swap()
        return torch.stack(out, 1)

    def edge(self, v):
        v = v.clone()
        for ax, n, nt in ((0, self.s.ny, 20), (1, self.s.nx, 20), (2, self.s.nz, 10)):
            if n > 2 * nt:
                w = torch.ones(n, dtype=torch.float64, device=DEV)
                w[:nt] = 0.5 * (1 - torch.cos(math.pi * torch.arange(nt, device=DEV).double() / nt))
                w[-nt:] = w[:nt].flip(0)
                v *= w.reshape([-1 if i == ax else 1 for i in range(3)])
        return v

    def rtm(self, steps, interval):
        d, snaps = self.d, {}
        for it in range(steps):
            self.step()
            self.inject(d["src"], d["src_tr"], it - 1)
            if it % interval == 0:
                snaps[it // interval] = self.w0.clone()
            self.swap()
        self.reset()
        image = torch.zeros(self.s.shape, dtype=torch.float64, device=DEV)
        for it in range(steps - 1, -1, -1):
            self.step()
            self.inject(d["rcv"], d["rcv_tr"], it + 1)
            if it % interval == 0 and it // interval in snaps:
                image += self.edge(snaps[it // interval]) * self.edge(self.w0)
            self.swap()
        return image.reshape(-1)


def _exact_codec(case, seed):
    v = _codec_volume(case, seed).double()
    pad = [(-n) % 8 for n in v.shape]
    v = torch.nn.functional.pad(v, (0, pad[2], 0, pad[1], 0, pad[0]))
    by, bx, bz = (n // 8 for n in v.shape)
    # blocks of 8^3 cells, each cell at its Morton index (bits z y x from the least significant)
    b = v.reshape(by, 2, 2, 2, bx, 2, 2, 2, bz, 2, 2, 2).permute(0, 4, 8, 5, 1, 9, 6, 2, 10, 7, 3, 11)
    b = b.reshape(-1, 512)
    sc = b.abs().amax(1)
    x = b / torch.where(sc > 0, sc, torch.ones_like(sc))[:, None]
    params, o, lat = torch.as_tensor(_codec_params(seed), device=DEV).double(), 0, None
    for l, (k, n, rows, act) in enumerate(AE.LAYERS):
        wt, bias = params[o:o + k * n].reshape(k, n), params[o + k * n:o + k * n + n]
        o += k * n + n
        x = x.reshape(-1, k) @ wt + bias
        x = torch.where(x > 0, x, 0.1 * x) if act else x
        if l == 3:
            lat = x.reshape(-1, AE.LATENT)
    out = (x.reshape(-1, 512) * sc[:, None]).reshape(by, bx, bz, 2, 2, 2, 2, 2, 2, 2, 2, 2)
    out = out.permute(0, 4, 7, 10, 1, 3, 6, 9, 2, 5, 8, 11).reshape(by * 8, bx * 8, bz * 8)
    return {"latent": lat, "scales": sc, "volume": out[:case["ny"], :case["nx"], :case["nz"]].contiguous()}


def exact(case, seed):
    if case["kind"] == "codec":
        return _exact_codec(case, seed)
    if case["kind"] == "batch":
        return [_Exact(_inputs(c, seed + k)).modelling(c["steps"]) for k, c in enumerate(_batch_layout(case))]
    e = _Exact(_inputs(case, seed))
    if case["kind"] == "rtm":
        return e.rtm(case["steps"], case["interval"])
    return e.modelling(case["steps"])
