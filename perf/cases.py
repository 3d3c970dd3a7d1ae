"""The work that users of this library have it do, as cases that can be timed and compared.

Every case runs through the public entry points on device data: the frame call (``capon_frames`` on
``DeviceFrame``), the differentiable power (``capon_power``), the stage objects ``BuildR`` and ``Solver``, and the C
ABI calls for time-domain steering and for LCA window selection.  The sizes come from the library's synthetic
configurations, its tests and its benchmark:

* frames: M = 32..128 channels with subarrays of M/2 or M/3, odd and ragged sizes among them, windows of 1 to 9 range
  rows, relative loading 1e-3 to 5e-2, z and P alone or with the weights w;
* data: circular Gaussian noise with point scatterers (a phase ramp across channels, a Gaussian envelope in range),
  the generator of ``cos_gb300.synth``, formed on the device.

``exact`` restates each result in complex128 with plain torch.
"""
import ctypes
import math

import torch

from cos_gb300 import _lib, autograd, capon

DEV = "cuda"


# ---- the cases ----------------------------------------------------------------------------------------------------
def listed():
    return [
        # one beam line of a live display: a call of a few dozen pixels, where launch latency is all
        frame("live_line", Nx=1, Ny=64, M=32, L=16, K=1),
        # a sector scan whose channel count is no multiple of anything (dead elements taken out), with weights
        frame("ragged_l16_w", Nx=61, Ny=507, M=37, L=16, K=1, w=True),
        # the throughput frame: 256 beams x 2048 range rows, half-aperture subarrays; amplitude and power
        frame("frame_l32", Nx=256, Ny=2048, M=64, L=32, K=2, scatterers=8, amplitude=10.0),
        # a subarray length of the user's own choice (half of 48 channels), odd frame, with weights
        frame("subarray_24_w", Nx=119, Ny=509, M=48, L=24, K=2, w=True),
        # forward-backward averaging, the usual choice against coherent echoes
        frame("forward_backward_l32", Nx=64, Ny=1024, M=64, L=32, K=2, fb=True),
        # two coherent scatterers at 40 dB under light loading: long subarrays, adaptive refinement
        frame("coherent_l64", Nx=64, Ny=1024, M=128, L=64, K=4, d=1e-3, refine=2, scatterers=2, amplitude=100.0,
              coherent=True),
        # several frames of different M, L and Nb in one call
        dict(name="uneven_frames", kind="frames", shapes="32,16,0;64,32,0;96,48,3;128,64,5", Nx=256, Ny=1024, K=1,
             d=0.01),
        # beamspace with more beams than the narrow main-lobe fan, with weights
        frame("beamspace_8_w", Nx=128, Ny=512, M=64, L=32, K=1, Nb=8, w=True),
        # one training step through the power: gradients of samples, loading and delays
        dict(name="gradient_step", kind="gradient", Nx=128, Ny=1024, M=64, L=32, K=2, d=0.05),
        # the reference's stage interfaces on device memory: covariances, then a batched general solve
        dict(name="stages_l32", kind="stages", Nx=32, Ny=512, M=64, L=32, K=2, d=0.01),
        # steering of matched-filtered channel data to the frame's pixels: cube and delay-and-sum image
        dict(name="steering", kind="steering", Nx=256, Ny=2048, M=64, samples=4096),
        # window selection over a frame's pixels, 8 windows, a filter along range
        dict(name="window_selection", kind="select", Nx=256, Ny=2048, Nw=8, Yf=5, Xf=1),
    ]


def frame(name, **v):
    c = dict(name=name, kind="frame", Nb=0, d=0.01, w=False, fb=False, refine=0, scatterers=3, amplitude=5.0,
             coherent=False)
    c.update(v)
    return c


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["live", "frame", "frame", "frame", "frame", "own", "own", "frames", "beamspace", "gradient",
                       "stages", "steering", "select"])
    if kind == "live":
        L = rng.choice([8, 16, 24, 32])
        K = rng.randint(0, 2)
        c = frame("", Nx=rng.randint(1, 4), Ny=rng.randint(2 * K + 1, 160), M=rng.randint(L, 2 * L + 8), L=L, K=K,
                  w=rng.random() < 0.3)
    elif kind == "frame":
        # the common subarray lengths, every option
        L = rng.choice([16, 32, 32, 48, 64])
        c = frame("", Nx=_log(rng, 2, 256), Ny=_log(rng, 40, 2048), M=rng.randint(L + L // 2, min(128, 2 * L + 8)), L=L,
                  K=rng.randint(0, 2 if L < 48 else 4), w=rng.random() < 0.4, fb=rng.random() < 0.2,
                  refine=rng.choice([0, 0, 0, 1, 2]), d=rng.choice([0.05, 0.01, 0.01]),
                  scatterers=rng.randint(1, 8), amplitude=rng.choice([3.0, 10.0]))
    elif kind == "own":
        # any subarray length
        L = rng.randint(4, 64)
        c = frame("", Nx=_log(rng, 2, 256), Ny=_log(rng, 40, 1024), M=rng.randint(L + L // 2, min(128, 2 * L + 8)), L=L,
                  K=rng.randint(0, 3), w=rng.random() < 0.5, fb=rng.random() < 0.3)
    elif kind == "frames":
        some = ["32,16,0", "33,16,0", "64,32,0", "60,30,0", "96,48,3", "128,64,5", "64,32,2", "48,24,0"]
        c = dict(kind="frames", shapes=";".join(rng.sample(some, rng.randint(2, 4))), Nx=_log(rng, 4, 128),
                 Ny=_log(rng, 64, 1024), K=rng.randint(0, 2), d=0.01)
    elif kind == "beamspace":
        L = rng.choice([16, 24, 32])
        c = frame("", Nx=_log(rng, 2, 256), Ny=_log(rng, 40, 512), M=rng.randint(L + L // 2, 2 * L), L=L,
                  K=rng.randint(0, 2), Nb=rng.randint(2, 12), w=rng.random() < 0.5)
    elif kind == "gradient":
        L = rng.choice([8, 16, 24, 32])
        c = dict(kind="gradient", Nx=_log(rng, 4, 128), Ny=_log(rng, 40, 1024), M=2 * L + rng.randint(-3, 3), L=L,
                 K=rng.randint(0, 2), d=rng.choice([0.02, 0.05]))
    elif kind == "stages":
        L = rng.randint(4, 48)
        c = dict(kind="stages", Nx=_log(rng, 1, 32), Ny=_log(rng, 20, 512), M=2 * L + rng.randint(-3, 3), L=L,
                 K=rng.randint(0, 2), d=0.01)
    elif kind == "steering":
        c = dict(kind="steering", Nx=_log(rng, 8, 256), Ny=_log(rng, 40, 2048), M=rng.randint(16, 128),
                 samples=rng.choice([2048, 4096]))
        c["Ny"] = min(c["Ny"], max(40, (256 * 2048 * 64) // (c["Nx"] * c["M"])))
    else:
        Yf, Xf = rng.choice([(5, 1), (3, 3), (1, 1), (7, 5)])
        c = dict(kind="select", Nx=_log(rng, 16, 256), Ny=_log(rng, 40, 2048), Nw=rng.randint(2, 9), Yf=Yf, Xf=Xf)
        c["Ny"] = min(c["Ny"], max(40, (256 * 2048 * 8) // (c["Nx"] * c["Nw"])))
    c.pop("name", None)
    # no drawn case costs more than the listed throughput frame
    most = work(listed()[2])["flops"] / 2
    while c["Nx"] > 1 and work(c)["flops"] > most:
        c["Nx"] = max(1, c["Nx"] // 2)
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------
def _cube(Nx, Ny, M, seed, scatterers=3, amplitude=5.0, coherent=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn((Nx, Ny, M), dtype=torch.complex64, device=DEV, generator=g)
    u = torch.rand((max(1, scatterers), 2), generator=g, device=DEV)
    if coherent:   # one range, one beam apart, the same phase
        u[:, 0] = u[0, 0]
        u[:, 1] = u[0, 1] + torch.arange(u.shape[0], device=DEV) / max(Nx, 2)
    lo, hi = min(12.0, Ny / 4), max(Ny - 12.0, 3 * Ny / 4)
    y0 = lo + u[:, 0] * (hi - lo)
    b0 = torch.floor(u[:, 1] * Nx)
    env = amplitude * torch.exp(-(torch.arange(Ny, device=DEV)[None, :] - y0[:, None]) ** 2 / 32.0)
    b = torch.arange(Nx, device=DEV)[None, :] - b0[:, None]
    ramp = math.pi * 2.0 / M * b[:, :, None] * torch.arange(M, device=DEV)
    for k in range(u.shape[0]):
        ph = torch.polar(torch.ones_like(ramp[k]), ramp[k])
        x += (env[k][None, :, None] * ph[:, None, :]).to(torch.complex64)
    return x


def _shapes(c):
    return [tuple(int(v) for v in s.split(",")) for s in c["shapes"].split(";")]


def _device_frame(x, L, K, d, Nb, w):
    Nx, Ny, _ = x.shape
    n = Ny - 2 * K
    f = capon.DeviceFrame(x=x, L=L, K=K, d=d, Nb=Nb, z=torch.empty((Nx, n), dtype=torch.complex64, device=DEV),
                          P=torch.empty((Nx, n), dtype=torch.float32, device=DEV))
    if w:
        f.w = torch.empty((Nx, n, L), dtype=torch.complex64, device=DEV)
    return f


def _geometry(c, seed):
    """A towed line of receivers over a fan of pixels, and noise as the channel data."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    M, S = c["M"], c["samples"]
    fs, cs, fc, t0 = 5.0e4, 1480.0, 1.0e5, 30.0 / 1480.0
    mf = torch.randn((M, S), dtype=torch.complex64, device=DEV, generator=g)
    x_r = torch.linspace(-0.02 * M, 0.02 * M, M, dtype=torch.float64, device=DEV)
    depth = 0.02 * torch.randn(M, dtype=torch.float64, device=DEV, generator=g)
    # slant ranges whose two-way delays stay inside the recorded time
    rng0, rng1 = 0.52 * cs * t0 + 3.0, 0.48 * cs * (t0 + S / fs)
    r = torch.linspace(rng0, rng1, c["Ny"], dtype=torch.float64, device=DEV)[None, :]
    th = torch.linspace(-0.6, 0.6, c["Nx"], dtype=torch.float64, device=DEV)[:, None]
    jitter = 1.0 + 1e-3 * torch.rand((1, 1), dtype=torch.float64, device=DEV, generator=g)
    return dict(mf=mf, x_r=x_r, D=depth, X=(jitter * r * torch.sin(th)).contiguous(),
                Y=(jitter * r * torch.cos(th)).contiguous(), t0=t0, dt=1.0 / fs, cs=cs, fc=fc)


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "frame":
        x = _cube(c["Nx"], c["Ny"], c["M"], seed, c["scatterers"], c["amplitude"], c["coherent"])
        return dict(kind=k, frames=[_device_frame(x, c["L"], c["K"], c["d"], c["Nb"], c["w"])],
                    opts=capon.opts(fb=int(c["fb"]), refine=c["refine"]))
    if k == "frames":
        fs = [_device_frame(_cube(c["Nx"], c["Ny"], M, seed * 10 + i), L, c["K"], c["d"], Nb, False)
              for i, (M, L, Nb) in enumerate(_shapes(c))]
        return dict(kind=k, frames=fs, opts=capon.opts())
    if k == "gradient":
        x = _cube(c["Nx"], c["Ny"], c["M"], seed).requires_grad_(True)
        tau, gP = _gradient_inputs(c, seed)
        delta = torch.tensor(c["d"], dtype=torch.float32, device=DEV, requires_grad=True)
        return dict(kind=k, x=x, tau=tau.requires_grad_(True), delta=delta, gP=gP, L=c["L"], K=c["K"])
    if k == "stages":
        n = c["Ny"] - 2 * c["K"]
        L, batch = c["L"], c["Nx"] * n
        return dict(kind=k, case=c, x=_cube(c["Nx"], c["Ny"], c["M"], seed), build=capon.BuildR(), solver=capon.Solver(),
                    R=torch.empty((c["Nx"], n, L, L), dtype=torch.complex64, device=DEV), b=_right_sides(c, seed),
                    v=torch.empty((c["Nx"], n, L), dtype=torch.complex64, device=DEV), batch=batch)
    if k == "steering":
        return dict(kind=k, case=c, g=_geometry(c, seed), ctx=capon.Context(),
                    Xd=torch.empty((c["Nx"], c["Ny"], c["M"]), dtype=torch.complex64, device=DEV),
                    image=torch.empty((c["Ny"], c["Nx"]), dtype=torch.complex64, device=DEV))
    Z, wrf = _windows(c, seed)
    return dict(kind=k, case=c, Z=Z, wrf=wrf, wrf_c=(ctypes.c_double * len(wrf))(*wrf), ctx=capon.Context(),
                img=torch.empty((c["Ny"], c["Nx"]), dtype=torch.complex64, device=DEV),
                win=torch.empty((c["Ny"], c["Nx"]), dtype=torch.int32, device=DEV))


def _gradient_inputs(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 77)
    tau = torch.rand(c["M"], device=DEV, generator=g) * 0.1 - 0.05
    gP = torch.randn((c["Nx"], c["Ny"] - 2 * c["K"]), device=DEV, generator=g)
    return tau, gP


def _right_sides(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 99)
    return torch.randn((c["Nx"], c["Ny"] - 2 * c["K"], c["L"]), dtype=torch.complex64, device=DEV, generator=g)


def _windows(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    Z = torch.randn((c["Ny"], c["Nx"], c["Nw"]), dtype=torch.complex64, device=DEV, generator=g)
    return Z, [1.0] * (c["Yf"] * c["Xf"])


# ---- one pass -----------------------------------------------------------------------------------------------------
def run(state):
    s, k = state, state["kind"]
    if k in ("frame", "frames"):
        capon.capon_frames(s["frames"], o=s["opts"])
        return [[v for v in (f.z, f.P, f.w) if v is not None] for f in s["frames"]]
    if k == "gradient":
        P = autograd.capon_power(s["x"], s["delta"], s["tau"], s["L"], s["K"])
        gx, gd, gt = torch.autograd.grad(P, [s["x"], s["delta"], s["tau"]], s["gP"])
        return dict(P=P.detach(), gx=gx, gdelta=gd, gtau=gt)
    c = s["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if k == "stages":
        e = s["build"].getR(s["R"].data_ptr(), s["x"].data_ptr(), c["d"], c["L"], c["K"], c["M"], c["Nx"], c["Ny"], 0,
                            R_on_gpu=True, x_on_gpu=True)
        _lib.check(e, "getR")
        e = s["solver"].solve(s["v"].data_ptr(), s["R"].data_ptr(), s["b"].data_ptr(), c["L"], s["batch"],
                              x_on_gpu=True, A_on_gpu=True, b_on_gpu=True)
        _lib.check(e, "solve")
        return dict(R=s["R"], v=s["v"])
    if k == "steering":
        g = s["g"]
        e = _lib.lib.cos_capon_tdib(s["ctx"].handle, g["mf"].data_ptr(), c["M"], c["samples"], g["t0"], g["dt"],
                                    g["x_r"].data_ptr(), g["D"].data_ptr(), g["cs"], g["fc"], g["X"].data_ptr(),
                                    g["Y"].data_ptr(), c["Nx"], c["Ny"], s["Xd"].data_ptr(), s["image"].data_ptr(), 1,
                                    stream)
        _lib.check(e, "cos_capon_tdib")
        return dict(Xd=s["Xd"], image=s["image"])
    e = _lib.lib.cos_capon_lca(s["ctx"].handle, s["Z"].data_ptr(), c["Ny"], c["Nx"], c["Nw"], s["wrf_c"], c["Yf"],
                               c["Xf"], s["img"].data_ptr(), s["win"].data_ptr(), 1, stream)
    _lib.check(e, "cos_capon_lca")
    return dict(img=s["img"], win=s["win"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _frame_work(Nx, Ny, M, L, K, Nb, w):
    T, Ns = 2 * K + 1, M - L + 1
    rows, px = Nx * Ny, Nx * (Ny - 2 * K)
    n = Nb or L
    tri = n * (n + 1) / 2
    if Nb:   # sliding DFT of each row, then the products of its beams
        row = Ns * Nb * 8 + L * Nb * 8 + Ns * tri * 8
    else:    # the first covariance row, then two products per entry along the diagonals
        row = Ns * L * 8 + tri * 16
    # the window's sum carried along range, the factorisation, two right-hand sides, the output sums
    pixel = tri * 4 + 8 * n ** 3 / 6 + 2 * 8 * n * n / 2 + 8 * n + (8 * n * n / 2 + (8 * L * Nb) if w else 0)
    return dict(bytes=8.0 * Nx * Ny * M + px * (12 + (8 * L if w else 0)), flops=float(rows * row + px * pixel))


def work(case):
    c, k = case, case["kind"]
    if k == "frame":
        return _frame_work(c["Nx"], c["Ny"], c["M"], c["L"], c["K"], c["Nb"], c["w"])
    if k == "frames":
        each = [_frame_work(c["Nx"], c["Ny"], M, L, c["K"], Nb, False) for M, L, Nb in _shapes(c)]
        return {q: sum(e[q] for e in each) for q in ("bytes", "flops")}
    Nx, Ny = c["Nx"], c["Ny"]
    if k == "gradient":
        f = _frame_work(Nx, Ny, c["M"], c["L"], c["K"], 0, True)
        T, Ns, px = 2 * c["K"] + 1, c["M"] - c["L"] + 1, Nx * (Ny - 2 * c["K"])
        # samples in, P and the gradient out, gP in; w^H x and its adjoint for every snapshot
        return dict(bytes=16.0 * Nx * Ny * c["M"] + 8.0 * px, flops=f["flops"] + px * T * Ns * c["L"] * 16.0)
    if k == "stages":
        L, T, px = c["L"], 2 * c["K"] + 1, Nx * (Ny - 2 * c["K"])
        f = _frame_work(Nx, Ny, c["M"], L, c["K"], 0, False)
        return dict(bytes=8.0 * Nx * Ny * c["M"] + px * (16.0 * L * L + 16.0 * L),
                    flops=f["flops"] + px * 8.0 * L ** 3 / 3)
    if k == "steering":
        n = Nx * Ny
        return dict(bytes=8.0 * n * c["M"] + 24.0 * n + 8.0 * c["M"] * c["samples"], flops=40.0 * n * c["M"])
    n = Nx * Ny
    return dict(bytes=8.0 * n * c["Nw"] + 12.0 * n, flops=n * c["Nw"] * (3.0 + 2.0 * c["Yf"] * c["Xf"]))


# ---- the same in 64 bits ------------------------------------------------------------------------------------------
def _butler(Nb, L):
    b = torch.arange(Nb, dtype=torch.float64, device=DEV)
    bins = torch.where(b > Nb // 2, b + (L - 2 * (Nb // 2) - 1), b)
    ph = -2.0 * math.pi / L * bins[:, None] * torch.arange(L, dtype=torch.float64, device=DEV)
    return torch.polar(torch.full_like(ph, 1.0 / math.sqrt(L)), ph)


def _covariance(x, L, K, fb):
    """Normalised, unloaded [b, n, L, L] of x [b, Ny, M] in complex128, and the subarray means of the centre rows."""
    n, T, Ns = x.shape[1] - 2 * K, 2 * K + 1, x.shape[2] - L + 1
    sub = x.unfold(2, L, 1)
    rows = torch.matmul(sub.transpose(2, 3), sub.conj())
    R = sum(rows[:, t:t + n] for t in range(T)) / (Ns * T)
    if fb:
        R = 0.5 * (R + R.transpose(2, 3).flip(2, 3))
    return R, sub[:, K:K + n].mean(2)


def _chunks(Nx, Ny, L):
    step = max(1, int(4e7 / (Ny * L * L)))
    return [(b, min(Nx, b + step)) for b in range(0, Nx, step)]


def _load(R, d, absolute=False):
    L = R.shape[-1]
    tr = torch.diagonal(R, dim1=2, dim2=3).real.sum(-1)
    dl = torch.full_like(tr, d) if absolute else d * tr / L
    return dl[:, :, None, None] * torch.eye(L, dtype=R.dtype, device=R.device)


def _exact_frame(x, L, K, d, Nb=0, fb=False, absolute=False):
    d = float(torch.tensor(d, dtype=torch.float32))
    out = []
    for b0, b1 in _chunks(x.shape[0], x.shape[1], L):
        R, g = _covariance(x[b0:b1].to(torch.complex128), L, K, fb)
        dl = _load(R, d, absolute)
        a = torch.ones(L, dtype=R.dtype, device=R.device)
        if Nb:
            B = _butler(Nb, L)
            A = B @ (R + dl) @ B.conj().T
            v = torch.linalg.solve(A, (B @ a).expand(*R.shape[:2], Nb).unsqueeze(-1))[..., 0]
            ria = v @ B.conj()
        else:
            ria = torch.linalg.solve(R + dl, a.expand(*R.shape[:2], L).unsqueeze(-1))[..., 0]
        den = ria.sum(-1).real
        w = ria / den[..., None]
        out.append(((w.conj() * g).sum(-1), 1.0 / den, w))
    return [torch.cat(v) for v in zip(*out)]


def _exact_gradient(c, seed):
    x = _cube(c["Nx"], c["Ny"], c["M"], seed).to(torch.complex128)
    tau, gP = (v.double() for v in _gradient_inputs(c, seed))
    L, K, M = c["L"], c["K"], c["M"]
    T, Ns, n = 2 * K + 1, M - L + 1, c["Ny"] - 2 * K
    f = 2.0 * math.pi * 0.25
    phase = torch.polar(torch.ones_like(tau), -f * tau)
    xp = x * phase
    _, P, w = _exact_frame(xp, L, K, c["d"], absolute=True)
    gx = torch.zeros_like(xp)
    for b0, b1 in _chunks(c["Nx"], c["Ny"], L):
        wb = w[b0:b1]
        for t in range(T):
            e = torch.matmul(xp[b0:b1, t:t + n].unfold(2, L, 1), wb.conj().unsqueeze(-1))[..., 0]
            e = e * (gP[b0:b1] / (Ns * T))[..., None]
            for l in range(L):
                gx[b0:b1, t:t + n, l:l + Ns] += e * wb[..., l:l + 1]
    gtheta = 2.0 * (gx.real * xp.imag - gx.imag * xp.real).sum((0, 1))
    gd = (gP * (w.abs() ** 2).sum(-1)).sum()
    return dict(P=P, gx=2.0 * phase.conj() * gx, gdelta=gd, gtau=f * gtheta)


def _exact_steering(c, seed):
    g = _geometry(c, seed)
    xx, zz = 0.5 * g["x_r"].mean(), 0.5 * g["D"].mean()
    Xd, mf = [], g["mf"].to(torch.complex128)
    ax, Y2 = xx + g["X"], g["Y"] ** 2
    rt = torch.sqrt(ax ** 2 + Y2 + zz ** 2)
    for m in range(c["M"]):
        rr = torch.sqrt((ax - g["x_r"][m]) ** 2 + Y2 + (zz - g["D"][m]) ** 2)
        tau = (rt + rr) / g["cs"]
        u = (tau - g["t0"]) / g["dt"]
        i = torch.floor(u)
        ok = (i >= 0) & (u <= c["samples"] - 1)
        i0 = i.clamp(0, c["samples"] - 1).long()
        i1 = (i0 + 1).clamp(max=c["samples"] - 1)
        v = mf[m][i0] + (u - i) * (mf[m][i1] - mf[m][i0])
        cyc = g["fc"] * tau
        v = v * torch.polar(torch.ones_like(u), 2.0 * math.pi * (cyc - torch.floor(cyc)))
        Xd.append(torch.where(ok, v, torch.full_like(v, complex(math.nan, math.nan))))
    Xd = torch.stack(Xd, -1)
    return dict(Xd=Xd, image=Xd.mean(-1).T)


def _exact_select(c, seed):
    Z, wrf = _windows(c, seed)
    Yf, Xf, Ny, Nx = c["Yf"], c["Xf"], c["Ny"], c["Nx"]
    p = Z.to(torch.complex128).abs() ** 2
    s = torch.zeros((Ny - Yf + 1, Nx - Xf + 1, c["Nw"]), dtype=torch.float64, device=DEV)
    for yy in range(Yf):
        for xx in range(Xf):
            s += wrf[yy * Xf + xx] * p[yy:yy + Ny - Yf + 1, xx:xx + Nx - Xf + 1]
    best = s.argmin(-1)
    ym, xm = (Yf - 1) // 2, (Xf - 1) // 2
    img = torch.zeros((Ny, Nx), dtype=torch.complex128, device=DEV)
    inner = Z[ym:ym + best.shape[0], xm:xm + best.shape[1]].to(torch.complex128)
    img[ym:ym + best.shape[0], xm:xm + best.shape[1]] = torch.gather(inner, 2, best[..., None])[..., 0]
    return dict(img=img, win=None)   # near-ties may fall either way in 32 bits


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "frame":
        x = _cube(c["Nx"], c["Ny"], c["M"], seed, c["scatterers"], c["amplitude"], c["coherent"])
        z, P, w = _exact_frame(x, c["L"], c["K"], c["d"], c["Nb"], c["fb"])
        return [[z, P, w] if c["w"] else [z, P]]
    if k == "frames":
        return [_exact_frame(_cube(c["Nx"], c["Ny"], M, seed * 10 + i), L, c["K"], c["d"], Nb)[:2]
                for i, (M, L, Nb) in enumerate(_shapes(c))]
    if k == "gradient":
        return _exact_gradient(c, seed)
    if k == "stages":
        x, b = _cube(c["Nx"], c["Ny"], c["M"], seed), _right_sides(c, seed).to(torch.complex128)
        R, _ = _covariance(x.to(torch.complex128), c["L"], c["K"], False)
        R = (R + _load(R, float(torch.tensor(c["d"], dtype=torch.float32))))
        R = R * ((c["M"] - c["L"] + 1) * (2 * c["K"] + 1))
        # memory holds each matrix by columns
        return dict(R=R.transpose(2, 3).contiguous(), v=torch.linalg.solve(R, b.unsqueeze(-1))[..., 0])
    if k == "steering":
        return _exact_steering(c, seed)
    return _exact_select(c, seed)
