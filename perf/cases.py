"""What the performance work on this solver is measured on.

Every case is one call pattern of a user's program through the public entry
points, at sizes of the tests, the workload builders (``kwave/workloads.py``)
and the benchmark, or generic ones:

* ``gradient``  the allocation-free k-space gradient of a 2D field that the
  caller already holds on the device (``kspace_gradient_noalloc``);
* ``front``     ``kspaceFirstOrder2D`` / ``3D``, the whole call with its
  pre- and post-processing;
* ``solve``     ``kwave.solve`` on prepared input datasets: set-up, upload,
  every time step, read-back (what the MEX gateway and a server's request do);
* ``resident``  a ``Session`` kept on the device and advanced by some time
  steps per pass, then read (monitoring, serving, the benchmark);
* ``batch``     several sessions advanced together (``Batch``), then read.

The outputs of a pass are everything the call returns.  ``exact`` restates
the time loop in FP64 with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-wave_b200"))

DX = 1e-4
PML = {2: 20, 3: 10}
MAX_SOLVE_POINT_STEPS = 45e6 * 24  # grid points x steps of the largest listed case


def listed():
    return [
        # the smallest call: the gradient of a field an application already has on the device
        dict(name="gradient_2d", kind="gradient", nx=384, ny=320),
        # a first simulation: 2D homogeneous lossless, initial pressure, Cartesian circle of sensors, default call
        dict(name="p0_2d_whole_call", kind="front", nx=128, ny=128, nz=1, nt=533, source="p0", absorbing=0.0,
             nonlinear=False, het=False, record="p"),
        # a served 2D request: heterogeneous absorbing medium, plane tone-burst source, point sensors
        dict(name="absorbing_2d_request", kind="solve", nx=540, ny=540, nz=1, nt=800, source="plane",
             absorbing=1.4, nonlinear=False, het=True, record="p"),
        # a large lossless 2D field driven by a velocity source, kept resident (parameter studies on big 2D grids)
        dict(name="velocity_2d_resident", kind="resident", nx=1024, ny=768, nz=1, nt=200, source="u",
             absorbing=0.0, nonlinear=False, het=True, record="p_max,u_max,u_final"),
        # a small 3D therapy-style run: nonlinear, absorbing, where launches count
        dict(name="nonlinear_3d_small", kind="solve", nx=64, ny=72, nz=80, nt=600, source="plane", absorbing=1.5,
             nonlinear=True, het=True, record="p,p_max,p_rms"),
        # a photoacoustic forward run: 3D homogeneous lossless, initial pressure, p and u series on a sphere of points
        dict(name="p0_3d_series", kind="solve", nx=128, ny=128, nz=128, nt=400, source="p0", absorbing=0.0,
             nonlinear=False, het=False, record="p,u,p_max,p_rms"),
        # time-reversal reconstruction: every boundary point driven with its own signal, the final field returned
        dict(name="time_reversal_3d", kind="solve", nx=144, ny=120, nz=96, nt=400, source="dirichlet",
             absorbing=0.0, nonlinear=False, het=True, record="p_final"),
        # a grid picked without regard to the transform: edges with a factor 7
        dict(name="radix7_3d_resident", kind="resident", nx=112, ny=98, nz=126, nt=100, source="plane",
             absorbing=1.5, nonlinear=False, het=True, record="p_max,p_rms,u_final"),
        # Stokes absorption and an additive velocity source on an uneven 3D grid, u recorded
        dict(name="stokes_3d_resident", kind="resident", nx=180, ny=150, nz=125, nt=100, source="u",
             absorbing=2.0, nonlinear=True, het=True, record="p_rms,u_max,u_rms,u_final"),
        # independent small simulations on uneven grids advanced together
        dict(name="batch_3d_uneven", kind="batch", shapes="64x160x75,96x81x180,135x72x100,80x128x90,162x64x108,125x144x64",
             nt=120, absorbing=1.1, record="p_max,p_rms"),
        # the benchmark's configuration: 256^3 heterogeneous absorbing nonlinear, p_max and p_rms at every point
        dict(name="nonlinear_3d_256", kind="resident", nx=256, ny=256, nz=256, nt=200, source="plane",
             absorbing=1.5, nonlinear=True, het=True, record="p_max,p_rms", dense=True),
        # the largest: a clinical-size heterogeneous absorbing field with edges above 256
        dict(name="absorbing_3d_large", kind="resident", nx=432, ny=360, nz=288, nt=24, source="plane",
             absorbing=1.5, nonlinear=False, het=True, record="p_max,p_rms"),
    ]


def _lengths(lo, hi):
    """Edges in [lo, hi] whose largest prime factor is 7, odd ones among them."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def _edge(rng, lo, hi):
    """An admissible edge, spread over the logarithm of the range."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_lengths(lo, hi), key=lambda n: abs(n - v))


def draw(rng):
    kind = rng.choice(["gradient", "solve", "solve", "resident", "resident", "resident"])
    if kind == "gradient":
        return dict(kind=kind, nx=_edge(rng, 45, 1024), ny=_edge(rng, 45, 1024))
    three_d = rng.random() < 0.6
    absorbing = rng.choice([0.0, 0.0, 2.0, round(rng.uniform(1.05, 1.8), 3), round(rng.uniform(1.05, 1.8), 3)])
    case = dict(kind=kind, nx=_edge(rng, 48, 400 if three_d else 1080), ny=_edge(rng, 48, 400 if three_d else 1080),
                nz=_edge(rng, 45, 300) if three_d else 1)
    npts = case["nx"] * case["ny"] * case["nz"]
    nt = int(min(600, 0.12 * MAX_SOLVE_POINT_STEPS / npts))
    case.update(nt=max(10, nt if kind == "solve" else nt // 3), source=rng.choice(["p0", "plane", "u"]),
                absorbing=absorbing, nonlinear=rng.random() < 0.4, het=rng.random() < 0.75)
    if kind == "solve":
        case["record"] = rng.choice(["p", "p,u", "p_max,p_rms", "p,p_final"])
    else:
        case["record"] = rng.choice(["p_max,p_rms", "p_max,u_max", "p_max_all,u_final"])
        if case["source"] == "p0":
            case["source"] = "plane"  # a resident field is driven while it is advanced
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _f32(v):
    return float(np.float32(v))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grid_vectors(shape):
    """Index vectors along each axis of a [z][y][x] array, broadcastable."""
    n = len(shape)
    return [torch.arange(s, device="cuda", dtype=torch.float64).reshape([-1 if a == i else 1 for a in range(n)])
            for i, s in enumerate(shape)]


def _noise(shape, g, sigma=4.0):
    """Unit-variance white noise smoothed by a Gaussian of `sigma` points, [z][y][x], on the GPU."""
    z = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    for a, s in enumerate(shape):
        k = torch.fft.rfftfreq(s, device="cuda") if a == len(shape) - 1 else torch.fft.fftfreq(s, device="cuda")
        z *= torch.exp(-2 * (math.pi * sigma * k) ** 2).reshape([-1 if b == a else 1 for b in range(len(shape))])
    z = torch.fft.irfftn(z, s=shape)
    z -= z.mean()
    return z / z.std()


def _blobs(shape, rng):
    """Two smooth Gaussian blobs of pressure near the middle of the grid."""
    v = _grid_vectors(shape)
    p0 = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for amp in (5.0, 3.0):
        r2 = 0
        for s, x in zip(shape, v):
            r2 = r2 + (x - s * rng.uniform(0.35, 0.65)) ** 2
        p0 += amp * torch.exp(-r2 / (2 * 2.5 ** 2))
    return p0.float()


def _host(t):
    """A [z][y][x] GPU array as the (Nx, Ny[, Nz]) x-fastest host array the package takes."""
    return np.asfortranarray(t.cpu().numpy().T)


def _burst(nt, dt, f0, cycles, rng):
    t = np.arange(nt) * dt
    centre = cycles / f0 / 2 * 1.5
    return np.sin(2 * np.pi * f0 * t + rng.uniform(0, np.pi)) * np.exp(-((t - centre) * f0 / cycles * 3) ** 2)


def _datasets(case, seed):
    """The input datasets of one simulation (the names of the HDF5 input
    file), what to record, and the number of steps of a pass."""
    rng = np.random.default_rng(seed)
    g = _generator(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dim = 3 if nz > 1 else 2
    shape = (nz, ny, nx)[3 - dim:]
    pml = min(PML[dim], min(shape) // 5)
    resident = case["kind"] in ("resident", "batch")
    y = case["absorbing"]
    if case["het"]:
        c = 1500.0 + 40.0 * _noise(shape, g)
        rho = 1000.0 + 30.0 * _noise(shape, g)
        c_max = float(c.max())
    else:
        c, rho, c_max = None, None, 1500.0
    dt = _f32(0.3 * DX / c_max)
    inp = dict(Nx=nx, Ny=ny, Nz=nz, Nt=10_000_000 if resident else case["nt"], dx=_f32(DX), dy=_f32(DX),
               dz=_f32(DX) if dim == 3 else 0.0, dt=dt, c_ref=_f32(c_max))
    for a in "xyz"[:dim]:
        inp[f"pml_{a}_size"], inp[f"pml_{a}_alpha"] = pml, 2.0
    if case["het"]:
        inp["c0"], inp["rho0"] = _host(c), _host(rho)
        for i, a in enumerate("xyz"[:dim]):
            s = rho.clone()
            ax = dim - 1 - i
            n = shape[ax]
            s.narrow(ax, 0, n - 1).copy_(0.5 * (rho.narrow(ax, 0, n - 1) + rho.narrow(ax, 1, n - 1)))
            inp[f"rho0_sg{a}"] = _host(s)
    else:
        inp["c0"], inp["rho0"] = np.float32(1500.0), np.float32(1000.0)
        for a in "xyz"[:dim]:
            inp[f"rho0_sg{a}"] = np.float32(1000.0)
    if y:
        inp["absorbing_flag"], inp["alpha_power"] = (2 if y == 2.0 else 1), _f32(y)
        inp["alpha_coeff"] = np.float32(0.75)
    if case["nonlinear"]:
        inp["nonlinear_flag"], inp["BonA"] = 1, np.float32(6.0)

    src = case["source"]
    if src == "p0":
        inp["p0_source_flag"], inp["p0_source_input"] = 1, _host(_blobs(shape, rng))
    else:
        # one plane of points inside the layer; a resident field is driven by a long continuous wave
        zz, yy = np.meshgrid(np.arange(pml, nz - pml) if dim == 3 else np.zeros(1, int), np.arange(pml, ny - pml),
                             indexing="ij")
        pos = ((zz * ny + yy) * nx + pml + 1).ravel() + 1
        amp = 1e5 * rng.uniform(0.8, 1.2)
        if src == "dirichlet":
            # recorded boundary data of a point inside the grid, reversed in time
            cy, cz = rng.uniform(0.4, 0.6) * ny, rng.uniform(0.4, 0.6) * nz
            dist = np.sqrt((yy.ravel() - cy) ** 2 + (zz.ravel() - cz) ** 2 + (0.4 * nx) ** 2)
            t0 = (case["nt"] - dist[:, None] / 0.3)
            sig = np.exp(-((np.arange(case["nt"])[None, :] - t0) / 12.0) ** 2) * (1.0 / dist[:, None])
            sig = amp * sig / (dim * 1500.0 ** 2)
            mode, many = 0, 1
        else:
            nsig = 200_000 if resident else case["nt"]
            if resident:
                t = np.arange(nsig) * dt
                sig = np.sin(2 * np.pi * 1e6 * t + rng.uniform(0, np.pi)) * np.minimum(1.0, t * 1e6)
            else:
                sig = _burst(nsig, dt, 1e6, 3, rng)
            sig = (amp * sig * (2 * dt / (dim * 1500.0 * DX)))[None, :]
            mode, many = 2, 0
        if src == "u":
            sig = sig / 1e6
            inp.update(ux_source_flag=sig.shape[1], ux_source_input=sig.astype(np.float32), u_source_mode=1,
                       u_source_many=many, u_source_index=pos)
        else:
            inp.update(p_source_flag=sig.shape[1], p_source_mode=mode, p_source_many=many, p_source_index=pos,
                       p_source_input=sig.astype(np.float32))
    npts = nx * ny * nz
    if case.get("dense") or src == "dirichlet":
        idx = np.arange(1, npts + 1)
    else:
        idx = np.sort(rng.choice(npts, 200, replace=False)) + 1
    inp["sensor_mask_type"], inp["sensor_mask_index"] = 0, idx.astype(np.uint64)
    return inp, tuple(case["record"].split(",")), case["nt"]


def _members(case, seed):
    out = []
    for i, s in enumerate(case["shapes"].split(",")):
        nx, ny, nz = (int(v) for v in s.split("x"))
        m = dict(kind="batch", nx=nx, ny=ny, nz=nz, nt=case["nt"], source="plane", absorbing=case["absorbing"],
                 nonlinear=False, het=True, record=case["record"])
        out.append(_datasets(m, 1000 * int(seed) + i))
    return out


def _front_inputs(case, seed):
    """kgrid, medium, source, sensor of the front end (2D, smooth initial pressure, circle of 50 points)."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"])
    p0 = _host(_blobs(n[::-1], rng)).astype(np.float64)
    ang = 2 * np.pi * (np.arange(50) + rng.uniform(0, 1)) / 50
    cart = 0.31 * min(n) * DX * np.stack([np.cos(ang), np.sin(ang)])
    return n, p0, cart


def _front_dt():
    return 0.3 * DX / 1500.0


# ---------------------------------------------------------------------------
# the measured interface
# ---------------------------------------------------------------------------
def prepare(case, seed):
    from kwave import _lib

    kind = case["kind"]
    if kind == "gradient":
        f = _noise((case["ny"], case["nx"]), _generator(seed), 2.0).float().contiguous()
        return dict(kind=kind, lib=_lib, f=f, gx=torch.empty_like(f), gy=torch.empty_like(f), nx=case["nx"],
                    ny=case["ny"])
    if kind == "front":
        from kwave import KWaveGrid, kspaceFirstOrder2D

        n, p0, cart = _front_inputs(case, seed)
        kgrid = KWaveGrid(n, (DX, DX))
        kgrid.set_time(case["nt"], _front_dt())
        return dict(kind=kind, call=kspaceFirstOrder2D, kgrid=kgrid, medium={"sound_speed": 1500.0, "density": 1000.0},
                    source={"p0": p0}, sensor={"mask": cart, "record": case["record"].split(",")})
    if kind == "solve":
        inp, record, _ = _datasets(case, seed)
        return dict(kind=kind, lib=_lib, inp=inp, record=record)
    if kind == "resident":
        inp, record, nt = _datasets(case, seed)
        return dict(kind=kind, session=_lib.Session(inp, record), nt=nt)
    members = _members(case, seed)
    sessions = [_lib.Session(inp, record) for inp, record, _ in members]
    return dict(kind=kind, sessions=sessions, batch=_lib.Batch(sessions), nt=case["nt"])


def run(state):
    kind = state["kind"]
    if kind == "gradient":
        state["lib"].kspace_gradient_noalloc(state["f"].data_ptr(), state["gx"].data_ptr(), state["gy"].data_ptr(),
                                             state["nx"], state["ny"], DX, DX, 1500.0, _front_dt(),
                                             torch.cuda.current_stream().cuda_stream)
        return [state["gx"], state["gy"]]
    if kind == "front":
        return state["call"](state["kgrid"], state["medium"], state["source"], state["sensor"], smooth_p0=False)
    if kind == "solve":
        return state["lib"].solve(state["inp"], record=state["record"])
    if kind == "resident":
        state["session"].advance(state["nt"])
        return state["session"].read()
    state["batch"].advance(state["nt"])
    return [s.read() for s in state["sessions"]]


def _step_arrays(dim, het, y, nonlinear, ndense):
    """Full-grid FP32 arrays one time step reads or writes, each once; a
    transform of the grid reads and writes its field."""
    ffts = 2 * (1 + 3 * dim)                       # p, the gradient, u, the divergence
    arrays = 2 * dim + (dim if het else 0)         # u, 1 / rho0 on the staggered grids
    arrays += 2 * dim + (2 if het else 0)          # the split density, rho0 and c0^2
    if y and y != 2.0:
        ffts += 2 * 4
        arrays += 2 if het else 0                  # tau and eta
    elif y:
        arrays += 1 if het else 0
    return ffts + arrays + ndense


def work(case):
    kind = case["kind"]
    if kind == "gradient":
        n = case["nx"] * case["ny"]
        return dict(bytes=4 * n * 3, flops=3 * 2.5 * n * math.log2(n) + 20 * n)
    shapes = ([tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")] if kind == "batch"
              else [(case["nx"], case["ny"], case["nz"])])
    total = {"bytes": 0.0, "flops": 0.0}
    for s in shapes:
        n = s[0] * s[1] * s[2]
        dim = 3 if s[2] > 1 else 2
        y, het = case["absorbing"], case.get("het", True)
        nonlinear = case.get("nonlinear", False)
        dense = 4 if case.get("dense") else 0
        total["bytes"] += 4.0 * n * case["nt"] * _step_arrays(dim, het, y, nonlinear, dense)
        ffts = 1 + 3 * dim + (4 if y and y != 2.0 else 0)
        total["flops"] += case["nt"] * (ffts * 2.5 * n * math.log2(n) + 60.0 * n)
    return total


def tolerance(case):
    """Other correct single-precision transforms and orders of the sums give
    results this far apart after the steps of a pass (measured against the
    FP64 restatement below: 2e-7 to 7e-6 relative, the largest for a velocity
    component that a plane wave barely excites)."""
    if case["kind"] == "gradient":
        return {"rel": 3e-6, "max": 1e-4}
    return {"rel": 3e-5, "max": 1e-3}


# ---------------------------------------------------------------------------
# the time loop in FP64
# ---------------------------------------------------------------------------
def _wavenumbers(n, d):
    k = torch.fft.fftfreq(n, d=d, device="cuda", dtype=torch.float64) * 2 * math.pi
    return k


def _pml_profile(n, d, dt, c, size, alpha, staggered):
    x = torch.arange(1, size + 1, device="cuda", dtype=torch.float64) + (0.5 if staggered else 0.0)
    prof = torch.ones(n, device="cuda", dtype=torch.float64)
    if size:
        prof[:size] = torch.exp(-alpha * (c / d) * ((x - size - 1) / -size) ** 4 * dt / 2)
        prof[n - size:] = torch.exp(-alpha * (c / d) * (x / size) ** 4 * dt / 2)
    return prof


def _simulate(inp, record, steps):
    """Outputs of the first `steps` time steps, in FP64."""
    f8 = torch.float64
    nx, ny, nz = inp["Nx"], inp["Ny"], inp["Nz"]
    dim = 3 if nz > 1 else 2
    shape = (nz, ny, nx)[3 - dim:]
    axes = [dim - 1 - i for i in range(dim)]  # array axis of x, y, z
    d = [inp["dx"], inp["dy"], inp["dz"]][:dim]
    dt, c_ref = inp["dt"], inp["c_ref"]

    def along(v, i):
        return v.reshape([-1 if a == axes[i] else 1 for a in range(dim)])

    def fld(name):
        v = np.asarray(inp[name])
        if v.size == 1:
            return float(v)
        return torch.from_numpy(np.ascontiguousarray(v.T)).cuda().to(f8)

    def fwd(a):
        return torch.fft.rfftn(a)

    def inv(a):
        return torch.fft.irfftn(a, s=shape)

    kv = []
    for i in range(dim):
        k = _wavenumbers(inp["N" + "xyz"[i]], d[i])
        if i == 0:
            k = k[: nx // 2 + 1].abs()  # the half spectrum
        kv.append(along(k, i))
    k2 = sum(k ** 2 for k in kv)
    kk = torch.sqrt(k2)
    arg = c_ref * kk * dt / 2
    kappa = torch.where(arg == 0, torch.ones_like(arg), torch.sin(arg) / torch.where(arg == 0, torch.ones_like(arg), arg))
    src_kappa = torch.cos(arg)
    pos, neg = [], []
    for i in range(dim):
        n = inp["N" + "xyz"[i]]
        # the factor of the Nyquist bin is the part that survives taking the real part
        p, q = 1j * kv[i] * torch.exp(1j * kv[i] * d[i] / 2), 1j * kv[i] * torch.exp(-1j * kv[i] * d[i] / 2)
        if n % 2 == 0:
            at = [slice(None)] * dim
            at[axes[i]] = n // 2
            p[tuple(at)] = p[tuple(at)].real.to(p.dtype)
            q[tuple(at)] = q[tuple(at)].real.to(q.dtype)
        pos.append(p)
        neg.append(q)
    pml, pml_sg = [], []
    for i in range(dim):
        a = "xyz"[i]
        args = (inp["N" + a], d[i], dt, c_ref, inp[f"pml_{a}_size"], inp[f"pml_{a}_alpha"])
        pml.append(along(_pml_profile(*args, False), i))
        pml_sg.append(along(_pml_profile(*args, True), i))
    c0, rho0 = fld("c0"), fld("rho0")
    rinv = [1.0 / fld("rho0_sg" + a) for a in "xyz"[:dim]]
    eos = inp.get("absorbing_flag", 0)
    if eos:
        y = inp["alpha_power"]
        al = 100 * float(inp["alpha_coeff"]) * (1e-6 / (2 * math.pi)) ** y / (20 * math.log10(math.e))
        tau = -2 * al * c0 ** (y - 1)
        if eos == 1:
            eta = 2 * al * c0 ** y * math.tan(math.pi * y / 2)
            safe = torch.where(kk == 0, torch.ones_like(kk), kk)
            nab1, nab2 = (torch.where(kk == 0, torch.zeros_like(kk), safe ** e) for e in (y - 2, y - 1))
            if y == 1:
                nab2 = torch.ones_like(kk)
    bona = float(inp["BonA"]) if inp.get("nonlinear_flag") else None

    def signal(prefix):
        if not inp.get(prefix + "_source_flag"):
            return None
        s = np.asarray(inp[prefix + "_source_input"])[:, :steps]
        return torch.from_numpy(np.ascontiguousarray(s.T)).cuda().to(f8)

    p_sig, u_sig = signal("p"), signal("ux")

    def points(name):
        return torch.from_numpy(np.asarray(inp[name]).astype(np.int64) - 1).cuda()

    p_idx = points("p_source_index") if p_sig is not None else None
    u_idx = points("u_source_index") if u_sig is not None else None
    sensors = points("sensor_mask_index")
    p = torch.zeros(shape, device="cuda", dtype=f8)
    u = [torch.zeros_like(p) for _ in range(dim)]
    rho = [torch.zeros_like(p) for _ in range(dim)]
    acc, series, run_max, run_sq = {}, {}, {}, {}
    wanted = set(record)
    for t in range(steps):
        pk = fwd(p) * kappa
        for i in range(dim):
            u[i] = pml_sg[i] * (pml_sg[i] * u[i] - dt * rinv[i] * inv(pos[i] * pk))
        if u_sig is not None and t < u_sig.shape[0]:
            v = u[0].reshape(-1)
            if inp["u_source_mode"] == 1:
                v[u_idx] += u_sig[t]
            else:
                raise ValueError("source mode")
        du = [inv(neg[i] * kappa * fwd(u[i])) for i in range(dim)]
        r = rho0 if bona is None else 2 * sum(rho) + rho0
        rho = [pml[i] * (pml[i] * rho[i] - dt * r * du[i]) for i in range(dim)]
        if p_sig is not None and t < p_sig.shape[0]:
            if inp["p_source_mode"] == 0:
                for x in rho:
                    x.reshape(-1)[p_idx] = p_sig[t]
            else:
                s = torch.zeros_like(p)
                s.reshape(-1)[p_idx] = p_sig[t]
                s = inv(src_kappa * fwd(s))
                rho = [x + s for x in rho]
        rs = sum(rho)
        term = rs
        if eos == 1:
            term = term + tau * inv(nab1 * fwd(rho0 * sum(du))) - eta * inv(nab2 * fwd(rs))
        elif eos == 2:
            term = term + tau * rho0 * sum(du)
        if bona is not None:
            term = term + bona * rs ** 2 / (2 * rho0)
        p = c0 ** 2 * term
        if t == 0 and inp.get("p0_source_flag"):
            p = fld("p0_source_input")
            rho = [p / (dim * c0 ** 2) for _ in range(dim)]
            pk = fwd(p) * kappa
            u = [dt * rinv[i] * inv(pos[i] * pk) / 2 for i in range(dim)]
        fields = {"p": p}
        fields.update({"u" + a: u[i] for i, a in enumerate("xyz"[:dim])})
        for name, x in fields.items():
            q = "u" if name[0] == "u" else "p"
            at = x.reshape(-1)[sensors]
            if q in wanted:
                series.setdefault(name, []).append(at.clone())
            if q + "_max" in wanted:
                run_max[name] = at.clone() if t == 0 else torch.maximum(run_max[name], at)
            if q + "_max_all" in wanted:
                acc[name + "_max_all"] = x.clone() if t == 0 else torch.maximum(acc[name + "_max_all"], x)
            if q + "_rms" in wanted:
                run_sq[name] = at ** 2 if t == 0 else run_sq[name] + at ** 2
            if q + "_final" in wanted and t == steps - 1:
                acc[name + "_final"] = x
    out = {k: torch.stack(v, 1) for k, v in series.items()}
    out.update({k + "_max": v for k, v in run_max.items()})
    out.update({k + "_rms": torch.sqrt(v / steps) for k, v in run_sq.items()})
    out.update({k: v.permute(*range(dim - 1, -1, -1)) for k, v in acc.items()})
    return {k: v.cpu().numpy() for k, v in out.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        f = _noise((case["ny"], case["nx"]), _generator(seed), 2.0).double()
        kx = _wavenumbers(case["nx"], _f32(DX)).reshape(1, -1)
        ky = _wavenumbers(case["ny"], _f32(DX)).reshape(-1, 1)
        kappa = torch.sinc(_f32(1500.0) * torch.sqrt(kx ** 2 + ky ** 2) * _f32(_front_dt()) / (2 * math.pi))
        fk = torch.fft.fft2(f) * kappa
        return [torch.fft.ifft2(1j * k * torch.exp(1j * k * _f32(DX) / 2) * fk).real for k in (kx, ky)]
    if kind == "front":
        n, p0, cart = _front_inputs(case, seed)
        dt = _f32(_front_dt())
        inp = dict(Nx=n[0], Ny=n[1], Nz=1, dx=_f32(DX), dy=_f32(DX), dz=0.0, dt=dt, c_ref=1500.0, c0=1500.0,
                   rho0=1000.0, rho0_sgx=1000.0, rho0_sgy=1000.0, p0_source_flag=1, p0_source_input=p0)
        for a in "xy":
            inp[f"pml_{a}_size"], inp[f"pml_{a}_alpha"] = PML[2], 2.0
        ix = [np.floor(np.abs(cart[i] / DX) + 0.5) * np.sign(cart[i]) + n[i] // 2 for i in range(2)]
        inp["sensor_mask_index"] = (ix[1] * n[0] + ix[0] + 1).astype(np.int64)
        return _simulate(inp, case["record"].split(","), case["nt"])
    if kind == "batch":
        return [_simulate(inp, record, nt) for inp, record, nt in _members(case, seed)]
    inp, record, nt = _datasets(case, seed)
    return _simulate(inp, record, nt)
