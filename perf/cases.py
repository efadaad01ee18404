"""The work that a user of this framework has it do, as cases to measure.

A case names one call sequence of the public Python API (package `grt` in
gr-ray-tracer_b200, a ctypes binding of the C ABI in include/grt.h) with its
sizes and options:

  frame    one image the way the reference renders it: camera rays, the step
           loop, the image products on the host
  batch    a set of images (inclinations x frequency channels, mixed sizes) in
           one launch through the render graph, products as one device block
  stream   host photon blocks rendered asynchronously on two contexts in turn
  disk     disk-mode scattering Monte Carlo: emission, transport, photons back
  adjoint  a Stokes-I image of line-of-sight rays and the gradient of a loss
           on it with respect to per-cell multipliers (torch autograd)
  inplace  photons and grid in device memory the caller owns, traced without
           any allocation

The black hole, the torus and the camera are those of grt.workloads; a seed
moves the camera (azimuth, a degree of inclination), the turbulence of the
torus and the frequencies, so that no two seeds see the same rays or cells.
"""

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gr-ray-tracer_b200"))

from grt import abi, autograd, lib, torus, workloads  # noqa: E402

CHANNELS_GHZ = workloads.FREQ_CHANNELS_GHZ


def _frame(**kw):
    case = dict(kind="frame", nx=256, ny=256, nr=128, ntheta=64, nphi=64, spin=0.94, incl=17.0, integrator="rk45",
                mixed=False, random_screen=False, generator="custom", stop=1.0, interval=10**9)
    case.update(kw)
    return case


def _batch(**kw):
    case = dict(kind="batch", inclinations=1, channels=4, px_lo=256, px_hi=256, sizes_seed=3, nr=128, ntheta=64, nphi=64,
                spin=0.94, incl=17.0, incl_hi=17.0, mixed=True)
    case.update(kw)
    return case


def listed():
    return [
        # a thumbnail while a camera is being placed: a handful of rays, all latency and launches
        _frame(name="frame_thumbnail_16", nx=16, ny=16, nr=64, ntheta=32, nphi=32, spin=0.9, incl=60.0),
        # the RK4 workload of the benchmark (fixed steps, 64x64, 60 degrees): one lane per ray, a long serial chain
        _frame(name="frame_rk4_64", nx=64, ny=64, nr=64, ntheta=32, nphi=32, spin=0.9, incl=60.0, integrator="rk4"),
        # the reference's own defaults for its step loop: the termination test on every step, stop at 90%
        _frame(name="frame_every_step_128", nx=128, ny=128, spin=0.9, incl=45.0, stop=0.9, interval=1),
        # the RK45 workload of the benchmark: one 256x256 image, FP64 form
        _frame(name="frame_rk45_256", nx=256, ny=256),
        # a wide screen with odd sides seen almost edge on, mixed form, the reference's random screen and its
        # default (blackbody) generator on a grid with odd extents
        _frame(name="frame_ragged_509x283", nx=509, ny=283, nr=97, ntheta=49, nphi=35, spin=0.5, incl=84.0,
               mixed=True, random_screen=True, generator="blackbody"),
        # the benchmark's headline: the 256x256 image at four frequency channels, mixed form
        _batch(name="batch_channels_256x4"),
        # the benchmark's image library: 16 inclinations x 4 channels, sizes 64..512
        _batch(name="batch_library_64", inclinations=16, px_lo=64, px_hi=512, spin=0.9, incl=5.0, incl_hi=85.0),
        # a host program that owns the photons and streams renders: upload, trace and products of two renders
        dict(name="stream_256x4", kind="stream", nx=256, ny=256, channels=4, nr=128, ntheta=64, nphi=64, spin=0.94,
             incl=17.0, mixed=True),
        # disk mode, a quick look: about 1e5 packets on a small torus
        dict(name="disk_small", kind="disk", nr=64, ntheta=32, nphi=32, spin=0.9, norm=20.0),
        # disk mode at production size: about 2e6 packets on the full torus
        dict(name="disk_large", kind="disk", nr=128, ntheta=64, nphi=64, spin=0.9, norm=45.0),
        # the benchmark's differentiable render: 128x128, forward and backward
        dict(name="adjoint_128", kind="adjoint", nx=128, ny=128, nr=96, ntheta=48, nphi=48, spin=0.9, incl=60.0, every=64),
        # a solver that embeds the tracer and owns all device memory: 100x100 rays traced in place
        dict(name="inplace_100", kind="inplace", nx=100, ny=100, nr=64, ntheta=48, nphi=32, spin=0.7, incl=30.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    grid = dict(nr=rng.randint(48, 128), ntheta=rng.randint(24, 64), nphi=rng.randint(16, 64),
                spin=round(rng.uniform(0.0, 0.98), 3))
    incl = round(rng.uniform(5.0, 85.0), 1)
    kind = rng.choice(["frame", "frame", "frame", "batch", "batch", "stream", "disk", "disk", "adjoint", "inplace"])
    if kind == "frame":
        integrator = rng.choice(["rk45", "rk45", "rk45", "rk4"])
        nx = _log(rng, 12, 160 if integrator == "rk4" else 640)
        every_step = integrator == "rk45" and rng.random() < 0.25
        return _frame(nx=nx, ny=max(8, int(nx * rng.uniform(0.5, 1.5))), incl=incl, integrator=integrator,
                      mixed=rng.random() < 0.4, random_screen=rng.random() < 0.3,
                      generator=rng.choice(["custom", "custom", "blackbody", "power_law"]),
                      stop=0.9 if every_step else 1.0, interval=1 if every_step else 10**9, **grid)
    if kind == "batch":
        lo = _log(rng, 24, 200)
        return _batch(inclinations=rng.randint(1, 10), channels=rng.randint(1, 4), px_lo=lo,
                      px_hi=min(450, int(lo * rng.uniform(1.0, 3.0))), sizes_seed=rng.randint(0, 10**6),
                      incl=incl, incl_hi=min(88.0, incl + rng.uniform(0.0, 40.0)), mixed=rng.random() < 0.6, **grid)
    if kind == "stream":
        nx = _log(rng, 48, 400)
        return dict(kind=kind, nx=nx, ny=max(32, int(nx * rng.uniform(0.6, 1.4))), channels=rng.randint(1, 4), incl=incl,
                    mixed=rng.random() < 0.6, **grid)
    if kind == "disk":
        return dict(kind=kind, norm=float(_log(rng, 15, 60)), **grid)
    nx = _log(rng, 20, 200)
    ny = max(16, int(nx * rng.uniform(0.6, 1.4)))
    if kind == "adjoint":
        return dict(kind=kind, nx=nx, ny=ny, every=rng.choice([16, 32, 64]), incl=incl, **grid)
    return dict(kind=kind, nx=nx, ny=ny, incl=incl, **grid)


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=4)
def _still_torus(nr, ntheta, nphi, spin):
    return torus.benchmark_torus(nr, ntheta, nphi, spin=spin)


def _torus(case, rng):
    """The workloads' torus with 10% lognormal turbulence in temperature and density (disk mode: in temperature, as
    the density sets the number of packets)."""
    still = _still_torus(case["nr"], case["ntheta"], case["nphi"], case["spin"])
    inside = still["rho.npy"] > 1.0e-6
    out = dict(still)
    for field in ("Tgas.npy",) if case["kind"] == "disk" else ("rho.npy", "Tgas.npy"):
        wind = np.exp(rng.normal(0.0, 0.1, inside.shape))
        out[field] = np.where(inside, still[field] * wind, still[field])
    return out


def _params(case, rng):
    if case["kind"] == "disk":
        w = workloads.DiskWorkload("disk", (case["nr"], case["ntheta"], case["nphi"]), case["spin"], case["norm"])
        return w.params().update(scattering_seed=int(rng.integers(1, 2**31)))
    rk4 = case.get("integrator") == "rk4"
    extra = dict(workloads.C4.extra) if case["kind"] == "adjoint" else {}
    w = workloads.ImageWorkload("image", (case["nr"], case["ntheta"], case["nphi"]), case["spin"], case["incl"],
                                case.get("nx", case.get("px_lo")), abi.RK4 if rk4 else abi.RK45,
                                0.002 if rk4 else 0.01, 1200 if rk4 else 4000, extra=extra)
    p = w.params()
    p.update(camera_theta=math.radians(case["incl"] + rng.uniform(-0.5, 0.5)), camera_phi=rng.uniform(0.0, 2.0 * math.pi),
             custom_frequency_hz=2.3e11 * math.exp(rng.normal(0.0, 0.05)),
             precision=abi.PREC_MIXED if case.get("mixed") else abi.PREC_FP64,
             generator={"custom": abi.GEN_CUSTOM, "blackbody": abi.GEN_BLACKBODY,
                        "power_law": abi.GEN_POWER_LAW}[case.get("generator", "custom")],
             termination_percent=case.get("stop", 1.0), output_interval=case.get("interval", 10**9))
    if "nx" in case:
        p.update(image_nx=case["nx"], image_ny=case["ny"], nphotons=case["nx"] * case["ny"])
    return p


def _images(case):
    """(inclination, pixels a side, channel) of every image of a batch."""
    size = np.random.default_rng(case["sizes_seed"])
    lo, hi = case["px_lo"], case["px_hi"]
    steps = [v for v in (64, 128, 256, 512) if lo <= v <= hi]
    out = []
    for incl in np.linspace(case["incl"], case["incl_hi"], case["inclinations"]):
        for f in CHANNELS_GHZ[:case["channels"]]:
            if lo == 64 and hi == 512:  # the benchmark's library: sizes of its list
                px = steps[size.integers(0, len(steps))]
            else:
                px = int(size.integers(lo, hi + 1))
            out.append((float(incl), int(px), f))
    return out


def _specs(case, p):
    """The image specs of a case's batch: its images' cameras, moved as the params' camera was moved."""
    if case["kind"] == "stream":
        images = [(case["incl"], (case["nx"], case["ny"]), f) for f in CHANNELS_GHZ[:case["channels"]]]
    else:
        images = [(incl, (px, px), f) for incl, px, f in _images(case)]
    moved = p.camera_theta - math.radians(case["incl"])
    return [abi.ImageSpec.from_params(p, nx, ny, camera_theta=math.radians(incl) + moved,
                                      custom_frequency_hz=p.custom_frequency_hz * f / 230.0,
                                      emission_coefficient=p.emission_coefficient * f / 230.0)
            for incl, (nx, ny), f in images]


def _pinned_products(p, nx, ny):
    out = abi.ProductArrays(0, 0, 0)
    out.nx, out.ny, out.bins = nx, ny, int(p.spectrum_bins)
    for field, shape in (("image_I", (ny, nx)), ("image_Q", (ny, nx)), ("image_U", (ny, nx)), ("image_V", (ny, nx)),
                         ("spectrum_frequency_hz", (out.bins,)), ("spectrum_I", (out.bins,))):
        setattr(out, field, torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy())
    out.arrived_count = torch.zeros(1, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    return out


def _pinned_photons(n):
    return abi.PhotonArrays.block(n, torch.zeros(146 * n, dtype=torch.uint8, pin_memory=True).numpy())


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 20])
    p, grid = _params(case, rng), _torus(case, rng)
    state = dict(case=case, params=p)
    kind = case["kind"]
    if kind == "adjoint":
        shape = grid["r.npy"].shape
        state["renderer"] = autograd.ImageRenderer(p, grid, checkpoint_interval=case["every"],
                                                   back_distance=workloads.C4_BACK_DISTANCE)
        state["grid"] = grid
        for name in ("m_abs", "m_emis"):
            state[name] = torch.from_numpy(np.exp(rng.normal(0.0, 0.1, shape))).cuda()
        state["weights"] = torch.from_numpy(rng.normal(0.0, 1.0, (case["ny"], case["nx"]))).cuda()
        return state
    if kind == "inplace":
        with lib.Context(p) as ctx:
            ctx.upload_grid(None)
            ctx.init_image_photons(case["nx"], case["ny"])
            photons = ctx.download_photons()
        state["start"] = {f: torch.from_numpy(getattr(photons, f).view(np.int64) if f == "id" else getattr(photons, f)).cuda()
                          for f in abi.PHOTON_FIELDS}
        state["photons"] = {f: t.clone() for f, t in state["start"].items()}
        state["soa"] = abi.PhotonSoA(*[abi.C.cast(state["photons"][f].data_ptr(), kind_of)
                                       for f, kind_of in abi.PhotonSoA._fields_])
        state["fields"] = [torch.from_numpy(grid[k]).cuda() for k in torus.FIELD_FILES]
        state["grid"] = abi.DeviceGrid(*grid["r.npy"].shape, *[t.data_ptr() for t in state["fields"]])
        return state
    count = 2 if kind == "stream" else 1
    state["contexts"] = [lib.Context(p) for _ in range(count)]
    for ctx in state["contexts"]:
        ctx.upload_grid(grid)
    ctx = state["contexts"][0]
    if kind == "frame":
        state["products"] = abi.ProductArrays.for_params(p)
    elif kind == "disk":
        state["photons"] = _pinned_photons(ctx.init_disk_photons())
    else:
        state["stream"] = torch.cuda.Stream()
        specs = _specs(case, p)
        for c in state["contexts"]:
            c.set_stream(state["stream"].cuda_stream)
            c.init_image_batch(specs)
        if kind == "batch":
            state["block"] = torch.empty(ctx.products_block_bytes // 8, dtype=torch.float64, device="cuda")
            state["split"] = [4 * sum(s.nx * s.ny for s in specs), len(specs) * int(p.spectrum_bins), len(specs)]
        else:
            state["photons"] = [_pinned_photons(c.n) for c in state["contexts"]]
            for c, photons in zip(state["contexts"], state["photons"]):
                c.download_photons(photons)
            state["products"] = [[_pinned_products(p, s.nx, s.ny) for s in specs] for _ in state["contexts"]]
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _counts(stats):
    return {k: stats[k] for k in ("steps_done", "n_terminated", "accepted_steps", "photon_calls")}


def _run_frame(state):
    case, (ctx,) = state["case"], state["contexts"]
    if case["random_screen"]:
        ctx.init_image_photons_random(case["nx"] * case["ny"])
    else:
        ctx.init_image_photons(case["nx"], case["ny"])
    stats = ctx.run()
    return dict(ctx.image_products(state["products"]).as_dict(), **_counts(stats))


def _run_batch(state):
    (ctx,), block = state["contexts"], state["block"]
    stats = ctx.render_graph()
    ctx.copy_products_block(block.data_ptr(), block.numel() * 8)
    images, spectra, arrived = torch.split(block, state["split"])
    return dict(images=images, spectra=spectra, arrived=arrived.view(torch.int64), **_counts(stats))


def _run_stream(state):
    for ctx, photons, products in zip(state["contexts"], state["photons"], state["products"]):
        ctx.render_async(photons, products)
    stats = [ctx.render_wait() for ctx in state["contexts"]]
    return [dict(_counts(s), images=[o.as_dict() for o in products]) for s, products in zip(stats, state["products"])]


def _run_disk(state):
    (ctx,) = state["contexts"]
    ctx.init_disk_photons()
    stats = ctx.run()
    return dict(ctx.download_photons(state["photons"]).as_dict(), **_counts(stats))


def _run_adjoint(state):
    m_abs = state["m_abs"].clone().requires_grad_(True)
    m_emis = state["m_emis"].clone().requires_grad_(True)
    image = state["renderer"].render(m_abs, m_emis)
    loss = (image * state["weights"]).sum()
    g_abs, g_emis = torch.autograd.grad(loss, (m_abs, m_emis))
    return dict(image=image, g_abs=g_abs, g_emis=g_emis)


def _run_inplace(state):
    for f, t in state["photons"].items():
        t.copy_(state["start"][f])
    stats = lib.trace_device_noalloc(state["params"], state["grid"], state["soa"], state["start"]["id"].numel())
    return dict(state["photons"], **_counts(stats))


# ---------------------------------------------------------------- the work of a pass
def work(case):
    """FP64 operations (one right-hand side is 243, an RK4 step 1100, an RK45 attempt 1691; the steps and attempts
    per ray are means of the benchmark's workloads) and bytes (grid, photons and products once each)."""
    cells = case["nr"] * case["ntheta"] * case["nphi"]
    kind = case["kind"]
    if kind == "disk":
        packets = 47000.0 * case["norm"] * cells / (128 * 64 * 64)
        return dict(bytes=80 * cells + 146 * packets, flops=packets * (48 * 243 + 70 * 1691))
    rk45 = 34 * 243 + 55 * 1691
    if kind == "batch":
        sizes = _images(case)
        rays = sum(px * px for _, px, _ in sizes)
        geodesics = sum(px * px for _, px in {(incl, px) for incl, px, _ in sizes})
        return dict(bytes=80 * cells + (146 + 32) * rays, flops=geodesics * rk45)
    n = case["nx"] * case["ny"]
    if kind == "stream":
        return dict(bytes=2 * (80 * cells + (2 * 146 + 32) * n * case["channels"]), flops=2 * n * rk45)
    if kind == "adjoint":
        return dict(bytes=112 * cells + (2 * 146 + 8) * n, flops=2 * n * (45 * 243 + 60 * 1691))
    per_ray = 950 * 1100 if case.get("integrator") == "rk4" else rk45
    return dict(bytes=80 * cells + (146 + 32) * n, flops=n * per_ray)


# ---------------------------------------------------------------- the values in 64 bits, without the framework's code
# The step-size controller amplifies rounding (far from the hole the error estimate of a step IS rounding), so the
# expressions below keep the reference's order of operations: in another order the rays land in other cells.
def _radius(x, y, z, a):
    rsq = x * x + y * y + z * z
    A = rsq - a * a
    return torch.sqrt(0.5 * (A + torch.sqrt(A * A + 4.0 * ((a * z) * (a * z)))))


def _metric(x, y, z, r, a, M):
    """l_mu and g_{mu nu} = eta + 2 H l_mu l_nu."""
    B = r * r + a * a
    ell = [torch.ones_like(r), (r * x + a * y) / B, (r * y - a * x) / B, z / r]
    two_h = 2.0 * (M * (r * r * r) / (r * r * r * r + (a * z) * (a * z)))
    g = [[two_h * ell[m] * ell[n] + (0.0 if m != n else -1.0 if m == 0 else 1.0) for n in range(4)] for m in range(4)]
    return ell, g


def _lower(g, u):
    return [((g[m][0] * u[0] + g[m][1] * u[1]) + g[m][2] * u[2]) + g[m][3] * u[3] for m in range(4)]


def _dot(g, u, v):
    total = 0.0
    for m in range(4):
        for n in range(4):
            total = total + g[m][n] * u[m] * v[n]
    return total


def _rhs(s, pt, a, M):
    """d(t, x, y, z, p_x, p_y, p_z)/dlambda of the Kerr-Schild Hamiltonian."""
    x, y, z, px, py, pz = s[1], s[2], s[3], s[4], s[5], s[6]
    rsq = x * x + y * y + z * z
    A = rsq - a * a
    S = torch.sqrt(A * A + 4.0 * ((a * z) * (a * z)))
    r = torch.sqrt(0.5 * (A + S))
    one = 1.0 + A / S
    dr = [x * one / (2.0 * r), y * one / (2.0 * r), (z * one + 2.0 * (a * a) * z / S) / (2.0 * r)]
    B = r * r + a * a
    l1, l2, l3 = (r * x + a * y) / B, (r * y - a * x) / B, z / r
    r2 = r * r
    r3 = r2 * r
    D = r3 * r + (a * z) * (a * z)
    H = M * r3 / D
    lp = ((-pt + l1 * px) + l2 * py) + l3 * pz
    two_h = 2.0 * H
    out = [-pt - (-two_h) * lp, px - two_h * l1 * lp, py - two_h * l2 * lp, pz - two_h * l3 * lp]
    lp2, c = lp * lp, two_h * lp
    for k in range(3):
        dB = 2.0 * r * dr[k]
        d1 = (dr[k] * x + r if k == 0 else dr[k] * x + a if k == 1 else dr[k] * x) - l1 * dB
        d2 = (dr[k] * y - a if k == 0 else dr[k] * y + r if k == 1 else dr[k] * y) - l2 * dB
        dl1, dl2, dl3 = d1 / B, d2 / B, ((1.0 if k == 2 else 0.0) - l3 * dr[k]) / r
        dD = 4.0 * r3 * dr[k]
        if k == 2:
            dD = dD + 2.0 * (a * a) * z
        dH = M * (3.0 * r2 * dr[k] * D - r3 * dD) / (D * D)
        out.append(dH * lp2 + c * ((dl1 * px + dl2 * py) + dl3 * pz))
    return torch.stack(out)


def _fourth_root(x):
    """x^(1/4) to well under an ulp: two square roots and a correction from the residual in double-double."""
    y = torch.sqrt(torch.sqrt(x))

    def product(u, v):
        uh, vh = u * 134217729.0, v * 134217729.0
        uh, vh = uh - (uh - u), vh - (vh - v)
        ul, vl, top = u - uh, v - vh, u * v
        return top, ((uh * vh - top) + uh * vl + ul * vh) + ul * vl

    sq, sq_lo = product(y, y)
    q, q_lo = product(sq, sq)
    rest = (x - q) - (q_lo + 2.0 * sq * sq_lo)
    better = y + rest / (4.0 * sq * y)
    return torch.where(torch.isfinite(better), better, y)


_A = ((1 / 4,), (3 / 32, 9 / 32), (1932 / 2197, -7200 / 2197, 7296 / 2197), (439 / 216, -8.0, 3680 / 513, -845 / 4104),
      (-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40))
_B4 = (25 / 216, 0.0, 1408 / 2565, 2197 / 4104, -1 / 5, 0.0)
_B5 = (16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55)


def _combine(weights, k):
    total = None
    for w, ki in zip(weights, k):
        if w:
            total = w * ki if total is None else total + w * ki
    return total


def _rk4(s, pt, dl, a, M):
    k = _rhs(s, pt, a, M)
    total = k
    for c, w in ((0.5, 2.0), (0.5, 2.0), (1.0, 1.0)):
        k = _rhs(s + (c * dl) * k, pt, a, M)
        total = total + w * k
    return s + dl / 6.0 * total


def _rk45(s, pt, dl, p):
    """One call of the adaptive step (up to 12 attempts): the new state, the step taken, the next one, accepted."""
    a, M = p.spin, p.mass
    new, nxt = s.clone(), dl.clone()
    taken, done = dl.clone(), torch.zeros_like(dl, dtype=torch.bool)
    at = torch.arange(dl.numel(), device=dl.device)
    k1 = _rhs(s, pt, a, M)
    for _ in range(12):
        if at.numel() == 0:
            break
        h, s0, k, e = nxt[at], s[:, at], [k1[:, at]], pt[at]
        for row in _A:
            k.append(_rhs(s0 + h * _combine(row, k), e, a, M))
        x4, x5 = s0 + h * _combine(_B4, k), s0 + h * _combine(_B5, k)
        err = ((x5 - x4).abs() / (p.atol + p.rtol * torch.maximum(x5.abs(), x4.abs()))).amax(0)
        scale = torch.clamp(p.safety * _fourth_root(1.0 / err), p.min_step_scale, p.max_step_scale)
        scale = torch.where(err == 0.0, torch.full_like(scale, p.max_step_scale), scale)
        finite = torch.isfinite(x5).all(0) & torch.isfinite(err)
        scale = torch.where(finite, scale, torch.full_like(scale, p.min_step_scale))
        ok = finite & (err <= 1.0)
        taken[at] = h
        nxt[at] = h * scale
        new[:, at[ok]] = x5[:, ok]
        done[at[ok]] = True
        at = at[~ok]
    return new, taken, nxt, done


class _Fluid:
    """Nearest-cell lookup and cell data of a separable grid."""

    def __init__(self, grid, p, dev):
        self.p = p
        f = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in grid.items()}
        self.shape = tuple(f["r.npy"].shape)
        self.axes = [f["r.npy"][:, 0, 0].contiguous(), f["theta.npy"][0, :, 0].contiguous(), f["phi.npy"][0, 0, :].contiguous()]
        ratio, polar, turn = torch.log(self.axes[0]), self.axes[1], self.axes[2]
        self.half = []
        for axis, periodic in ((ratio, False), (polar, False), (turn, True)):
            gap = (axis[1:] - axis[:-1]).abs()
            if periodic:
                gap = torch.minimum(gap, 2.0 * math.pi - gap)
            none = gap.new_zeros(1)
            self.half.append(0.500001 * torch.maximum(torch.cat([gap, none]), torch.cat([none, gap])))
        self.rho = f["rho.npy"].reshape(-1) * p.density_g_cm3_per_code
        self.T = f["Tgas.npy"].reshape(-1) * p.temperature_k_per_code
        self.vel = f["vel.npy"].reshape(-1, 4)
        self.r, self.th, self.ph = (f[k].reshape(-1) for k in ("r.npy", "theta.npy", "phi.npy"))

    @staticmethod
    def _near(axis, q):
        hi = torch.searchsorted(axis, q.contiguous()).clamp(1, axis.numel() - 1)
        return torch.where((axis[hi] - q).abs() < (q - axis[hi - 1]).abs(), hi, hi - 1)

    def four_velocity(self, cell):
        a, r, v = self.p.spin, self.r[cell], self.vel[cell]
        st, ct, sp, cp = self.th[cell].sin(), self.th[cell].cos(), self.ph[cell].sin(), self.ph[cell].cos()
        u = [v[:, 0],
             cp * st * v[:, 1] + (r * cp - a * sp) * ct * v[:, 2] + (-r * sp - a * cp) * st * v[:, 3],
             sp * st * v[:, 1] + (r * sp + a * cp) * ct * v[:, 2] + (r * cp - a * sp) * st * v[:, 3],
             ct * v[:, 1] - r * st * v[:, 2]]
        return [ui * self.p.four_velocity_cm_s_per_code for ui in u]

    def sample(self, s):
        """(cell or -1, the fluid's unit four-velocity there) at each position."""
        a, x, y, z = self.p.spin, s[1], s[2], s[3]
        r = _radius(x, y, z, a)
        az = torch.atan2(r * y - a * x, r * x + a * y)
        az = torch.where(az < 0.0, az + 2.0 * math.pi, az)
        polar = torch.acos(torch.clamp(z / r, -1.0, 1.0))
        lr = torch.log(self.axes[0])
        i, j = self._near(lr, torch.log(r)), self._near(self.axes[1], polar)
        turn = torch.cat([self.axes[2][-1:] - 2.0 * math.pi, self.axes[2], self.axes[2][:1] + 2.0 * math.pi])
        k = (self._near(turn, az) - 1) % self.shape[2]
        da = (az - self.axes[2][k]).abs()
        da = torch.minimum(da, 2.0 * math.pi - da)
        ok = ((torch.log(r) - lr[i]).abs() <= self.half[0][i]) & ((polar - self.axes[1][j]).abs() <= self.half[1][j])
        ok &= da <= self.half[2][k]
        cell = (i * self.shape[1] + j) * self.shape[2] + k
        ok &= self.rho[cell] > 0.0
        u = self.four_velocity(cell)
        _, g = _metric(x, y, z, r, a, self.p.mass)
        norm = _dot(g, u, u)
        ok &= norm < 0.0
        inverse = 1.0 / torch.sqrt(-norm)
        sign = torch.where(u[0] >= 0.0, 1.0, -1.0).to(inverse.dtype)
        return torch.where(ok, cell, torch.full_like(cell, -1)), [sign * v * inverse for v in u]


def _camera(specs, dev, back):
    rows = []
    for s in specs:
        st, ct, sp, cp = math.sin(s.camera_theta), math.cos(s.camera_theta), math.sin(s.camera_phi), math.cos(s.camera_phi)
        rows.append([st * cp, st * sp, ct, ct * cp, ct * sp, -st, -sp, cp, 0.0, s.camera_distance, s.camera_width,
                     s.camera_height, s.custom_frequency_hz, s.absorption_coefficient, s.emission_coefficient])
        for D in (s.camera_distance, -back):  # where a backward, a forward ray through the centre starts
            rows[-1] += [D * st * cp, D * st * sp, D * ct]
    return torch.tensor(rows, dtype=torch.float64, device=dev)


def _rays(p, specs, cam, dev, back=0.0):
    """Camera rays through the pixel centres of every image: state [7, n], p_t, image index, screen position."""
    img, u, v = [], [], []
    for q, s in enumerate(specs):
        ix = -0.5 * s.camera_width + (torch.arange(s.nx, dtype=torch.float64, device=dev) + 0.5) * s.camera_width / s.nx
        iy = -0.5 * s.camera_height + (torch.arange(s.ny, dtype=torch.float64, device=dev) + 0.5) * s.camera_height / s.ny
        u.append(ix.repeat(s.ny))
        v.append(iy.repeat_interleave(s.nx))
        img.append(torch.full((s.nx * s.ny,), q, dtype=torch.int64, device=dev))
    img, u, v = torch.cat(img), torch.cat(u), torch.cat(v)
    c = cam[img].T
    x, y, z = (c[(18 if back else 15) + q] + u * c[3 + q] + v * c[6 + q] for q in range(3))
    K = [(1.0 if back else -1.0) * c[15 + q] for q in range(3)]
    length = torch.sqrt(K[0] * K[0] + K[1] * K[1] + K[2] * K[2])
    K = [k / length for k in K]
    _, g = _metric(x, y, z, _radius(x, y, z, p.spin), p.spin, p.mass)
    qa, qb = g[0][0], 2.0 * (g[0][1] * K[0] + g[0][2] * K[1] + g[0][3] * K[2])
    qc = 0.0
    for i in range(3):
        for j in range(3):
            qc = qc + g[i + 1][j + 1] * K[i] * K[j]
    root = torch.sqrt(qb * qb - 4.0 * qa * qc)
    k0 = (-qb + root) / (2.0 * qa)
    k0 = torch.where(k0 > 0.0, k0, (-qb - root) / (2.0 * qa))
    low = _lower(g, [k0] + K)
    return torch.stack([torch.zeros_like(x), x, y, z, *low[1:]]), low[0], img, u, v


def _trace(p, grid, specs, dev, back=0.0, mult=None):
    """The step loop on every ray of `specs`; with `mult`, the transfer updates of each step are kept for the gradient."""
    cam = _camera(specs, dev, back)
    fluid = _Fluid(grid, p, dev)
    s, pt, img, u, v = _rays(p, specs, cam, dev, back)
    n = pt.numel()
    c = cam[img].T
    full = lambda value: torch.full((n,), float(value), dtype=torch.float64, device=dev)  # noqa: E731
    ph = dict(s=s, pt=pt, img=img, u=u, v=v, I=full(0.0), dl=full(p.initial_step * (back or p.camera_distance)),
              freq=c[12].clone() if back else full(0.0), emit=-pt.clone() if back else full(1.0),
              phase=torch.full((n,), 2 if back else 1, dtype=torch.uint8, device=dev),
              term=torch.zeros(n, dtype=torch.bool, device=dev))
    tape = []
    for step in range(p.max_steps):
        at = torch.nonzero(~ph["term"])[:, 0]
        if at.numel() == 0:
            break
        st = ph["s"][:, at]
        r = _radius(st[1], st[2], st[3], p.spin)
        sunk, gone = r <= p.r_term_min, r > p.r_term_max
        ph["I"][at[sunk]] = 0.0
        ph["phase"][at[sunk | gone]] = 4
        ph["term"][at[sunk | gone]] = True
        at = at[~(sunk | gone)]
        st, dl = ph["s"][:, at], ph["dl"][at]
        if p.integrator == abi.RK4:
            new, taken, nxt, ok = _rk4(st, ph["pt"][at], dl, p.spin, p.mass), dl, dl, torch.ones_like(dl, dtype=torch.bool)
        else:
            new, taken, nxt, ok = _rk45(st, ph["pt"][at], dl, p)
        ph["dl"][at] = nxt
        ph["term"][at[~ok]] = True
        at, new, taken = at[ok], new[:, ok], taken[ok]
        ph["s"][:, at] = new
        before = ph["phase"][at]
        cell, e0 = fluid.sample(new)
        # first contact of a backward ray: its packet, and the way back
        g = (before == 1) & (cell >= 0)
        if bool(g.any()):
            w, where = at[g], cell[g]
            packets = (fluid.rho[where] / p.density_g_cm3_per_code * p.superphoton_count_normalization).to(torch.int64)
            made = packets > 0
            low = [ph["pt"][w], new[4][g], new[5][g], new[6][g]]
            ph["emit"][w] = torch.where(made, -sum(a * b[g] for a, b in zip(low, e0)), ph["emit"][w])
            ph["freq"][w] = torch.where(made, c[12][w], ph["freq"][w])
            ph["I"][w] = torch.where(made, p.energy_per_cell_erg / packets.clamp(min=1).double(), 0.0)
            ph["dl"][w] = torch.where(made, -ph["dl"][w].abs(), ph["dl"][w])
            ph["phase"][w] = torch.where(made, 2, 4).to(torch.uint8)
            ph["term"][w] |= ~made
        # transfer through a cell
        g = (before != 1) & (cell >= 0)
        if bool(g.any()):
            w, where, length = at[g], cell[g], taken[g].abs()
            tau = torch.clamp(c[13][w] * fluid.rho[where] * length, min=0.0)
            emission = torch.clamp(c[14][w] * fluid.rho[where] * fluid.T[where] * length, min=0.0)
            I = ph["I"][w]
            att = torch.exp(-(tau if mult is None else mult[0][where] * tau))
            if mult is not None:
                tape.append((w, where, tau, emission, I, att))
            ph["I"][w] = I * att + (emission if mult is None else mult[1][where] * emission)
        # the camera plane
        g = before == 2
        w, (t, x, y, z) = at[g], (new[q][g] for q in range(4))
        k = c[:, w]
        across = x * k[0] + y * k[1] + z * k[2] >= k[9]
        rel = [x - k[9] * k[0], y - k[9] * k[1], z - k[9] * k[2]]
        uu, vv = (sum(rel[q] * k[base + q] for q in range(3)) for base in (3, 6))
        inside = across & (uu.abs() <= 0.5 * k[10]) & (vv.abs() <= 0.5 * k[11])
        _, m = _metric(x, y, z, _radius(x, y, z, p.spin), p.spin, p.mass)
        seen, emitted = -ph["pt"][w] * (1.0 / torch.sqrt(-m[0][0])), ph["emit"][w]
        good = (m[0][0] < 0.0) & (seen > 0.0) & (emitted > 0.0)
        ph["freq"][w] = torch.where(inside & good, ph["freq"][w] * (seen / emitted), ph["freq"][w])
        ph["I"][w] = torch.where((inside & ~good) | (across & ~inside), 0.0, ph["I"][w])
        ph["u"][w] = torch.where(inside, uu, ph["u"][w])
        ph["v"][w] = torch.where(inside, vv, ph["v"][w])
        ph["phase"][w] = torch.where(inside, 3, torch.where(across, 4, ph["phase"][w])).to(torch.uint8)
        ph["term"][w] |= across
        if (step % p.output_interval == 0 or step == p.max_steps - 1) and float(ph["term"].double().mean()) >= p.termination_percent:
            break
    return ph, tape


def _bin(x, lo, hi, bins):
    return (((x - lo) / (hi - lo)).clamp(0.0, 1.0) * (bins - 1)).to(torch.int64)


def _products(p, spec, ph, q, nx, ny):
    m = (ph["phase"] == 3) & (ph["img"] == q)
    I, f = ph["I"][m], ph["freq"][m]
    pix = _bin(ph["v"][m], -0.5 * spec.camera_height, 0.5 * spec.camera_height, ny) * nx
    pix = pix + _bin(ph["u"][m], -0.5 * spec.camera_width, 0.5 * spec.camera_width, nx)
    image = torch.zeros(nx * ny, dtype=torch.float64, device=I.device).index_add_(0, pix, I).view(ny, nx)
    bins, lo, hi = int(p.spectrum_bins), math.log10(p.spectrum_min_hz), math.log10(p.spectrum_max_hz)
    inside = (f >= p.spectrum_min_hz) & (f <= p.spectrum_max_hz)
    spectrum = torch.zeros(bins, dtype=torch.float64, device=I.device)
    spectrum.index_add_(0, _bin(torch.log10(f[inside]), lo, hi, bins), I[inside])
    return image, spectrum


def exact(case, seed):
    rng = np.random.default_rng([int(seed), 20])
    p, grid = _params(case, rng), _torus(case, rng)
    kind = case["kind"]
    # scattering, random screens and the drawn spectra follow the framework's own random streams
    if kind == "disk" or case.get("random_screen") or case.get("generator", "custom") != "custom":
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    none = dict.fromkeys(("steps_done", "n_terminated", "accepted_steps", "photon_calls"))
    if kind in ("batch", "stream"):
        specs = _specs(case, p)
    else:
        specs = [abi.ImageSpec.from_params(p, case["nx"], case["ny"])]
    if kind == "adjoint":
        shape = grid["r.npy"].shape
        mult = [torch.from_numpy(np.exp(rng.normal(0.0, 0.1, shape))).to(dev).reshape(-1) for _ in range(2)]
        weights = torch.from_numpy(rng.normal(0.0, 1.0, (case["ny"], case["nx"]))).to(dev)
        ph, tape = _trace(p, grid, specs, dev, back=workloads.C4_BACK_DISTANCE, mult=mult)
        image, _ = _products(p, specs[0], ph, 0, case["nx"], case["ny"])
        px = _bin(ph["u"], -0.5 * p.camera_width, 0.5 * p.camera_width, case["nx"])
        py = _bin(ph["v"], -0.5 * p.camera_height, 0.5 * p.camera_height, case["ny"])
        lam = torch.where(ph["phase"] == 3, weights[py, px], 0.0)
        g_abs, g_emis = torch.zeros_like(mult[0]), torch.zeros_like(mult[1])
        for w, cell, tau, emission, I, att in reversed(tape):
            g_emis.index_add_(0, cell, lam[w] * emission)
            g_abs.index_add_(0, cell, -lam[w] * I * att * tau)
            lam[w] = lam[w] * att
        return dict(image=image, g_abs=g_abs.view(shape), g_emis=g_emis.view(shape))
    ph, _ = _trace(p, grid, specs, dev)
    if kind == "inplace":
        s = ph["s"]
        fields = dict(x0=s[0], x1=s[1], x2=s[2], x3=s[3], k0=ph["pt"], k1=s[4], k2=s[5], k3=s[6], frequency=ph["freq"],
                      emission_frame_energy=ph["emit"], I=ph["I"], dlambda=ph["dl"], theta_disp=ph["u"], phi_disp=ph["v"])
        return dict(fields, id=None, Q=None, U=None, V=None, terminate=None, phase=None, **none)
    got = [_products(p, sp, ph, q, int(sp.nx), int(sp.ny)) for q, sp in enumerate(specs)]
    if kind == "batch":
        images = torch.cat([torch.cat([im.reshape(-1), im.new_zeros(3 * im.numel())]) for im, _ in got])
        return dict(images=images, spectra=torch.cat([sp for _, sp in got]), arrived=None, **none)
    lo, hi = math.log10(p.spectrum_min_hz), math.log10(p.spectrum_max_hz)
    nu = 10.0 ** np.linspace(lo, hi, int(p.spectrum_bins))
    outs = [dict(image_I=im, image_Q=torch.zeros_like(im), image_U=torch.zeros_like(im), image_V=torch.zeros_like(im),
                 spectrum_frequency_hz=nu, spectrum_I=sp, arrived_count=None) for im, sp in got]
    if kind == "frame":
        return dict(outs[0], **none)
    return [dict(none, images=outs) for _ in range(2)]
