"""Performance cases of the n-body library: what its users have it compute, through
its public Python entry points (nbody_gb300).

A case is one call, or the few calls that belong together in a user's loop.  Kinds:

  step        advance() by a few iterations, then export_device(): the inner loop of a
              simulation whose positions stay on the GPU (a renderer, an analysis)
  frame       DiskGalaxySimulator.stepSim(): the reference's per-frame call, its
              iterations and then the whole state back in host arrays
  ensemble    many independent systems advanced by one captured graph per pass
  adjoint     a T-step forward run and the gradients of its initial state
  diagnostics FP64 energy and momenta, the conservation check of a long run
  render      one headless frame into a device image
  noalloc     accelerations on the caller's own device buffers

Inputs are drawn here with torch from the seed alone, so that exact() can start from
the same numbers without the library.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "cuda-to-sycl-nbody_gb300"))
import nbody_gb300 as nb  # noqa: E402

ACCUMULATOR = {"compensated": nb.ACC_COMPENSATED, "plain": nb.ACC_PLAIN,
               "reference_order": nb.ACC_REFERENCE_ORDER}
FRAME = {"G": 2.0, "dt": 1e-3, "damping": 0.999, "distEps": 1e-3}
CAMERA = (0.6, 0.5, 12.0)  # azimuth, elevation, distance of the rendered view


def listed():
    return [
        # A small system stepped once per call: launches and latency are what count.
        {"name": "step_2k", "kind": "step", "ic": "disk", "n": 2048, "iters": 1,
         "accumulator": "compensated", "masses": "equal", "eps": 1e-3, "dt": 1e-3},
        # The reference's own performance run (arguments 50 5 0.999 0.001 1.0e-3 2.0):
        # 12,800 unit masses, 5 iterations a frame, the state back on the host each frame.
        {"name": "frame_12800", "kind": "frame", "n": 12800, "iters": 5},
        # The CPU-runnable thin disk, ten steps between outputs.
        {"name": "disk_25600", "kind": "step", "ic": "disk", "n": 25600, "iters": 10,
         "accumulator": "compensated", "masses": "equal", "eps": 1e-3, "dt": 1e-3},
        # A ragged star cluster with a mass function, plain accumulator.
        {"name": "cluster_100003", "kind": "step", "ic": "plummer", "n": 100003, "iters": 1,
         "accumulator": "plain", "masses": "own", "eps": 1e-4, "dt": 1e-4},
        # The two-disk collision of the precision study.
        {"name": "collision_262k", "kind": "step", "ic": "two_disks", "n": 262144, "iters": 1,
         "accumulator": "compensated", "masses": "equal", "eps": 1e-3, "dt": 1e-3},
        # The headline workload: one step of the million-body Plummer sphere.
        {"name": "plummer_1m", "kind": "step", "ic": "plummer", "n": 1048576, "iters": 1,
         "accumulator": "compensated", "masses": "equal", "eps": 1e-4, "dt": 1e-4},
        # Drop-in bit-exact replacement of the reference's kernel at its default size.
        {"name": "reference_order_12800", "kind": "step", "ic": "disk", "n": 12800, "iters": 4,
         "accumulator": "reference_order", "masses": "equal", "eps": 1e-3, "dt": 1e-3},
        # 4,096 systems of 64 to 8,192 bodies, a captured graph of two steps per output.
        {"name": "ensemble_4096", "kind": "ensemble", "systems": 4096, "lo": 64, "hi": 8192,
         "size_seed": 20261203, "iters": 2, "eps": 1e-3, "dt": 1e-3},
        # Fitting initial conditions by gradient: a 32-step run and its adjoint.
        {"name": "adjoint_16k", "kind": "adjoint", "n": 16384, "T": 32, "every": 8,
         "eps": 1e-3, "dt": 1e-3},
        # The conservation check of a long run.
        {"name": "diagnostics_65k", "kind": "diagnostics", "ic": "two_disks", "n": 65536,
         "eps": 1e-3},
        # One full-HD frame of the million-body sphere.
        {"name": "render_1080p", "kind": "render", "n": 1048576, "width": 1920, "height": 1080},
        # An engine that owns its GPU memory asks for the accelerations of its bodies.
        {"name": "noalloc_20000", "kind": "noalloc", "ic": "disk", "n": 20000,
         "masses": "own", "eps": 1e-3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "frame", "reference_order", "ensemble", "adjoint",
                       "diagnostics", "render", "noalloc"])
    if kind == "step":
        n = _log_int(rng, 64, 1048576)
        ic = rng.choice(["disk", "plummer", "two_disks"])
        return {"kind": "step", "ic": ic, "n": n - n % 2 if ic == "two_disks" else n,
                "iters": 1 if n > 60000 else rng.choice([1, 4, 10]),
                "accumulator": rng.choice(["compensated", "compensated", "plain"]),
                "masses": rng.choice(["equal", "equal", "own"]),
                "eps": rng.choice([1e-3, 1e-4]), "dt": 1e-4}
    if kind == "frame":
        return {"kind": "frame", "n": 256 * rng.randint(1, 160), "iters": rng.choice([1, 5])}
    if kind == "reference_order":
        n = _log_int(rng, 256, 262144)
        return {"kind": "step", "ic": "disk", "n": n, "iters": 1 if n > 60000 else 4,
                "accumulator": "reference_order", "masses": "equal", "eps": 1e-3, "dt": 1e-3}
    if kind == "ensemble":
        return {"kind": "ensemble", "systems": _log_int(rng, 16, 4096), "lo": 64,
                "hi": _log_int(rng, 256, 8192), "size_seed": rng.randrange(1 << 30), "iters": 2,
                "eps": 1e-3, "dt": 1e-3}
    if kind == "adjoint":
        return {"kind": "adjoint", "n": _log_int(rng, 512, 16384), "T": rng.choice([8, 16, 32]),
                "every": rng.choice([4, 8]), "eps": 1e-3, "dt": 1e-3}
    if kind == "diagnostics":
        return {"kind": "diagnostics", "ic": rng.choice(["disk", "plummer"]),
                "n": _log_int(rng, 1000, 65536), "eps": 1e-3}
    if kind == "render":
        w = rng.randint(320, 1920)
        return {"kind": "render", "n": _log_int(rng, 1000, 1048576), "width": w,
                "height": w * 9 // 16}
    return {"kind": "noalloc", "ic": rng.choice(["disk", "plummer"]),
            "n": _log_int(rng, 64, 262144), "masses": "own", "eps": 1e-3}


# ------------------------------------------------------------------------- inputs
def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=gen.device, dtype=torch.float64)


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=gen.device, dtype=torch.float64)


def _disk(gen, n, eps):
    """Thin disk of total mass 1: r = sqrt(u), z ~ N(0, 0.01^2), near-circular speeds."""
    r, th = _rand(gen, n).sqrt(), 2 * math.pi * _rand(gen, n)
    vt = r * r / (r * r + eps) ** 0.75
    x = torch.stack((r * th.cos(), r * th.sin(), 0.01 * _randn(gen, n)))
    v = torch.stack((-vt * th.sin(), vt * th.cos(), torch.zeros_like(r))) + 0.01 * _randn(gen, 3, n)
    return x, v


def _direction(gen, n):
    c, ph = 1 - 2 * _rand(gen, n), 2 * math.pi * _rand(gen, n)
    s = (1 - c * c).sqrt()
    return torch.stack((s * ph.cos(), s * ph.sin(), c))


def _plummer(gen, n):
    """Plummer sphere of scale radius 1 and total mass 1 in equilibrium: the speed in
    units of the escape speed squared is Beta(3/2, 9/2) distributed."""
    r = ((0.999 * _rand(gen, n).clamp_min(1e-12)) ** (-2 / 3) - 1).rsqrt()
    a, b = _randn(gen, 3, n).square().sum(0), _randn(gen, 9, n).square().sum(0)
    speed = (2 * a / (a + b)).sqrt() * (1 + r * r) ** -0.25
    return r * _direction(gen, n), speed * _direction(gen, n)


def _bodies(case, seed):
    """(positions [3, n], velocities [3, n], masses [n]) in float64, on float32 values."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    ic, n = case.get("ic", "plummer"), case["n"]
    if ic == "disk":
        x, v = _disk(gen, n, case["eps"])
    elif ic == "two_disks":
        x, v = _disk(gen, n // 2, case["eps"])
        y, w = _disk(gen, n // 2, case["eps"])
        c, s = math.cos(math.pi / 6), math.sin(math.pi / 6)
        tilt = torch.tensor([[1, 0, 0], [0, c, -s], [0, s, c]], dtype=x.dtype, device=x.device)
        y, w = tilt @ y, tilt @ w
        x[0] -= 2
        v[0] += 0.3
        y[0] += 2
        w[0] -= 0.3
        x, v = torch.cat((x, y), 1), torch.cat((v, w), 1)
    else:
        x, v = _plummer(gen, n)
    m = torch.full((n,), (2.0 if ic == "two_disks" else 1.0) / n, dtype=x.dtype, device=x.device)
    if case.get("masses") == "own":
        m = m * (0.5 + _rand(gen, n))
    return tuple(t.float().double() for t in (x, v, m))


def _frame_bodies(case, seed):
    """A disk like the reference's: unit masses, radius up to 100, thickness 4."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n = case["n"]
    th, r = 2 * math.pi * _rand(gen, n), 0.01 + 100 * _rand(gen, n)
    speed = (2 * r).sqrt()
    x = torch.stack((r * th.cos(), r * th.sin(), 4 * _rand(gen, n)))
    v = torch.stack((-speed * th.sin(), speed * th.cos(), torch.zeros_like(r)))
    return x.float().double(), v.float().double()


def _sizes(case):
    rng = np.random.default_rng(case["size_seed"])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["systems"]))
    return sizes.astype(np.uint32)


def _ensemble_bodies(case, seed):
    """(sizes, positions, velocities, masses): Plummer spheres of log-uniform sizes."""
    sizes = _sizes(case)
    x, v, _ = _bodies({"ic": "plummer", "n": int(sizes.sum())}, seed)
    m = torch.from_numpy(np.repeat(1.0 / sizes, sizes)).to(x.device).float().double()
    return sizes, x, v, m


def _cotangents(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed) + 1)
    return _randn(gen, case["n"], 3).float(), _randn(gen, case["n"], 3).float()


def _host(t):
    return [row.float().cpu().numpy() for row in t]


def _buffers(n, count=2):
    return [torch.empty((n, 4), dtype=torch.float32, device="cuda") for _ in range(count)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        x, v = _frame_bodies(case, seed)
        p = nb.SimParam(numParticles=case["n"], simIterationsPerFrame=case["iters"], **FRAME)
        return {"case": case, "galaxy": nb.DiskGalaxySimulator(p, _host(x), _host(v))}
    if kind == "noalloc":
        x, _, m = _bodies(case, seed)
        xyzm = torch.cat((x, m[None])).t().float().contiguous()
        return {"case": case, "xyzm": xyzm, "out": _buffers(case["n"], 1)[0]}
    p = nb.SimParam(G=1.0, dt=case.get("dt", 1e-3), damping=0.999, distEps=case.get("eps", 1e-4),
                    numParticles=case.get("n", 1),
                    accumulator=ACCUMULATOR[case.get("accumulator", "compensated")])
    if kind == "ensemble":
        sizes, x, v, m = _ensemble_bodies(case, seed)
        sim = nb.Simulation(p, _host(x), _host(v), m.float().cpu().numpy(), sizes=sizes)
        stream = torch.cuda.Stream()  # graphs are captured on a stream of their own
        sim.set_stream(stream.cuda_stream)
        sim.graph_capture(case["iters"])
        return {"case": case, "sim": sim, "stream": stream, "out": _buffers(sim.n)}
    x, v, m = _bodies(case, seed)
    sim = nb.Simulation(p, _host(x), _host(v), m.float().cpu().numpy())
    sim.set_stream(torch.cuda.current_stream().cuda_stream)
    state = {"case": case, "sim": sim}
    if kind == "step":
        state["out"] = _buffers(case["n"])
    elif kind == "adjoint":
        state["gT"] = _cotangents(case, seed)
        state["g0"] = [torch.empty((case["n"], 3), dtype=torch.float32, device="cuda")
                       for _ in range(2)]
        state["out"] = _buffers(case["n"])
    elif kind == "render":
        w, h = case["width"], case["height"]
        state["camera"] = nb.camera_matrices(*CAMERA, w, h)
        state["image"] = torch.empty((h, w, 4), dtype=torch.float32, device="cuda")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim, (pos, vel) = state["sim"], state["out"]
        sim.advance(case["iters"])
        sim.export_device(pos.data_ptr(), vel.data_ptr())
        return {"pos": pos, "vel": vel}
    if kind == "frame":
        galaxy = state["galaxy"]
        galaxy.stepSim()
        return {"pos": galaxy.getParticlePos(), "vel": galaxy.getParticleVel()}
    if kind == "ensemble":
        sim, stream, (pos, vel) = state["sim"], state["stream"], state["out"]
        stream.wait_stream(torch.cuda.current_stream())
        sim.graph_launch()
        sim.export_device(pos.data_ptr(), vel.data_ptr())
        torch.cuda.current_stream().wait_stream(stream)
        return {"pos": pos, "vel": vel}
    if kind == "adjoint":
        sim, (gx, gv), (gx0, gv0), (pos, vel) = (state[k] for k in ("sim", "gT", "g0", "out"))
        sim.adjoint_forward(case["T"], case["every"])
        sim.adjoint_backward_device(gx.data_ptr(), gv.data_ptr(), gx0.data_ptr(), gv0.data_ptr())
        sim.export_device(pos.data_ptr(), vel.data_ptr())
        return {"gx": gx0, "gv": gv0, "pos": pos, "vel": vel}
    if kind == "diagnostics":
        return {k: np.asarray(d) for k, d in state["sim"].diagnostics().items()}
    if kind == "render":
        view, proj = state["camera"]
        state["sim"].render(view, proj, case["width"], case["height"], state["image"].data_ptr())
        return state["image"]
    nb.accelerations_noalloc(state["xyzm"].data_ptr(), case["n"], 1.0, case["eps"],
                             state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return state["out"]


def _pairs(case):
    """Unordered pairs of one force evaluation."""
    if case["kind"] == "ensemble":
        sizes = _sizes(case).astype(np.float64)
        return float((sizes * (sizes - 1)).sum()) / 2
    return case["n"] * (case["n"] - 1) / 2


def work(case):
    """Each pair counted once: 24 flop give the force on both particles (difference 3,
    softened square 6, cube 2, root 1, both sums 12), 40 the adjoint's two products, 12
    the potential.  State: position and velocity, 32 bytes, in and out."""
    kind = case["kind"]
    pairs = 0 if kind == "render" else _pairs(case)
    if kind == "ensemble":
        n = int(_sizes(case).sum())
        return {"bytes": 64 * n, "flops": 24 * pairs * case["iters"]}
    n = case["n"]
    if kind in ("step", "frame"):
        return {"bytes": 64 * n, "flops": 24 * pairs * case["iters"]}
    if kind == "adjoint":
        return {"bytes": (64 + 48) * n, "flops": (24 + 40) * pairs * case["T"]}
    if kind == "diagnostics":
        return {"bytes": 32 * n + 80, "flops": 12 * pairs}
    if kind == "render":  # about 8 x 8 pixels under a sprite, 3 channels
        return {"bytes": 32 * n + 16 * case["width"] * case["height"], "flops": 64 * 6 * n}
    return {"bytes": 32 * n, "flops": 24 * pairs}


# -------------------------------------------------------------------- 64-bit results
def _blocks(n):
    rows = max(1, (1 << 25) // n)
    return [(i, min(n, i + rows)) for i in range(0, n, rows)]


def _accel64(x, m, eps):
    a = torch.empty_like(x)
    for lo, hi in _blocks(x.shape[1]):
        d = [x[c][None, :] - x[c, lo:hi, None] for c in range(3)]
        inv = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps).rsqrt()
        s = inv * inv * inv * m
        for c in range(3):
            a[c, lo:hi] = (s * d[c]).sum(1)
    return a


def _steps64(x, v, m, G, dt, damping, eps, steps):
    x, v = x.clone(), v.clone()
    for _ in range(steps):
        v = damping * v + dt * G * _accel64(x, m, eps)
        x = x + dt * v
    return x, v


def _vjp64(x, mu, m, eps):
    """sum_j K_ij (m_i mu_j - m_j mu_i), K = s I - 3 s r r^T / (r^2 + eps)."""
    g = torch.empty_like(x)
    for lo, hi in _blocks(x.shape[1]):
        d = [x[c][None, :] - x[c, lo:hi, None] for c in range(3)]
        u = [m[lo:hi, None] * mu[c][None, :] - m[None, :] * mu[c, lo:hi, None] for c in range(3)]
        inv = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps).rsqrt()
        inv2 = inv * inv
        s = inv2 * inv
        q = -3 * inv2 * (d[0] * u[0] + d[1] * u[1] + d[2] * u[2])
        for c in range(3):
            g[c, lo:hi] = (s * (u[c] + q * d[c])).sum(1)
    return g


def _f32(v):
    return float(np.float32(v))


def _rows4(x, w):
    """[n, 4] rows as export_device writes them: x, y, z and a last column."""
    last = w if torch.is_tensor(w) else torch.full_like(x[0], w)
    return torch.cat((x, last[None])).t().contiguous()


def _sample(img, s, t):
    """Bilinear fetch of img [h, w, c] at normalised coordinates, clamped to the edge."""
    h, w = img.shape[:2]
    u, v = s * w - 0.5, t * h - 0.5
    fu, fv = u.floor(), v.floor()
    a, b = (u - fu)[None, :, None], (v - fv)[:, None, None]
    x0, y0 = fu.long(), fv.long()
    ix = [(x0 + k).clamp(0, w - 1) for k in (0, 1)]
    iy = [(y0 + k).clamp(0, h - 1) for k in (0, 1)]
    top = img[iy[0]][:, ix[0]] * (1 - a) + img[iy[0]][:, ix[1]] * a
    bottom = img[iy[1]][:, ix[0]] * (1 - a) + img[iy[1]][:, ix[1]] * a
    return top * (1 - b) + bottom * b


def _camera64(width, height):
    az, el, dist = (_f32(c) for c in CAMERA)
    eye = np.array([math.cos(az) * math.cos(el), math.sin(az) * math.cos(el), math.sin(el)]) * dist
    f = -eye / np.linalg.norm(eye)
    side = np.cross(f, [0, 0, 1])
    side /= np.linalg.norm(side)
    up = np.cross(side, f)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = side, up, -f
    view[:3, 3] = -view[:3, :3] @ eye
    proj = np.zeros((4, 4))
    proj[1, 1] = 1 / math.tan(math.radians(15))
    proj[0, 0] = proj[1, 1] * height / width
    proj[2, 2] = proj[3, 2] = -1
    proj[2, 3] = -2
    return proj @ view


def _render64(x, v, width, height):
    """Flare sprites, half-resolution Gaussian bloom, exposure and gamma, all in float64."""
    dev, margin, nf = x.device, 50, 16
    bw, bh = width + 2 * margin, height + 2 * margin
    pv = torch.from_numpy(_camera64(width, height)).to(dev)
    clip = pv[:, :3] @ x + pv[:, 3:]
    keep = (clip[3] > 0) & (clip[2] >= -clip[3]) & (clip[2] <= clip[3])
    clip, v = clip[:, keep], v[:, keep]
    t = ((v * v).sum(0) + 1).mul(0.0006).clamp(0, 1)
    colour = torch.stack((t, 0.4 * (1 - t) + 0.2 * t, torch.ones_like(t)), 1)
    i = torch.arange(nf, dtype=torch.float64, device=dev) - nf // 2
    flare = torch.exp(-(i[:, None] ** 2 + i[None, :] ** 2) / nf) ** 2.2
    lo, first, span = [], [], []
    for c, (half, size) in enumerate(((nf / (2 * width), bw), (nf / (2 * height), bh))):
        ndc = clip[c] / clip[3]
        lo.append(ndc - half)
        first.append(((ndc - half + 1) * 0.5 * size - 0.5).ceil().long())
        span.append((((ndc + half + 1) * 0.5 * size - 0.5).ceil().long() - first[c], 2 * half, size))
    hdr = torch.zeros((bh * bw, 3), dtype=torch.float64, device=dev)

    def axis(c, k):  # pixel, whether it is covered, texel and weight along one axis
        px = first[c] + k
        count, width_ndc, size = span[c]
        inside = (k < count) & (px >= 0) & (px < size)
        u = (((px + 0.5) / size * 2 - 1) - lo[c]) / width_ndc * nf - 0.5
        return px, inside, u.floor().long(), u - u.floor()

    for ky in range(int(span[1][0].max())):
        py, in_y, ty, b = axis(1, ky)
        for kx in range(int(span[0][0].max())):
            px, in_x, tx, a = axis(0, kx)
            m = in_y & in_x
            x0, x1, y0, y1 = tx % nf, (tx + 1) % nf, ty % nf, (ty + 1) % nf
            alpha = (flare[y0, x0] * (1 - a) * (1 - b) + flare[y0, x1] * a * (1 - b)
                     + flare[y1, x0] * (1 - a) * b + flare[y1, x1] * a * b)
            hdr.index_add_(0, (py * bw + px)[m], (colour * alpha[:, None])[m])
    hdr = hdr.view(bh, bw, 3)
    w = np.exp(-np.arange(25) ** 2 / 200.0)
    w /= 2 * w[1:].sum() + w[0]
    taps = [(0.0, w[0])]
    for k in range(1, 25, 2):  # pairs of neighbouring taps as one bilinear sample
        pair = w[k] + w[k + 1]
        taps.append(((k * w[k] + (k + 1) * w[k + 1]) / pair, pair))
    ow, oh = bw // 2, bh // 2
    s = (torch.arange(ow, dtype=torch.float64, device=dev) + 0.5) / ow
    q = (torch.arange(oh, dtype=torch.float64, device=dev) + 0.5) / oh
    across = _sample(hdr, s, q) * taps[0][1]
    for off, wt in taps[1:]:
        across += wt * (_sample(hdr, s + off * 2 / width, q) + _sample(hdr, s - off * 2 / width, q))
    bloom = _sample(across, s, q) * taps[0][1]
    for off, wt in taps[1:]:
        bloom += wt * (_sample(across, s, q + off * 2 / height)
                       + _sample(across, s, q - off * 2 / height))
    ls = (2 * torch.arange(bw // 2, dtype=torch.float64, device=dev) + 1.5) / bw
    lt = (2 * torch.arange(bh // 2, dtype=torch.float64, device=dev) + 1.5) / bh
    lum = (_sample(hdr, ls, lt) * torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64,
                                               device=dev)).sum(2).mean()
    exposure = 1 / (10 * lum).clamp(0.2, 1000)
    ts = torch.arange(margin, margin + width, dtype=torch.float64, device=dev) / bw
    tt = torch.arange(margin, margin + height, dtype=torch.float64, device=dev) / bh
    light = hdr[margin:margin + height, margin:margin + width] + _sample(bloom, ts, tt)
    rgb = (1 - torch.exp(-light * exposure)) ** (1 / 2.2)
    return torch.cat((rgb, torch.ones_like(rgb[..., :1])), 2)


def exact(case, seed):
    kind = case["kind"]
    steps = case.get("iters", 1) + 4 * case.get("T", 0)
    if kind != "render" and 2 * _pairs(case) * steps > 1.2e11:
        return None  # over about 20 seconds in float64
    eps = _f32(case.get("eps", 1e-4))
    if kind == "frame":
        x, v = _frame_bodies(case, seed)
        x, v = _steps64(x, v, torch.ones_like(x[0]), *(_f32(FRAME[k]) for k in
                        ("G", "dt", "damping", "distEps")), case["iters"])
        return {"pos": list(x), "vel": list(v)}
    dt, damping = _f32(case.get("dt", 1e-3)), _f32(0.999)
    if kind == "ensemble":
        sizes, x, v, m = _ensemble_bodies(case, seed)
        out, lo = [], 0
        for n in sizes.tolist():
            sl = slice(lo, lo + n)
            out.append(_steps64(x[:, sl], v[:, sl], m[sl], 1.0, dt, damping, eps, case["iters"]))
            lo += n
        x, v = (torch.cat([o[k] for o in out], 1) for k in (0, 1))
        return {"pos": _rows4(x, m), "vel": _rows4(v, 0.0)}
    x, v, m = _bodies(case, seed)
    if kind == "step":
        x, v = _steps64(x, v, m, 1.0, dt, damping, eps, case["iters"])
        return {"pos": _rows4(x, m), "vel": _rows4(v, 0.0)}
    if kind == "noalloc":
        return _rows4(_accel64(x, m, eps), 0.0)
    if kind == "render":
        return _render64(x, v, case["width"], case["height"])
    if kind == "diagnostics":
        pot = 0.0
        for lo, hi in _blocks(x.shape[1]):
            d2 = sum((x[c][None, :] - x[c, lo:hi, None]).square() for c in range(3)) + eps
            pot += float((m[lo:hi, None] * m * d2.rsqrt()).sum())
        pot = -0.5 * (pot - float((m * m).sum()) / math.sqrt(eps))
        kin = float((0.5 * m * v.square().sum(0)).sum())
        return {"kinetic": np.asarray(kin), "potential": np.asarray(pot),
                "total": np.asarray(kin + pot), "momentum": (m * v).sum(1),
                "angular_momentum": (m * torch.linalg.cross(x, v, dim=0)).sum(1),
                "mass": m.sum()}
    path = [x]  # adjoint: positions of every step, then the sweep back
    for _ in range(case["T"]):
        x, v = _steps64(x, v, m, 1.0, dt, damping, eps, 1)
        path.append(x)
    gx, gv = (g.double().t().contiguous() for g in _cotangents(case, seed))
    for t in range(case["T"] - 1, -1, -1):
        mu = gv + dt * gx
        gx, gv = gx + dt * _vjp64(path[t], mu, m, eps), damping * mu
    return {"gx": gx.t().contiguous(), "gv": gv.t().contiguous(), "pos": _rows4(x, m),
            "vel": _rows4(v, 0.0)}
