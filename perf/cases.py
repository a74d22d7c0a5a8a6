"""Performance cases: the work that programs have this engine do.

A case is a dict of plain values.  `prepare` builds what a program keeps (a
lattice, a batch, a network, device buffers), `run` makes one pass through the
public entry points, `work` says what a pass cannot do without and `exact`
gives the outputs in 64-bit arithmetic from torch alone.

Kinds of case:
  step     channel lattice: n steps, then rho, jx, jy into device arrays
           (averaging loops, the benchmark, the large-grid runs)
  frame    reference-edge lattice: n steps, then one frame into a device
           buffer and the same three fields (the redraw loop)
  edit     reference-edge lattice: a barrier stroke drawn, n steps, the curl
           summary and an RGBA frame in host memory (the interactive page)
  observe  n steps, then force, conservation sums and fields (drag, lift and
           Strouhal runs; f64 is the precision reference)
  batch    many channel domains of uneven size: n steps, the density of every
           domain and the conservation sums (parameter sweeps)
  closure  network inference on the lattice, then n steps with its records
           (the coarse runs; n is the refresh interval)
  train    forward, loss, backward and Adam of the closure network
  sample   n fine steps, populations to the device, one coarse training sample
"""
import ctypes
import math

import numpy as np
import torch

import lbm_gb300 as L
from lbm_gb300 import batch as B
from lbm_gb300 import closure as C

STORAGE = {"f32": L.F32, "f16": L.F16, "bf16": L.BF16, "f64": L.F64}
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}
FLOPS = 130  # of one cell's moments and relaxation
LAYERS = ((4, 32), (32, 32), (32, 32), (32, 1))


def listed():
    return [
        # the reference's page at its smallest preset: a few steps per redraw
        dict(name="frame_256x128", kind="frame", nx=256, ny=128, n=4, width=512, height=256),
        # the page while a barrier is being drawn, at a ragged window size
        dict(name="edit_1100x700", kind="edit", nx=1100, ny=700, n=20, points=300),
        # the closure's coarse grid without the closure: 20-step calls
        dict(name="step_f32_512x256", kind="step", nx=512, ny=256, n=20, storage="f32", sr=False, inlet=False),
        # the benchmark's channel in f32 and in 16-bit storage
        dict(name="step_f32_4096x2048", kind="step", nx=4096, ny=2048, n=50, storage="f32", sr=False, inlet=False),
        dict(name="step_f16_4096x2048", kind="step", nx=4096, ny=2048, n=50, storage="f16", sr=False, inlet=False),
        # an odd size with every 16-bit option on, an odd number of steps
        dict(name="step_bf16_sr_1531x769", kind="step", nx=1531, ny=769, n=31, storage="bf16", sr=True, inlet=True),
        # a large grid
        dict(name="step_f32_8192x4096", kind="step", nx=8192, ny=4096, n=20, storage="f32", sr=False, inlet=False),
        # the precision study's f64 lattice with its observables
        dict(name="observe_f64_1024x512", kind="observe", nx=1024, ny=512, n=25, storage="f64"),
        # a sweep of uneven domains, autotuned as the benchmark does
        dict(name="batch_f32_16", kind="batch", count=16, n=100, storage="f32", sr=False),
        # a coarse closure run: inference every 20 steps
        dict(name="closure_f32_512x256", kind="closure", nx=512, ny=256, n=20, storage="f32"),
        # a training step of the closure network on four coarse snapshots
        dict(name="train_4x256x512", kind="train", n=4, h=256, w=512),
        # one training sample of a fine run, every 20 fine steps
        dict(name="sample_2048x1024", kind="sample", nx=2048, ny=1024, n=20, factor=4),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["frame", "edit", "observe", "batch", "closure", "train", "sample"])
    if kind == "step":
        storage = rng.choice(["f32", "f32", "f16", "bf16"])
        nx, ny = _logint(rng, 96, 8192), _logint(rng, 48, 4096)
        n = max(1, min(_logint(rng, 1, 200), 400000000 // (nx * ny)))
        sr = storage != "f32" and rng.random() < 0.4
        return dict(kind=kind, nx=nx, ny=ny, n=n, storage=storage, sr=sr,
                    inlet=storage != "f32" and rng.random() < 0.4)
    if kind == "frame":
        nx, ny = _logint(rng, 64, 1400), _logint(rng, 40, 800)
        return dict(kind=kind, nx=nx, ny=ny, n=_logint(rng, 1, 32), width=2 * nx, height=2 * ny)
    if kind == "edit":
        return dict(kind=kind, nx=_logint(rng, 64, 1400), ny=_logint(rng, 40, 800), n=_logint(rng, 1, 32),
                    points=rng.randint(20, 600))
    if kind == "observe":
        return dict(kind=kind, nx=_logint(rng, 128, 1400), ny=_logint(rng, 64, 700), n=_logint(rng, 1, 50),
                    storage=rng.choice(["f64", "f64", "f32", "f16"]))
    if kind == "batch":
        storage = rng.choice(["f32", "f16", "bf16"])
        return dict(kind=kind, count=rng.randint(2, 16), n=_logint(rng, 10, 200), storage=storage,
                    sr=storage != "f32" and rng.random() < 0.3)
    if kind == "closure":
        return dict(kind=kind, nx=_logint(rng, 96, 2048), ny=_logint(rng, 48, 1024), n=rng.choice([10, 20, 40]),
                    storage=rng.choice(["f32", "f32", "f16"]))
    if kind == "train":
        return dict(kind=kind, n=rng.randint(1, 4), h=_logint(rng, 32, 256), w=_logint(rng, 48, 512))
    return dict(kind="sample", nx=_logint(rng, 256, 2048), ny=_logint(rng, 128, 1024), n=rng.choice([10, 20]),
                factor=rng.choice([2, 4]))


# ---- inputs, from the seed alone ------------------------------------------------------

U_IN, NOISE = 0.06, 0.01


def _omega(case):
    """tau 0.6 to 0.8: stable for any number of steps at these speeds."""
    return float(np.float32(1.0 / (0.8 if case.get("storage") == "f64" else 0.65)))


def _circles(nx, ny, seed, fraction=0.05):
    """Solid circles away from the inlet and the outflow up to a solid fraction."""
    rng = np.random.default_rng(seed)
    m = np.zeros((ny, nx), np.uint8)
    rmax = max(3.0, min(nx, ny) / 24.0)
    solid, clear = 0, max(4, nx // 10)
    for _ in range(400):
        if solid >= fraction * nx * ny:
            break
        r = rng.uniform(2.0, rmax)
        cx, cy = rng.uniform(clear + r, max(clear + r, nx - 1 - 2 * clear - r)), rng.uniform(0, ny - 1)
        y0, y1 = max(int(cy - r), 0), min(int(cy + r) + 2, ny)
        x0, x1 = max(int(cx - r), 0), min(int(cx + r) + 2, nx)
        yy, xx = np.mgrid[y0:y1, x0:x1]
        sub = m[y0:y1, x0:x1]
        before = int(sub.sum())
        sub[(xx - cx) ** 2 + (yy - cy) ** 2 <= r * r] = 1
        solid += int(sub.sum()) - before
    return m


def _mask(case, seed):
    m = _circles(case["nx"], case["ny"], seed)
    if case["kind"] in ("frame", "edit"):  # the reference's wall rows
        m[0, :] = 1
        m[-1, :] = 1
    return m


def _stroke(case, seed):
    """(location, value) pairs of a diagonal stroke, every eighth erasing."""
    rng = np.random.default_rng(seed + 77)
    nx, ny, k = case["nx"], case["ny"], case["points"]
    x = np.clip(nx // 3 + np.arange(k) % max(1, nx // 3), 1, nx - 2)
    y = np.clip(ny // 4 + (np.arange(k) * ny // (2 * k)) + rng.integers(0, 3, k), 1, ny - 2)
    return np.stack([x + y * nx, (np.arange(k) % 8 != 7)], 1).astype(np.uint32)


def _domains(case, seed):
    k = case["count"]
    rng = np.random.default_rng(1000 * k + case["n"])  # the sizes are the case's
    nx, ny = rng.integers(128, 1025, k).astype(np.uint32), rng.integers(64, 513, k).astype(np.uint32)
    rng = np.random.default_rng(seed)
    omega = (1.0 / rng.uniform(0.58, 0.8, k)).astype(np.float32)
    u = rng.uniform(0.02, 0.07, k).astype(np.float32)
    return nx, ny, omega, u, [_circles(int(a), int(b), seed * 1000 + d) for d, (a, b) in enumerate(zip(nx, ny))]


def _weights(seed):
    rng = np.random.default_rng(seed + 5)
    out = []
    for i, (ci, co) in enumerate(LAYERS):
        lim = math.sqrt(6.0 / (ci * 9)) * (0.1 if i == 3 else 1.0)
        out += [rng.uniform(-lim, lim, co * ci * 9), rng.uniform(-0.05, 0.05, co)]
    return np.concatenate(out).astype(np.float32)


def _snapshots(case, seed):
    """Features and loss coefficients of a coarse snapshot, as the samples have them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w = case["n"], case["h"], case["w"]

    def smooth(c, amp):
        a = torch.randn(n, c, h, w, generator=g, device="cuda")
        return amp * torch.nn.functional.avg_pool2d(a, 5, 1, 2, count_include_pad=False) * 5.0

    feat = torch.cat([smooth(1, 0.3), 0.6 + smooth(1, 0.2), smooth(1, 0.2),
                      (torch.rand(n, 1, h, w, generator=g, device="cuda") < 0.05).float()], 1)
    a = torch.rand(n, 1, h, w, generator=g, device="cuda") + 0.1
    label = 0.08 * torch.rand(n, 1, h, w, generator=g, device="cuda")
    return feat.contiguous(), torch.cat([a, a * label, a * label * label], 1).contiguous()


# ---- what a program keeps -----------------------------------------------------------------

def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _lattice(case, seed):
    edge = L.EDGE_REF if case["kind"] in ("frame", "edit") else L.EDGE_CHANNEL
    lat = L.Lattice(case["nx"], case["ny"], _omega(case), edge, STORAGE[case.get("storage", "f32")])
    if edge == L.EDGE_CHANNEL:
        lat.set_inlet_velocity(U_IN)
    if case.get("inlet"):
        lat.set_storage_reference(True)
    lat.init_equilibrium(1.0, U_IN, 0.0, NOISE, seed)
    lat.draw_mask(_mask(case, seed))
    if case.get("sr"):
        lat.set_rounding(L.ROUND_STOCHASTIC, seed)
    return lat


def prepare(case, seed):
    lib = L.load_library()
    st = dict(case=case, lib=lib)
    kind = case["kind"]
    if kind == "batch":
        nx, ny, omega, u, masks = _domains(case, seed)
        b = st["batch"] = B.Batch(nx, ny, omega, u, STORAGE[case["storage"]])
        for d, m in enumerate(masks):
            b.set_mask(d, m)
        if case["sr"]:
            b.set_rounding(L.ROUND_STOCHASTIC, seed)
        b.autotune(8)
        b.init_equilibrium(NOISE, seed)
        return st
    if kind == "train":
        net = st["net"] = C.ClosureNet(_weights(seed))
        st["feat"], st["coef"] = _snapshots(case, seed)
        g = torch.Generator(device="cuda").manual_seed(seed + 9)
        net.t = 10
        net.m.copy_(1e-4 * torch.randn(net.m.numel(), generator=g, device="cuda"))
        net.v.copy_(1e-7 * (0.5 + torch.rand(net.v.numel(), generator=g, device="cuda")))
        return st
    lat = st["lat"] = _lattice(case, seed)
    nx, ny = case["nx"], case["ny"]
    dev = torch.device("cuda")
    st["fields"] = [torch.zeros(ny, nx, device=dev) for _ in range(3)]
    if kind == "frame":
        st["rgb"] = torch.zeros(case["height"], case["width"], 3, device=dev)
    elif kind == "edit":
        st["pairs"] = _stroke(case, seed)
    elif kind == "closure":
        w = _weights(seed)
        L._check(lib.lbm_closure_set_weights(lat.handle, w.ctypes.data_as(ctypes.c_void_p), w.size))
        L._check(lib.lbm_closure_enable(lat.handle, 1.0))
    elif kind == "sample":
        f = case["factor"]
        h, w = ny // f, nx // f
        st["pops"] = torch.zeros(9, ny, nx, device=dev)
        st["solid"] = torch.from_numpy(_mask(case, seed)).to(dev)
        st["feat"], st["coef"] = torch.zeros(4, h, w, device=dev), torch.zeros(3, h, w, device=dev)
        st["scratch"] = torch.zeros(6 * h * w, device=dev)
        st["solid_c"] = torch.zeros(h, w, dtype=torch.uint8, device=dev)
        st["stream"] = ctypes.c_void_p(lat.get_stream())
    return st


def _read(st):
    for code, t in enumerate(st["fields"]):  # rho, jx, jy
        L._check(st["lib"].lbm_read_field_device(st["lat"].handle, code, _p(t)))
    return st["fields"]


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    n = case["n"]
    if kind == "batch":
        b = st["batch"]
        b.step(n)
        return [b.field(d, "rho") for d in range(case["count"])] + [b.conservation()]
    if kind == "train":
        net = st["net"]
        z = net.forward(st["feat"])
        loss, gz = net.loss(z, st["coef"], z.numel())
        net.backward(gz)
        net.adam(1e-3)
        return [z, loss, net.grads, net.params]
    lat = st["lat"]
    if kind == "step":
        lat.iterate(n)
        return _read(st)
    if kind == "frame":
        lat.iterate(n)
        L._check(st["lib"].lbm_render_device(lat.handle, L.SummaryStat.Curl, L.ColorMap.Jet, case["width"],
                                             case["height"], _p(st["rgb"])))
        return [st["rgb"]] + _read(st)
    if kind == "edit":
        lat.draw_points(st["pairs"])
        lat.iterate(n)
        return [lat.summary(L.SummaryStat.Curl), lat.render(rgba=True)]
    if kind == "observe":
        lat.iterate(n)
        force, sums = lat.force(), lat.conservation()
        return [force, sums] + _read(st)
    if kind == "closure":
        L._check(st["lib"].lbm_closure_infer(lat.handle))
        lat.iterate(n)
        return _read(st)
    lat.iterate(n)
    L._check(st["lib"].lbm_read_populations_device(lat.handle, _p(st["pops"])))
    C.sample(st["lib"], st["stream"], st["pops"], st["solid"], case["factor"], st["feat"], st["coef"], st["scratch"],
             st["solid_c"])
    return [st["feat"], st["coef"], st["solid_c"]]


def work(case):
    """State (populations, mask) in and out once, the outputs written once."""
    kind, n = case["kind"], case["n"]
    if kind == "batch":
        cells = case["count"] * 576 * 288  # mean domain
        return dict(bytes=cells * (18 * BYTES[case["storage"]] + 4), flops=cells * n * FLOPS)
    if kind == "train":
        px = n * case["h"] * case["w"]
        mac = sum(ci * co * 9 for ci, co in LAYERS)
        back = sum(ci * co * 9 for ci, co in LAYERS[1:])
        return dict(bytes=px * 4 * (4 + 3 + 1), flops=px * 2 * (2 * mac + back))
    cells = case["nx"] * case["ny"]
    es = BYTES[case.get("storage", "f32")]
    out = 12 * cells
    flops = cells * n * FLOPS
    if kind == "frame":
        out += 12 * case["width"] * case["height"]
    elif kind == "edit":
        out = 8 * cells
    elif kind == "closure":
        flops += 2 * cells * sum(ci * co * 9 for ci, co in LAYERS)
    elif kind == "sample":
        out = 7 * 4 * cells // case["factor"] ** 2
    return dict(bytes=cells * 18 * es + out + cells // 8, flops=flops)


# ---- the same in 64 bits -------------------------------------------------------------------

CX = [q % 3 - 1 for q in range(9)]
CY = [q // 3 - 1 for q in range(9)]  # row step: north is row - 1
W9 = [1 / 36, 1 / 9, 1 / 36, 1 / 9, 4 / 9, 1 / 9, 1 / 36, 1 / 9, 1 / 36]


def _equilibrium(rho, ux, uy):
    usq = 1.5 * (ux * ux + uy * uy)
    cu = [3.0 * (CX[q] * ux - CY[q] * uy) for q in range(9)]
    return torch.stack([W9[q] * rho * (1.0 + cu[q] + 0.5 * cu[q] * cu[q] - usq) for q in range(9)])


def _noise(seed, nx, ny):
    """The engine's documented noise: splitmix64 of (seed, cell, component), 24 bits."""
    def shr(z, k):
        return (z >> k) & ((1 << (64 - k)) - 1)

    def wrap(v):
        v &= (1 << 64) - 1
        return v - (1 << 64) if v >= 1 << 63 else v

    cell = torch.arange(nx * ny, dtype=torch.int64, device="cuda")
    out = []
    for comp in range(2):
        z = wrap(seed) + (2 * cell + comp + 1) * wrap(0x9E3779B97F4A7C15)
        z = (z ^ shr(z, 30)) * wrap(0xBF58476D1CE4E5B9)
        z = (z ^ shr(z, 27)) * wrap(0x94D049BB133111EB)
        z = z ^ shr(z, 31)
        out.append((shr(z, 40).double() / (1 << 24) * 2.0 - 1.0).view(ny, nx))
    return out


def _initial(nx, ny, u, seed, channel):
    u, amp = float(np.float32(u)), float(np.float32(NOISE))
    ax, ay = _noise(seed, nx, ny)
    ux, uy = u + amp * ax, amp * ay
    if channel:
        ux[:, 0] = u
        uy[:, 0] = 0.0
    f = _equilibrium(torch.ones_like(ux), ux, uy)
    f[7] -= uy * uy  # set_equil takes the s direction's square term with a minus sign
    return f


def _moments(f):
    jx = (f[2] + f[5] + f[8]) - (f[0] + f[3] + f[6])
    jy = (f[0] + f[1] + f[2]) - (f[6] + f[7] + f[8])
    return f.sum(0), jx, jy


def _channel(f, mask, omega, n, rate=None):
    """n channel steps: the collided state and the last collision's moments.
    `rate` gives a per-cell relaxation rate from the moments."""
    solid = torch.from_numpy(mask.astype(bool)).cuda()
    inert = solid.clone()
    inert[:, 0] = True
    ny, nx = mask.shape

    def up(a, q):  # a at the upstream cell of direction q
        a = torch.roll(a, CY[q], 0)
        return torch.cat([a[:, :1], a[:, :-1]], 1) if CX[q] > 0 else torch.cat([a[:, 1:], a[:, -1:]], 1) if CX[
            q] < 0 else a

    wall = [up(solid, q) for q in range(9)]
    for k in range(n):
        if k:
            g = torch.stack([torch.where(wall[q], f[8 - q], up(f[q], q)) if q != 4 else f[4] for q in range(9)])
            f = torch.where(inert, f, g)
        rho, jx, jy = _moments(f)
        w = omega if rate is None else rate(rho, jx, jy)
        f = torch.where(inert, f, f + w * (_equilibrium(rho, jx / rho, jy / rho) - f))
    return f, (rho, jx, jy), solid, wall


def _ref(f, mask, omega, n):
    """n steps with the reference's edges: two buffer sets, one rest plane."""
    ny, nx = mask.shape
    cells = nx * ny
    solid = torch.from_numpy(mask.astype(bool)).cuda().view(-1)
    i = torch.arange(cells, device="cuda")
    still = solid | (i % nx == 0) | (i // nx == ny - 1)
    src = []
    for q in range(9):
        j = (i - CX[q] - CY[q] * nx) & 0xFFFFFFFF
        src.append(torch.where(j >= cells, cells - 1, j))
    sets = [f.reshape(9, -1).clone(), f.reshape(9, -1).clone()]
    for k in range(n):
        a, b = sets[k % 2], sets[1 - k % 2]
        rho, jx, jy = _moments(a)
        a += omega * (_equilibrium(rho, jx / rho, jy / rho) - a)
        for q in range(9):
            if q == 4:
                b[4] = a[4]
            else:
                b[q] = torch.where(still, b[q], torch.where(solid[src[q]], a[8 - q], a[q][src[q]]))
    return [v.view(ny, nx) for v in (rho, jx, jy)]


def _curl(rho, jx, jy):
    ny, nx = rho.shape
    i = torch.arange(nx * ny, device="cuda")

    def at(a, j):
        j = j & 0xFFFFFFFF
        return a.reshape(-1)[torch.where(j >= nx * ny, nx * ny - 1, j)]

    c = 10.0 * (at(jy, i + 1) - at(jy, i - 1) - at(jx, i - nx) + at(jx, i + nx)) / rho.reshape(-1)
    c = torch.where((i % nx == 0) | (i // nx == ny - 1), torch.zeros_like(c), c)
    return c.view(ny, nx)


def _net64(x, w):
    o = 0
    for k, (ci, co) in enumerate(LAYERS):
        x = torch.nn.functional.conv2d(x, w[o:o + co * ci * 9].view(co, ci, 3, 3),
                                       w[o + co * ci * 9:o + co * ci * 9 + co], padding=1)
        o += co * ci * 9 + co
        x = torch.relu(x) if k < 3 else x
    return x


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "train":
        w = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_(True)
        feat, coef = (t.double() for t in _snapshots(case, seed))
        z = _net64(feat, w)
        dt = 0.25 * torch.sigmoid(z)
        loss = (coef[:, :1] * dt * dt - 2.0 * coef[:, 1:2] * dt + coef[:, 2:]).sum() / z.numel()
        loss.backward()
        g = w.grad
        gen = torch.Generator(device="cuda").manual_seed(seed + 9)
        m = (1e-4 * torch.randn(g.numel(), generator=gen, device="cuda")).double()
        v = (1e-7 * (0.5 + torch.rand(g.numel(), generator=gen, device="cuda"))).double()
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        step = 1e-3 * (m / (1 - 0.9 ** 11)) / (torch.sqrt(v / (1 - 0.999 ** 11)) + 1e-8)
        return [z.detach(), loss.detach().view(1), g, (w - step).detach()]
    if kind == "batch":
        nx, ny, omega, u, masks = _domains(case, seed)
        out, sums = [], []
        for d in range(case["count"]):
            f = _initial(int(nx[d]), int(ny[d]), u[d], seed + d, True)
            _, (rho, jx, jy), solid, _ = _channel(f, masks[d], float(omega[d]), n)
            out.append(rho.cpu().numpy())
            sums.append([float(v[~solid].sum()) for v in (rho, jx, jy)])
        return out + [np.array(sums)]
    nx, ny, omega = case["nx"], case["ny"], _omega(case)
    mask = _mask(case, seed)
    f = _initial(nx, ny, U_IN, seed, kind not in ("frame", "edit"))
    if kind == "frame":
        return [None] + _ref(f, mask, omega, n)
    if kind == "edit":
        for loc, val in _stroke(case, seed):
            mask.reshape(-1)[loc] = val
        return [_curl(*_ref(f, mask, omega, n)).cpu().numpy(), None]
    if kind == "closure":
        rho, jx, jy = _moments(f)
        solid = torch.from_numpy(mask.astype(bool)).cuda()
        zero = torch.zeros_like(rho)
        x = torch.stack([torch.where(solid, zero, (rho - 1.0) * 50.0), torch.where(solid, zero, jx / rho * 10.0),
                         torch.where(solid, zero, jy / rho * 10.0), solid.double()])[None]
        w = torch.from_numpy(_weights(seed)).bfloat16().double().cuda()
        dt = 0.25 * torch.sigmoid(_net64(x, w))[0, 0]
        speed = torch.where(solid, zero, torch.sqrt(jx * jx + jy * jy) / rho)

        def rate(rho, jx, jy):
            d = torch.clamp(speed, min=0.01)
            s = torch.sqrt(jx * jx + jy * jy) / rho
            keep = (s >= torch.clamp(speed - d, min=0.0)) & (s <= speed + d)
            return torch.where(keep, 1.0 / (1.0 / omega + dt), torch.full_like(dt, omega))

        return list(_channel(f, mask, omega, n, rate)[1])
    f, (rho, jx, jy), solid, wall = _channel(f, mask, omega, n)
    if kind == "step":
        return [rho, jx, jy]
    if kind == "observe":
        fluid = ~solid
        fluid[:, 0] = False
        fx = fy = 0.0
        for q in range(9):
            if q != 4:
                s = float(f[8 - q][wall[q] & fluid].sum())
                fx, fy = fx + 2.0 * s * CX[8 - q], fy - 2.0 * s * CY[8 - q]
        return [np.array([fx, fy]), np.array([float(v[~solid].sum()) for v in (rho, jx, jy)]), rho, jx, jy]
    # sample: the populations the next step would collide (streamed), coarsened
    g = torch.stack([torch.where(wall[q], f[8 - q], _upstream(f[q], q)) if q != 4 else f[4] for q in range(9)])
    inert = solid.clone()
    inert[:, 0] = True
    return _sample64(torch.where(inert, f, g), solid, case["factor"])


def _upstream(a, q):
    a = torch.roll(a, CY[q], 0)
    return torch.cat([a[:, :1], a[:, :-1]], 1) if CX[q] > 0 else torch.cat([a[:, 1:], a[:, -1:]], 1) if CX[q] < 0 else a


def _sample64(f, solid, k):
    ny, nx = solid.shape
    h, w = ny // k, nx // k

    def blocks(a):
        return a[:h * k, :w * k].reshape(h, k, w, k).sum((1, 3))

    rho, jx, jy = _moments(f)
    fl = (~solid).double()
    cnt, r = blocks(fl), blocks(rho * fl)
    rs = torch.where(cnt > 0, r, torch.ones_like(r))
    ux, uy = blocks(jx * fl) / rs, blocks(jy * fl) / rs

    def fine(a):
        out = torch.zeros(ny, nx, dtype=a.dtype, device=a.device)
        out[:h * k, :w * k] = a.repeat_interleave(k, 0).repeat_interleave(k, 1)
        return out

    vx, vy = jx / rho - fine(ux), jy / rho - fine(uy)
    txx, txy, tyy = (blocks(rho * fl * a) / rs for a in (vx * vx, vx * vy, vy * vy))
    avg = torch.where(cnt > 0, r / cnt.clamp(min=1.0), torch.zeros_like(r))
    solid_c = 2 * cnt < k * k

    def left(a):
        return torch.cat([a[:, :1], a[:, :-1]], 1)

    def right(a):
        return torch.cat([a[:, 1:], a[:, -1:]], 1)

    def north(a):
        return torch.roll(a, 1, 0)

    def south(a):
        return torch.roll(a, -1, 0)

    valid = ~(solid_c | left(solid_c) | right(solid_c) | north(solid_c) | south(solid_c))
    valid[:, 0] = False
    valid[:, -1] = False
    dxx = 0.5 * (right(ux) - left(ux))
    dyx = 0.5 * (right(uy) - left(uy))
    dxy = 0.5 * (north(ux) - south(ux))
    dyy = 0.5 * (north(uy) - south(uy))
    sxx, sxy, d = 0.5 * (dxx - dyy), 0.5 * (dxy + dyx), 0.5 * (txx - tyy)
    v, c = valid.double(), (~solid_c).double()
    feat = torch.stack([c * (avg - 1.0) * 50.0, c * ux * 10.0, c * uy * 10.0, solid_c.double()])
    coef = torch.stack([v * (8.0 / 9.0) * (sxx * sxx + sxy * sxy), v * (-4.0 / 3.0) * (d * sxx + txy * sxy),
                        v * 2.0 * (d * d + txy * txy)])
    return [feat, coef, solid_c.to(torch.uint8)]
