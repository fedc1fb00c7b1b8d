"""Workloads for timing the framework through its public entry points.

Every case is a dict of plain values.  ``listed()`` names the ones that are
always timed, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes
what a program holds before the call (contexts, networks, frames on the GPU),
``run`` is one pass, ``work`` the bytes and operations a pass cannot do
without, and ``exact`` the same results in 64 bits with plain torch.

Kinds of case:

* ``solve``: a camera frame in, a fixed number of FISTA iterations, the volume
  and the objective out - what the sparse-inverse-recon program does per frame;
* ``batch``: several small frames reconstructed by one call;
* ``operators``: the forward and the adjoint operator on device buffers,
  through the C ABI;
* ``predict`` / ``gradients``: the learned warm start's inference and the
  forward and backward pass of its training;
* ``segment``: particle segmentation of a volume of intensities.
"""
import ctypes
import importlib
import math
import os

import numpy as np
import torch

PACKAGE = "rihvr---regularized-inverse-holographic-volume-reconstruction_b200"

DEV = "cuda"


def _pkg():
    return importlib.import_module(PACKAGE)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _solve(name, width, height, nz, iterations, **kw):
    """`width` x `height` is the camera frame, before zero padding."""
    c = {"kind": "solve", "width": width, "height": height, "pad": 0, "nz": nz, "iterations": iterations,
         "mode": 7, "tv_iterations": 5, "storage": "f32", "record": True, "z0": 1000.0, "dz": 2.0,
         "dx": 1.1, "lam": 0.632, "l1": 0.15, "tv": 0.1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one small frame: launches and latency decide.  The size the packaged
        # warm-start network was trained on.
        _solve("solve_128x128x32", 128, 128, 32, 10),
        # the plain FISTA + TV configuration: a 256 x 256 frame padded to 384
        _solve("solve_384x384x40", 256, 256, 40, 10, pad=64, z0=0.0, dz=2000.0, dx=10.4, lam=0.633, l1=0.001,
               tv=0.01),
        # sparsity alone (TV weight 0), as a user without extended objects sets it
        _solve("solve_l1_512x512x200", 512, 512, 200, 5, mode=7, tv=0.0, dz=2.5),
        # 3-D total variation: objects that span several planes
        _solve("solve_tv3d_256x256x100", 256, 256, 100, 5, mode=6),
        # a whole 1280 x 1024 sensor: rectangular, no power of two, plane spacing with no short binary form
        _solve("solve_1280x1024x64", 1280, 1024, 64, 3, dz=12.7, dx=3.45),
        # the large-volume configuration (padded 2048 frame, half-precision
        # storage, 10 TV iterations) with fewer planes
        _solve("solve_f16_2304x2304x48", 2048, 2048, 48, 3, pad=128, tv_iterations=10, storage="f16", record=False,
               dz=4.0, dx=2.2, lam=0.532, l1=0.05, tv=0.05),
        # the headline volume
        _solve("solve_1024x1024x1000", 1024, 1024, 1000, 4, record=False, z0=2500.0),
        # a short time series of small frames in one call
        {"name": "batch_16x128x128x32", "kind": "batch", "frames": 16, "width": 128, "height": 128, "nz": 32,
         "iterations": 10, "tv_iterations": 5},
        # both directions of the operator alone, for a caller with an iteration
        # of its own; the series frames' side, planes that are not exactly evenly spaced
        {"name": "operators_640x640x150", "kind": "operators", "width": 640, "height": 640, "nz": 150, "dz": 7.3},
        # learned warm start: inference on the 512 x 512 frames the second set of
        # weights is for, with half the planes (a network holds 0.9 KB a voxel)
        {"name": "predict_100x512x512", "kind": "predict", "nz": 100, "height": 512, "width": 512},
        # its training: the gradients of one hologram
        {"name": "gradients_32x128x128", "kind": "gradients", "nz": 32, "height": 128, "width": 128},
        # particle segmentation of a reconstructed volume
        {"name": "segment_512x512x200", "kind": "segment", "width": 512, "height": 512, "nz": 200, "objects": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A supported plane side: even, prime factors 2, 3, 5 and 7."""
    while True:
        n = 2 * int(round(_log_int(rng, lo, hi) / 2))
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1 and lo <= n <= hi:
            return n


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "operators", "operators", "predict", "gradients", "segment"])
    dz = rng.choice([1.5, 2.0, 4.0, 8.0, round(rng.uniform(0.7, 20.0), 2)])
    if kind == "solve":
        mode = rng.choice([7, 7, 7, 7, 6, 5])
        square = rng.random() < 0.6
        w = rng.choice([64, 128, 256, 384, 512, 640, 768, 1024]) if square else _side(rng, 64, 1536)
        h = w if square else _side(rng, 64, 1536)
        most = 6e7 if square else 3e7
        nz = _log_int(rng, 6, max(7, min(400, most / (w * h))))
        return _solve(None, w, h, nz, rng.randint(3, 6), mode=7 if mode == 5 else mode,
                      tv=0.0 if mode == 5 else round(rng.uniform(0.02, 0.2), 3),
                      l1=round(rng.uniform(0.05, 0.2), 3), tv_iterations=rng.randint(1, 10),
                      storage="f16" if mode == 7 and rng.random() < 0.3 else "f32", record=rng.random() < 0.5,
                      dz=dz, dx=round(rng.uniform(1.0, 6.0), 2))
    if kind == "batch":
        return {"kind": "batch", "frames": rng.randint(4, 16), "width": rng.choice([64, 96, 128, 192]),
                "height": rng.choice([64, 128]), "nz": rng.randint(8, 40), "iterations": rng.randint(4, 10),
                "tv_iterations": rng.randint(2, 8)}
    if kind == "operators":
        w = rng.choice([64, 128, 256, 384, 512, 640, 768, 1024]) if rng.random() < 0.5 else _side(rng, 48, 1536)
        h = w if rng.random() < 0.6 else _side(rng, 48, 1536)
        return {"kind": "operators", "width": w, "height": h, "nz": _log_int(rng, 4, max(5, min(300, 6e7 / (w * h)))),
                "dz": dz}
    if kind == "predict":
        w = rng.choice([64, 100, 128, 256, 512, 512])
        return {"kind": "predict", "nz": 4 * rng.randint(4, 20), "height": 4 * rng.randint(16, 100), "width": w}
    if kind == "gradients":
        return {"kind": "gradients", "nz": 4 * rng.randint(2, 8), "height": 4 * rng.randint(12, 32),
                "width": rng.choice([52, 64, 96, 128, 128])}
    return {"kind": "segment", "width": rng.randint(100, 700), "height": rng.randint(100, 700),
            "nz": rng.randint(20, 150), "objects": rng.randint(50, 600)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _planes(z0, dz, nz):
    """Plane positions, in single precision as the parameter file gives them."""
    i = np.arange(nz, dtype=np.float32)
    return (np.float32(z0) + i * np.float32(dz)).astype(np.float32).astype(np.float64)


def _turns(W, H, dx, lam):
    """Phase of the propagation kernel per unit length, in turns, FP64."""
    lam, dx = float(np.float32(lam)), float(np.float32(dx))
    fy = torch.fft.fftfreq(H, dtype=torch.float64, device=DEV)[:, None]
    fx = torch.fft.fftfreq(W, dtype=torch.float64, device=DEV)[None, :]
    a = (lam / dx) ** 2 * (fx * fx + fy * fy)
    return torch.where(a >= 1.0, torch.full_like(a, -1.0), -a / (torch.sqrt((1.0 - a).clamp_min(0.0)) + 1.0)) / lam


def _kernel(z, turns, dtype=torch.complex128):
    """exp(2 pi i z turns) for the planes `z` (a list), [planes, H, W]."""
    u = torch.as_tensor(z, dtype=torch.float64, device=DEV)[:, None, None] * turns
    u = 2.0 * math.pi * (u - torch.round(u))
    return torch.polar(torch.ones_like(u), u).to(dtype)


def _chunk(W, H):
    return max(1, int(2.5e7 / (W * H)))


def _camera_frame(W, H, z, turns, seed):
    """An 8-bit camera frame (H x W, on the GPU) of opaque disks on the planes."""
    g = _generator(seed)
    nz = len(z)
    n = max(12, W * H // 1500)
    r = lambda lo, hi: lo + (hi - lo) * torch.rand(n, generator=g, device=DEV)  # noqa: E731
    x, y, rad = r(0, W), r(0, H), r(1.0, 4.0)
    k = torch.sort(torch.randint(0, nz, (n,), generator=g, device=DEV))[0]
    noise = torch.randn((H, W), generator=g, device=DEV)
    o = torch.arange(-4, 5, device=DEV)
    oy, ox = o.repeat_interleave(9), o.repeat(9)
    xi, yi = (x.floor().long()[:, None] + ox), (y.floor().long()[:, None] + oy)
    inside = (xi + 0.5 - x[:, None]) ** 2 + (yi + 0.5 - y[:, None]) ** 2 <= (rad * rad)[:, None]
    at = (k[:, None] * H + yi % H) * W + xi % W
    at = at[inside]
    S = torch.zeros((H, W), dtype=torch.complex64, device=DEV)
    step = _chunk(W, H)
    for a in range(0, nz, step):
        b = min(nz, a + step)
        m = torch.zeros((b - a) * H * W, dtype=torch.complex64, device=DEV)
        part = at[(at >= a * H * W) & (at < b * H * W)] - a * H * W
        m[part] = 1.0
        S += (torch.fft.fft2(m.view(b - a, H, W)) * _kernel(z[a:b], turns, torch.complex64)).sum(0)
    field = 1.0 - torch.fft.ifft2(S)
    image = field.real ** 2 + field.imag ** 2
    image = (0.4 * image + 0.01 * noise).clamp(0.0, 1.0)
    return torch.round(255.0 * image).to(torch.uint8)


def _hologram(frame, pad):
    """The preprocessing of a frame without a background, in FP64."""
    f = frame.double()
    return torch.nn.functional.pad(f / f.mean() - 1.0, (pad, pad, pad, pad))


def _back_propagated(case, seed):
    """t A^H b of a frame (complex64, on the GPU): the network's input."""
    W, H, nz = case["width"], case["height"], case["nz"]
    z, turns = _planes(1000.0, 2.0, nz), _turns(W, H, 1.1, 0.632)
    R = torch.fft.fft2(_hologram(_camera_frame(W, H, z, turns, seed), 0)).to(torch.complex64)
    out = torch.empty((nz, H, W), dtype=torch.complex64, device=DEV)
    step = _chunk(W, H)
    for a in range(0, nz, step):
        out[a:a + step] = torch.fft.ifft2(R * _kernel(z[a:a + step], turns, torch.complex64).conj()) / nz
    return out


def _solver_params(case):
    p = _pkg().default_params()
    p.start_plane, p.plane_stepsize, p.num_planes = case.get("z0", 1000.0), case.get("dz", 2.0), case["nz"]
    p.wavelength, p.resolution = case.get("lam", 0.632), case.get("dx", 1.1)
    p.zero_padding = case.get("pad", 0)
    p.num_inverse_iterations = case.get("iterations", 1)
    p.num_tv_iterations = case.get("tv_iterations", 5)
    p.regularization_param, p.regularization_TV_param = case.get("l1", 0.15), case.get("tv", 0.1)
    p.mode = case.get("mode", 7)
    p.storage = _pkg().STORE_F16 if case.get("storage") == "f16" else _pkg().STORE_F32
    p.record_objective = int(case.get("record", True))
    return p


class _Network:
    """A network with the packaged weights that its depth is nearest to."""

    def __init__(self, case):
        self.net = _pkg().UNet(case["nz"], case["height"], case["width"])
        name = "warmstart_unet_c4_200x128x128.npy" if case["nz"] > 64 else "warmstart_unet_32x128x128.npy"
        self.net.load(os.path.join(os.path.dirname(_pkg().__file__), name))

    def __del__(self):
        if hasattr(self, "net"):
            self.net.destroy()


def _target(xbp):
    """A sparse solution of the kind FISTA ends at: the strongest voxels."""
    a = xbp.abs()
    return xbp * (a > 3.0 * a.mean()) * 2.0


def _intensities(case, seed):
    """Bright balls in a weak background, [nz, H, W] FP32."""
    g = _generator(seed)
    nz, H, W, n = case["nz"], case["height"], case["width"], case["objects"]
    v = 1e-4 * torch.rand((nz, H, W), generator=g, device=DEV)
    r = lambda lo, hi: lo + (hi - lo) * torch.rand(n, generator=g, device=DEV)  # noqa: E731
    x, y, z, rad, amp = r(0, W), r(0, H), r(0, nz), r(1.0, 5.0), r(0.2, 1.0)
    o = torch.arange(-5, 6, device=DEV)
    oz, oy, ox = (t.reshape(-1) for t in torch.meshgrid(o, o, o, indexing="ij"))
    xi, yi, zi = x.long()[:, None] + ox, y.long()[:, None] + oy, z.long()[:, None] + oz
    d = ((xi - x[:, None]) ** 2 + (yi - y[:, None]) ** 2 + (zi - z[:, None]) ** 2).sqrt() / rad[:, None]
    ok = (d <= 1) & (xi >= 0) & (xi < W) & (yi >= 0) & (yi < H) & (zi >= 0) & (zi < nz)
    val = amp[:, None] * (1.0 - 0.5 * d)
    v.view(-1).scatter_reduce_(0, ((zi * H + yi) * W + xi)[ok], val[ok], "amax")
    return v


class _Context:
    """A solver context held through the C ABI."""

    def __init__(self, params, width, height):
        self.lib = _pkg().load_library()
        self.handle = ctypes.c_void_p()
        rc = self.lib.rihvr_create(ctypes.byref(params), width, height, ctypes.byref(self.handle))
        if rc:
            raise RuntimeError("rihvr_create: %d" % rc)

    def __del__(self):
        if self.handle:
            self.lib.rihvr_destroy(self.handle)
            self.handle = None


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("solve", "batch", "operators"):
        W, H = case["width"], case["height"]
        z = _planes(case.get("z0", 1000.0), case.get("dz", 2.0), case["nz"])
    if kind == "solve":
        pad = case["pad"]
        s["frame"] = _camera_frame(W, H, z, _turns(W, H, case["dx"], case["lam"]), seed)
        s["solver"] = _pkg().SparseCompressiveHolo(_solver_params(case), W + 2 * pad, H + 2 * pad)
    elif kind == "batch":
        turns = _turns(W, H, 1.1, 0.632)
        s["holograms"] = [_hologram(_camera_frame(W, H, z, turns, 1000 * seed + i), 0).float().cpu().numpy()
                          for i in range(case["frames"])]
        s["solvers"] = [_pkg().SparseCompressiveHolo(_solver_params(case), W, H) for _ in range(case["frames"])]
    elif kind == "operators":
        g = _generator(seed)
        s["context"] = _Context(_solver_params(case), W, H)
        s["volume"] = torch.randn((case["nz"], H, W), generator=g, device=DEV, dtype=torch.complex64)
        s["residual"] = torch.randn((H, W), generator=g, device=DEV)
        s["hologram"] = torch.empty((H, W), device=DEV)
        s["gradient"] = torch.empty_like(s["volume"])
    elif kind in ("predict", "gradients"):
        s["net"] = _Network(case)
        s["xbp"] = _back_propagated(case, seed)
        if kind == "gradients":
            s["xstar"] = _target(s["xbp"])
    else:
        s["intensity"] = _intensities(case, seed)
    torch.cuda.synchronize()  # the library's streams do not wait for torch's
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _volume(solver):
    """The solver's volume, viewed in its own device memory: the view keeps the solver."""
    v = solver.volume_device()
    v.solver = solver
    return v


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        solver = s["solver"]
        solver.setHologramFrame(s["frame"])
        solver.iterate(case["iterations"])
        out = {"objective": solver.calcObjectiveFunction()[0], "estimate": solver.getEstimate()}
        if case["record"]:
            out["trajectory"] = solver.iterations()["f_x"].astype(np.float32)
        volume = _volume(solver)
        # a volume that is stored in half precision is kept that way
        out["volume"] = torch.view_as_real(volume).half() if case["storage"] == "f16" else volume
        return out
    if kind == "batch":
        f = _pkg().reconstruct_batch(s["solvers"], s["holograms"])
        return {"objectives": np.array(f, np.float32), "volumes": [_volume(v) for v in s["solvers"]]}
    if kind == "operators":
        c = s["context"]
        for call, a, b in ((c.lib.rihvr_forward, "volume", "hologram"), (c.lib.rihvr_adjoint, "residual", "gradient")):
            rc = call(c.handle, ctypes.c_void_p(s[a].data_ptr()), ctypes.c_void_p(s[b].data_ptr()), 1)
            if rc:
                raise RuntimeError("operator: %d" % rc)
        return {"hologram": s["hologram"], "gradient": s["gradient"]}
    if kind == "predict":
        return s["net"].net.predict(s["xbp"])
    if kind == "gradients":
        loss, grad = s["net"].net.gradients(s["xbp"], s["xstar"])
        return {"loss": loss, "gradients": grad}
    objects, _ = _pkg().segment_intensity(s["intensity"])
    floats = ("x", "y", "z", "wx", "wy", "wz", "max_value", "mean_value")
    wholes = ("num_voxels", "xmin", "xmax", "ymin", "ymax", "zmin", "zmax")
    # one column an object that was planted; those below the threshold or merged leave zeros at the end
    table = lambda names, dtype: np.stack([np.pad(objects[k], (0, max(0, case["objects"] - len(objects))))  # noqa: E731
                                           for k in names]).astype(dtype)
    return {"floats": table(floats, np.float32), "wholes": table(wholes, np.int32)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

# (input channels, output channels, level) of the network's convolutions
LAYERS = ((16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1),
          (48, 16, 0), (16, 16, 0))


def work(case):
    kind = case["kind"]
    pad = case.get("pad", 0)
    W, H, nz = case["width"] + 2 * pad, case["height"] + 2 * pad, case["nz"]
    V = float(W) * H * nz
    fft = 5.0 * math.log2(W * H)  # operations a voxel of one 2-D transform
    if kind in ("solve", "batch"):
        # an iteration: the adjoint and the forward operator, each a volume
        # written and read between its row and column transforms, and the two
        # iterates read, the new one written and read by the forward operator
        e = 4 if case.get("storage") == "f16" else 8
        n = case["iterations"] * case.get("frames", 1)
        tv = 0 if case.get("tv", 0.1) == 0 else case["tv_iterations"]
        return {"bytes": n * V * (32 + 4 * e), "flops": n * V * (2 * fft + 40 * tv + 30)}
    if kind == "operators":
        return {"bytes": V * (8 + 16 + 16 + 8), "flops": V * (2 * fft + 16)}
    if kind in ("predict", "gradients"):
        macs = sum(27.0 * (1 if i == 0 else ci) * co / 8 ** lv for i, (ci, co, lv) in enumerate(LAYERS))
        passes = 1 if kind == "predict" else 3
        # activations of two bytes, each written and read once a pass
        act = sum(2.0 * 2 * co / 8 ** lv for _, co, lv in LAYERS)
        return {"bytes": V * (16 + passes * act), "flops": 2 * passes * V * macs}
    return {"bytes": 4 * V, "flops": 10 * V}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _shrink(v, thr):
    """Soft threshold of the real and the imaginary part."""
    if not thr > 0:
        return v
    r = torch.view_as_real(v)
    return torch.view_as_complex(torch.sign(r) * (r.abs() - thr).clamp_min(0.0))


def _roll(v, shift, axis):
    return torch.roll(v, shift, axis)


def _tv2d(xh, mu, s, n):
    gx, gy = torch.zeros_like(xh), torch.zeros_like(xh)
    for _ in range(n):
        y = xh - mu * (_roll(gx, -1, -1) - gx + _roll(gy, -1, -2) - gy)
        gx = gx + s * (_roll(y, 1, -1) - y)
        gy = gy + s * (_roll(y, 1, -2) - y)
        m = (gx.abs() ** 2 + gy.abs() ** 2).sqrt().clamp_min(1.0)
        gx, gy = gx / m, gy / m
    return xh - mu * (_roll(gx, -1, -1) - gx + _roll(gy, -1, -2) - gy)


def _tv3d(x, mu, s, n):
    g = [torch.zeros_like(x) for _ in range(3)]
    div = lambda: sum(_roll(g[a], -1, a) - g[a] for a in range(3))  # noqa: E731
    for _ in range(n):
        y = x - mu * div()
        g = [g[a] + s * (_roll(y, 1, a) - y) for a in range(3)]
    return x - mu * div()


class _Exact:
    """FISTA with backtracking, in FP64, plane chunks at a time."""

    def __init__(self, case, b):
        self.b, self.n_tv = b, case.get("tv_iterations", 5)
        self.H, self.W = b.shape
        self.z = _planes(case.get("z0", 1000.0), case.get("dz", 2.0), case["nz"])
        self.turns = _turns(self.W, self.H, case.get("dx", 1.1), case.get("lam", 0.632))
        self.l1 = float(np.float32(case.get("l1", 0.15)))
        self.tv = float(np.float32(case.get("tv", 0.1)))
        self.mode = 5 if self.tv == 0 else case.get("mode", 7)
        nz = len(self.z)
        step = nz if self.mode == 6 else _chunk(self.W, self.H)
        self.parts = [(a, min(nz, a + step)) for a in range(0, nz, step)]

    def adjoint(self, R, a, b):
        return torch.fft.ifft2(R * _kernel(self.z[a:b], self.turns).conj())

    def prox(self, xh, t):
        if self.mode == 5:
            return _shrink(xh, t * self.l1)
        mu, s = t * self.tv, 1.0 / (12.0 * t * self.tv)
        if self.mode == 7:
            return _shrink(_tv2d(xh, mu, s, self.n_tv), t * self.l1)
        return _shrink(_tv3d(_shrink(xh, 0.5 * t * self.l1), mu, s, self.n_tv), 0.5 * t * self.l1)

    def objective(self, x, r):
        f = 0.5 * (r * r).sum()
        for a, b in self.parts:
            v = x(a, b)
            f = f + self.l1 * v.abs().sum()
            if self.mode != 5:
                q = (_roll(v, 1, -1) - v).abs() ** 2 + (_roll(v, 1, -2) - v).abs() ** 2
                if self.mode == 6:
                    q = q + (_roll(v, 1, 0) - v).abs() ** 2
                f = f + self.tv * q.sqrt().sum()
        return float(f)

    def solve(self, iterations, record=False):
        nz, H, W = len(self.z), self.H, self.W
        P0 = torch.zeros((nz, H, W), dtype=torch.complex128, device=DEV)
        P1, P2 = torch.zeros_like(P0), torch.zeros_like(P0)
        d0 = torch.zeros_like(self.b)
        dx = d0
        t, alpha, beta = 1.0 / nz, 1.0, 0.0
        first = ((torch.arange(H * W, device=DEV) & 1023) < 512).view(H, W)
        wr = torch.where(first, 1.0, 0.0).double()
        wi = torch.where(first, 2.0, 1.0).double()
        r = dx - self.b
        before = float(0.5 * (r * r).sum())
        track = []
        for _ in range(iterations):
            R = torch.fft.fft2(r)
            x = lambda a, b: P1[a:b] + beta * (P1[a:b] - P0[a:b])  # noqa: E731
            for attempt in range(3):
                S = torch.zeros((H, W), dtype=torch.complex128, device=DEV)
                lim1 = lim2 = rs = 0.0
                for a, b in self.parts:
                    xa, g = x(a, b), self.adjoint(R, a, b)
                    p = self.prox(xa - t * g, t)
                    P2[a:b] = p
                    u = p - xa
                    lim1 += float((u.real * g.real + u.imag * g.imag).sum())
                    lim2 += float((u.abs() ** 2).sum())
                    q = p - P1[a:b]
                    rs += float((-(wr * u.real * q.real) - wi * u.imag * q.imag).sum())
                    S += (torch.fft.fft2(p) * _kernel(self.z[a:b], self.turns)).sum(0)
                d = torch.fft.ifft2(S).real
                f = float(0.5 * ((d - self.b) ** 2).sum())
                ratio = f / (before + lim1 + lim2 / (2.0 * t))
                if 0.0 <= ratio <= 1.0 or attempt == 2:
                    break
                t *= 0.5
            a0 = 1.0 if rs > 0 else alpha
            alpha = (1.0 + math.sqrt(1.0 + 4.0 * a0 * a0)) / 2.0
            beta = (a0 - 1.0) / alpha
            P0, P1, P2 = P1, P2, P0
            dx = d + beta * (d - d0)
            d0 = d
            r = dx - self.b
            before = float(0.5 * (r * r).sum())
            if record:
                x = lambda a, b: P1[a:b] + beta * (P1[a:b] - P0[a:b])  # noqa: E731
                track.append(self.objective(x, r))
        x = lambda a, b: P1[a:b] + beta * (P1[a:b] - P0[a:b])  # noqa: E731
        f = self.objective(x, r)
        for a, b in self.parts:
            P2[a:b] = x(a, b)
        return f, dx, track, P2


def _conv(X, Wk, b):
    """3 x 3 x 3 convolution of X [D, H, W, C], plane by plane, zero outside."""
    D, H, W, C = X.shape
    Xp = torch.nn.functional.pad(X, (0, 0, 1, 1, 1, 1, 1, 1))
    out = []
    step = max(1, int(4e6 / (H * W)))
    for a in range(0, D, step):
        n = min(step, D - a)
        y = b
        for k in range(27):
            dz, dy, dx = k // 9, (k // 3) % 3, k % 3
            y = y + Xp[a + dz:a + dz + n, dy:dy + H, dx:dx + W].reshape(-1, C) @ Wk[:, k, :].T
        out.append(y.view(n, H, W, -1))
    return torch.cat(out) if len(out) > 1 else out[0]


def _unpack(params):
    off, layers = 0, []
    for ci, co, _ in LAYERS:
        n = co * 27 * ci
        layers.append((params[off:off + n].view(co, 27, ci), params[off + n:off + n + co]))
        off += n + co
    return layers, params[off:off + 18]


def _network_forward(params, xbp):
    layers, head = _unpack(params)
    conv = lambda i, X: torch.relu(_conv(X, *layers[i]))  # noqa: E731

    def pool(X):
        D, H, W, C = X.shape
        return X.view(D // 2, 2, H // 2, 2, W // 2, 2, C).mean(dim=(1, 3, 5))

    def up(X):
        return X.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    mag = xbp.abs()
    X = torch.zeros(xbp.shape + (16,), dtype=torch.float64, device=DEV)
    X[..., 0] = mag / (mag * mag).mean().sqrt()
    s1 = conv(1, conv(0, X))
    s2 = conv(3, conv(2, pool(s1)))
    u = conv(5, conv(4, pool(s2)))
    u = conv(7, conv(6, torch.cat([up(u), s2], -1)))
    u = conv(9, conv(8, torch.cat([up(u), s1], -1)))
    gain = torch.sigmoid(u @ head[:16] + head[16])
    return gain * head[17] * xbp


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        W, H = case["width"], case["height"]
        z = _planes(case["z0"], case["dz"], case["nz"])
        frame = _camera_frame(W, H, z, _turns(W, H, case["dx"], case["lam"]), seed)
        e = _Exact(case, _hologram(frame, case["pad"]))
        f, d, track, x = e.solve(case["iterations"], case["record"])
        out = {"objective": f, "estimate": d, "volume": torch.view_as_real(x) if case["storage"] == "f16" else x}
        if case["record"]:
            out["trajectory"] = np.array(track)
        return out
    if kind == "batch":
        W, H = case["width"], case["height"]
        z, turns = _planes(1000.0, 2.0, case["nz"]), _turns(W, H, 1.1, 0.632)
        fs, xs = [], []
        for i in range(case["frames"]):
            b = _hologram(_camera_frame(W, H, z, turns, 1000 * seed + i), 0).float().double()
            f, _, _, x = _Exact(case, b).solve(case["iterations"])
            fs.append(f)
            xs.append(x)
        return {"objectives": np.array(fs), "volumes": xs}
    if kind == "operators":
        g = _generator(seed)
        W, H, nz = case["width"], case["height"], case["nz"]
        volume = torch.randn((nz, H, W), generator=g, device=DEV, dtype=torch.complex64)
        residual = torch.randn((H, W), generator=g, device=DEV)
        z, turns = _planes(1000.0, case["dz"], nz), _turns(W, H, 1.1, 0.632)
        S = torch.zeros((H, W), dtype=torch.complex128, device=DEV)
        R = torch.fft.fft2(residual.double())
        G = torch.empty((nz, H, W), dtype=torch.complex128, device=DEV)
        step = _chunk(W, H)
        for a in range(0, nz, step):
            k = _kernel(z[a:a + step], turns)
            S += (torch.fft.fft2(volume[a:a + step].to(torch.complex128)) * k).sum(0)
            G[a:a + step] = torch.fft.ifft2(R * k.conj())
        return {"hologram": torch.fft.ifft2(S).real, "gradient": G}
    if kind in ("predict", "gradients"):
        weights = _Network({**case, "width": 4, "height": 4})  # for the packaged weights alone
        params = torch.from_numpy(weights.net.params()).to(DEV).double()
        xbp = _back_propagated(case, seed)
        if kind == "predict":
            return _network_forward(params, xbp.to(torch.complex128))
        xstar = _target(xbp).to(torch.complex128)
        params.requires_grad_(True)
        e = _network_forward(params, xbp.to(torch.complex128)) - xstar
        loss = (e.real ** 2 + e.imag ** 2).sum() / (xstar.abs() ** 2).sum()
        loss.backward()
        return {"loss": float(loss), "gradients": params.grad}
    return None  # segmentation gives whole numbers and FP32 sums in a fixed order
