"""The frames and calls that users of this library make, as cases to time.

Every case goes through a public entry point of contour3d_gb300.lib.Library:

  device   render_pack: fields resident in HBM into a device image (an in-situ
           solver's frame)
  execute  contour3d_execute, the drop-in call: host field in, ppm file out
  host     contour3d_gb300_render: host field in, host image out
  batch    render_batch: many frames of fields of uneven shapes and types
  server   the served form: a stream of requests over resident fields
  offsets  cell_offsets_noalloc: per-cell triangle offsets without allocation

Fields are sums of Fourier modes (|k| from 1 to kmax, amplitude |k|^-power) or
of Gaussian blobs on the unit cube, as in bench.py, workloads.py and the
tests, made here from the seed with one matrix product per z-plane block.
Every result is bytes or whole numbers: none is a floating-point value.
"""
import ctypes
import os
import shutil
import tempfile
import weakref

import numpy as np
import torch

import contour3d_gb300
from contour3d_gb300 import _abi, workloads

CAM, CENTRE = (2.5, 2.0, 1.5), (0.5, 0.5, 0.5)
# levels in units of the Fourier field's standard deviation, and of a blob field's unit height
MODE_LEVELS = {1: (0.25,), 2: (-0.5, 0.5), 3: (-0.5, 0.0, 0.5), 4: (-1.0, -0.5, 0.5, 1.0)}
BLOB_LEVELS = {1: (0.5,), 2: (0.4, 0.6), 3: (0.3, 0.5, 0.7), 4: (0.3, 0.45, 0.6, 0.75)}


def _case(kind, nx, ny, nz, dtype="f64", field="modes", levels=1, width=1280, height=720, modes=64, kmax=16,
          power=5.0 / 6.0, lines=False, converter="identity"):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, field=field, levels=levels, width=width, height=height,
                modes=modes, kmax=kmax, power=power, lines=lines, converter=converter)


def listed():
    return [
        # the smallest scene of the tests with its box drawn: a preview, bound by latency and launches
        dict(_case("device", 28, 20, 24, field="blobs", modes=6, width=160, height=120, lines=True),
             name="device_28x20x24_f64"),
        # one surface of a coarse double field (the reference's example size) on a square image
        dict(_case("device", 128, 128, 128, field="blobs", modes=8, width=1024, height=1024),
             name="device_128_f64_blobs"),
        # a single-precision solver's frame as the served stream draws it
        dict(_case("device", 192, 192, 192, "f32", levels=2, modes=32, kmax=12), name="device_192_f32_2lv"),
        # uneven axes whose rows are not a multiple of 16 bytes
        dict(_case("device", 313, 269, 311, levels=3, width=1024, height=1024), name="device_313x269x311_f64_3lv"),
        # the benchmark's frame: a resolved double field, two surfaces, full HD
        dict(_case("device", 512, 512, 512, levels=2, width=1920, height=1080), name="device_512_f64_2lv"),
        # the largest: a single-precision field that takes many slabs, four surfaces, 4K
        dict(_case("device", 1536, 1536, 1536, "f32", levels=4, width=3840, height=2160, modes=256, kmax=48,
                   power=11.0 / 6.0), name="device_1536_f32_4lv"),
        # the drop-in call on the benchmark's field: upload, render, file
        dict(_case("execute", 512, 512, 512, levels=2, width=1920, height=1080), name="execute_512_f64_2lv"),
        # a small drop-in frame in memory, pageable field of odd size, box lines
        dict(_case("host", 131, 97, 119, levels=2, width=800, height=600, modes=32, kmax=8, lines=True),
             name="host_131x97x119_f64_2lv"),
        # curvilinear coordinates: the caller's converter, all shading in double precision
        dict(_case("host", 72, 64, 80, levels=1, width=800, height=600, modes=16, kmax=4, converter="warp"),
             name="host_72x64x80_warp"),
        # a post-processing batch: 16 fields of 64 to 384 nodes a side, f64 and f32 in turn, 1 to 4 levels
        dict(kind="batch", frames=16, nmin=64, nmax=384, workers=8, width=1024, height=1024, name="batch_16"),
        # a visualisation service: requests with cameras and levels of their own over resident fields
        dict(kind="server", requests=24, nmin=96, nmax=384, slots=8, width=1280, height=720, name="server_24"),
        # offsets for a solver that extracts geometry itself
        dict(_case("offsets", 389, 301, 257, "f32"), name="offsets_389x301x257_f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["device"] * 5 + ["host", "host", "execute", "batch", "server", "offsets"])
    width, height = rng.choice([(320, 240), (640, 480), (800, 600), (1024, 1024), (1280, 720), (1920, 1080),
                                (1001, 777)])
    if kind == "batch":
        return dict(kind=kind, frames=rng.randint(3, 24), nmin=rng.randint(32, 64), nmax=_log_int(rng, 96, 384),
                    workers=rng.choice([4, 6, 8]), width=width, height=height)
    if kind == "server":
        return dict(kind=kind, requests=rng.randint(4, 32), nmin=rng.randint(48, 96), nmax=_log_int(rng, 128, 384),
                    slots=rng.choice([4, 8]), width=width, height=height)
    # axes around one size, odd and uneven ones among them
    n = _log_int(rng, 24, 768 if kind == "device" else 384)
    nx, ny, nz = (max(8, int(round(n * rng.uniform(0.7, 1.3)))) for _ in range(3))
    if rng.random() < 0.4:
        nx = ny = nz = n
    dtype = rng.choice(["f64", "f32"]) if kind in ("device", "offsets") else "f64"
    field = rng.choice(["modes", "modes", "blobs"])
    modes = rng.randint(4, 32) if field == "blobs" else rng.choice([16, 32, 64])
    kmax = min(16, max(2, n // 12))
    converter = "identity"
    if kind == "host" and rng.random() < 0.4:
        converter = "warp"
        nx, ny, nz = (max(8, min(a, 96)) for a in (nx, ny, nz))
    return _case(kind, nx, ny, nz, dtype, field, rng.randint(1, 4), width, height, modes, kmax,
                 lines=rng.random() < 0.3, converter=converter)


# ---- inputs -------------------------------------------------------------

def _axis(n, dtype):
    return torch.arange(n, dtype=dtype, device="cuda") / (n - 1)


def _planes(factors, shape, dtype):
    """sum over m of z[m, k] y[m, j] x[m, i] for each (x, y, z) of factors, by blocks of z-planes."""
    nz, ny, nx = shape
    out = torch.empty(shape, dtype=dtype, device="cuda")
    step = max(1, (1 << 25) // (ny * sum(f[0].shape[0] for f in factors)))
    x = torch.cat([f[0] for f in factors])
    for k in range(0, nz, step):
        zy = torch.cat([f[2][:, k:k + step, None] * f[1][:, None, :] for f in factors])
        torch.matmul(zy.reshape(zy.shape[0], -1).T, x, out=out[k:k + step].view(-1, nx))
    return out


def _modes(shape, dtype, nmodes, kmax, power, rng):
    d = rng.standard_normal((nmodes, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    kv = np.rint(d * np.maximum(1.0, kmax * np.cbrt(rng.random((nmodes, 1)))))  # uniform in the ball
    kv[np.abs(kv).sum(axis=1) == 0] = (1, 0, 0)
    amp = np.linalg.norm(kv, axis=1) ** -power
    phase = rng.random(nmodes)
    re, im = [], []
    for a, n in enumerate(reversed(shape)):  # x, y, z
        turns = torch.from_numpy(kv[:, a:a + 1]).cuda() * _axis(n, torch.float64)
        if a == 2:
            turns = turns + torch.from_numpy(phase[:, None]).cuda()
        w = torch.from_numpy(amp[:, None]).cuda() if a == 0 else 1.0
        re.append((w * torch.cos(2 * np.pi * turns)).to(dtype))
        im.append((w * torch.sin(2 * np.pi * turns)).to(dtype))
    # the real part of the product of three phases
    terms = [(re[0], re[1], re[2]), (-re[0], im[1], im[2]), (-im[0], re[1], im[2]), (-im[0], im[1], re[2])]
    return _planes(terms, shape, dtype), float(np.sqrt((amp ** 2).sum() / 2))


def _blobs(shape, dtype, nblobs, rng):
    centre, size = rng.uniform(0.15, 0.85, (nblobs, 3)), rng.uniform(0.06, 0.18, nblobs)
    f = []
    for a, n in enumerate(reversed(shape)):
        q = (_axis(n, torch.float64) - torch.from_numpy(centre[:, a:a + 1]).cuda()) / \
            torch.from_numpy(size[:, None]).cuda()
        f.append(torch.exp(-0.5 * q * q).to(dtype))
    return _planes([tuple(f)], shape, dtype)


def _field(case, rng):
    """The device field and its levels."""
    shape = (case["nz"], case["ny"], case["nx"])
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    if case["field"] == "blobs":
        return _blobs(shape, dtype, case["modes"], rng), list(BLOB_LEVELS[case["levels"]])
    f, std = _modes(shape, dtype, case["modes"], case["kmax"], case["power"], rng)
    return f, [q * std for q in MODE_LEVELS[case["levels"]]]


def _pack(lib, field, levels, camera, width, height, lines=False):
    rgb = torch.empty(height, width, 3, dtype=torch.uint8, device="cuda")
    nz, ny, nx = field.shape
    grids = [_abi.unit_grid(n) for n in (nx, ny, nz)]
    fl = [(field.data_ptr(), 0 if field.dtype == torch.float64 else 1, (nx, ny, nz), grids, lv, col)
          for lv, col in zip(levels, workloads.PALETTE)]
    scene = _abi.make_scene(camera, CENTRE, width, height)
    if lines:
        scene.lines = _abi.cube_edges(nitems=5)
    return lib.frame(scene, fl, rgb.data_ptr()), rgb


class _State:
    pass


def _mixed(case, n, rng, shared):
    """Fields of uneven shapes, and per frame one of them with levels and a camera of its own."""
    fields = []
    for q in range(shared or n):
        shape = rng.integers(case["nmin"], case["nmax"] + 1, size=3)
        c = dict(nx=int(shape[2]), ny=int(shape[1]), nz=int(shape[0]), dtype="f64" if q % 2 == 0 else "f32",
                 field="blobs" if not shared and rng.random() < 0.5 else "modes", levels=1, modes=32,
                 kmax=max(2, min(12, case["nmin"] // 6)), power=5.0 / 6.0)
        fields.append(_field(c, rng)[0])
    frames = []
    for q in range(n):
        f = fields[int(rng.integers(len(fields)))] if shared else fields[q]
        levels = workloads.quantile_levels(f, rng, int(rng.integers(1, 4 if shared else 5)))
        frames.append((f, levels, workloads.random_camera(rng)))
    return fields, frames


def prepare(case, seed):
    lib = contour3d_gb300.load()
    rng = np.random.default_rng(seed)
    s = _State()
    s.lib, s.kind = lib, case["kind"]
    if s.kind in ("batch", "server"):
        n = case["frames"] if s.kind == "batch" else case["requests"]
        s.fields, frames = _mixed(case, n, rng, 0 if s.kind == "batch" else 6)
        made = [_pack(lib, f, lv, cam, case["width"], case["height"]) for f, lv, cam in frames]
        s.packs, s.images = [m[0] for m in made], [m[1] for m in made]
        if s.kind == "batch":
            s.workers = case["workers"]
        else:
            s.server = lib.server(case["slots"])
            weakref.finalize(s, s.server.close)
    else:
        field, levels = _field(case, rng)
        if s.kind == "device":
            s.field = field
            s.pack, s.image = _pack(lib, field, levels, CAM, case["width"], case["height"], case["lines"])
        elif s.kind == "offsets":
            s.field, s.level = field, levels[0]
            s.dtype = 0 if field.dtype == torch.float64 else 1
            s.sizes = (ctypes.c_size_t * 3)(case["nx"], case["ny"], case["nz"])
            cells = (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] - 1)
            s.offsets = torch.empty(cells + 1, dtype=torch.int32, device="cuda")
            s.total = torch.empty(1, dtype=torch.int64, device="cuda")
        else:
            host = torch.empty(field.shape, dtype=torch.float64, pin_memory=s.kind == "execute")
            host.copy_(field)
            s.host, s.scene = host, _abi.make_scene(CAM, CENTRE, case["width"], case["height"])
            s.scene.contours = [_abi.Contour(host.numpy(), lv, col, converter=case["converter"])
                                for lv, col in zip(levels, workloads.PALETTE)]
            if case["lines"]:
                s.scene.lines = _abi.cube_edges(nitems=5)
            if s.kind == "execute":
                d = tempfile.mkdtemp(prefix="contour3d_")
                s.path = os.path.join(d, "frame.ppm")
                weakref.finalize(s, shutil.rmtree, d, True)
    torch.cuda.synchronize()  # the library works on streams of its own
    return s


def run(s):
    lib = s.lib
    if s.kind == "device":
        if lib.render_pack(s.pack) != 0:
            raise RuntimeError("the frame failed")
        return s.image
    if s.kind == "execute":
        if lib.execute(s.scene, s.path) != 0:
            raise RuntimeError("the call failed")
        return np.memmap(s.path, dtype=np.uint8, mode="r")  # the file, mapped: read by whoever compares it
    if s.kind == "host":
        return lib.render(s.scene)
    if s.kind == "batch":
        lib.render_batch(s.packs, s.workers)
        return s.images
    if s.kind == "server":
        tickets = [s.server.submit(p) for p in s.packs]
        for t in tickets:
            s.server.wait(t)
        return s.images
    if lib.lib.contour3d_gb300_cell_offsets_noalloc(s.field.data_ptr(), s.dtype, s.sizes, s.level,
                                                    s.offsets.data_ptr(), s.total.data_ptr(), None) != 0:
        raise RuntimeError("the offsets failed")
    return {"offsets": s.offsets, "total": s.total}


def work(case):
    """Every field read once (by all of its levels together) and every result written once; one comparison
    per node and level."""
    if case["kind"] in ("batch", "server"):
        n = case["frames"] if case["kind"] == "batch" else case["requests"]
        nodes = n * ((case["nmin"] + case["nmax"]) / 2) ** 3  # the mean of the drawn shapes
        return {"bytes": 6 * nodes + 3 * n * case["width"] * case["height"], "flops": 2 * nodes}
    nodes = case["nx"] * case["ny"] * case["nz"]
    field = nodes * (8 if case["dtype"] == "f64" else 4)
    if case["kind"] == "offsets":
        return {"bytes": field + 4 * (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] - 1), "flops": nodes}
    return {"bytes": field + 3 * case["width"] * case["height"], "flops": nodes * case["levels"]}
