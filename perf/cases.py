"""The calls that the performance of this library is measured on, through its public Python API.

A case is a dict of plain values (``op``, sizes, options). ``listed`` gives the standing cases, ``draw``
one more of the same ranges, ``prepare`` what a program has in hand before the call, ``run`` one pass,
``work`` the bytes and operations a pass cannot do without, ``tolerance`` what two correct
implementations in single precision may differ by, and ``exact`` the outputs in double precision from
plain torch.

Values follow the library's synthetic workloads: volumes are spectra of white noise times
1 / max(|f|, 1/64), slices of white noise times exp(-B f^2 / 4) with B = 100, orientations uniform on SO(3).

Whether a sample lies inside the cutoff is decided, by definition, on single-precision coordinates
(lattice points lie exactly on the cutoff sphere, where rounding decides), so ``exact`` takes that one
decision as the definition does and everything else in double precision.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from noa_b200 import fourier_project as fp
from noa_b200.batch import ExtractBatch, ExtractRequest
from noa_b200.reconstruct import reconstruct
from noa_b200.synthetic import quaternion_to_matrix, random_quaternions

WINDOW_SIZE = {"linear": 2, "cubic": 4, "lanczos4": 4, "lanczos6": 6, "lanczos8": 8}

# What each option is when a case does not name it. `size`: the slices' box (0: the volume's). `kind`:
# c2c complex to complex, c2r complex to |z|^2, r2r real. `half_width`: the insertions' windowed-sinc
# half-width in voxels (1: the default window). `w_width`: the extraction's w-window, in z samples each
# side (1: none). `weights`: with weight arrays on both sides where the call takes them.
DEFAULTS = {"remap": "hc2h", "interp": "linear", "cutoff": 0.5, "size": 0, "kind": "c2c", "rotation": "matrix",
            "scaling": False, "weights": False, "half_width": 1.0, "w_width": 1.0, "outputs": 0}


def listed() -> list[dict]:
    return [
        # One call of a small box, as a refinement makes at its coarsest level: latency and launches.
        {"name": "extract_64", "op": "extract", "n": 64, "slices": 64},
        # A few projections of one reference: too few to amortise any preparation of the volume.
        {"name": "extract_few_200", "op": "extract", "n": 200, "slices": 150},
        # The headline workload: a full set of projections of a 256^3 volume.
        {"name": "extract_256", "op": "extract", "n": 256, "slices": 4096},
        # Projections with a thickness (w-windowed sinc, seven z samples per pixel) and their weights.
        {"name": "extract_w_256", "op": "extract", "n": 256, "slices": 1000, "w_width": 4.0, "weights": True},
        # High-quality projections: LANCZOS8, 512 taps per pixel.
        {"name": "extract_lanczos8_192", "op": "extract", "n": 192, "slices": 500, "interp": "lanczos8"},
        # Back-projection of the same small box: trilinear insertion with weights.
        {"name": "rasterize_64", "op": "rasterize", "n": 64, "slices": 64, "remap": "h2hc", "weights": True},
        # The headline workload's insertion: a full set of slices into 256^3 with weights.
        {"name": "rasterize_256", "op": "rasterize", "n": 256, "slices": 4096, "remap": "h2hc", "weights": True},
        # Windowed-sinc insertion into a large box (half-width 6 voxels): the deterministic gather form.
        {"name": "insert_512", "op": "insert", "n": 512, "slices": 400, "remap": "hc2hc", "weights": True,
         "half_width": 6.0},
        # The same insertion in its atomic scatter form, at an ordinary size.
        {"name": "scatter_256", "op": "scatter", "n": 256, "slices": 500, "remap": "hc2hc", "weights": True,
         "half_width": 6.0},
        # Each projection predicted from all the other images, without a volume in between.
        {"name": "insert_extract_256", "op": "insert_extract", "n": 256, "slices": 2000, "outputs": 64,
         "remap": "h2h", "weights": True},
        # Uneven requests over volumes of 128 to 384 as one captured batch (a multi-reference job).
        {"name": "batch_uneven_40", "op": "batch", "n": 384, "slices": 4000, "outputs": 40},
        # From the inserted grids to the real-space map: normalisation, inverse FFT, gridding correction.
        {"name": "reconstruct_250", "op": "reconstruct", "n": 250, "slices": 1},
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["extract", "extract", "extract", "rasterize", "rasterize", "insert", "scatter", "insert_extract",
                     "batch", "reconstruct"])
    c = {"op": op, "remap": rng.choice(["h2h", "h2hc", "hc2h", "hc2hc"])}
    if op == "extract":
        c["interp"] = rng.choice(["linear", "linear", "linear", "cubic", "lanczos6", "lanczos8"])
        c["n"] = log_int(32, 384 if c["interp"] == "linear" else 256)
        taps = WINDOW_SIZE[c["interp"]] ** 3
        pixels = c["n"] * (c["n"] // 2 + 1)
        # at most the pixels of 4096 slices of 256^2, an eighth of that per 64 taps for the wider windows
        c["slices"] = log_int(8, min(4096, max(9, int(135e6 / pixels / max(1, taps / 8)))))
        c["kind"] = rng.choice(["c2c", "c2c", "c2c", "c2r", "r2r"])
        c["weights"] = rng.random() < 0.3
        if c["interp"] == "linear" and c["slices"] <= 1000 and rng.random() < 0.25:
            c["w_width"] = float(rng.randint(2, 4))
    elif op == "rasterize":
        c["n"] = log_int(32, 384)
        c["slices"] = log_int(8, min(4096, int(135e6 / (c["n"] * (c["n"] // 2 + 1)))))
        c["kind"] = rng.choice(["c2c", "c2c", "c2c", "r2r"])
        c["weights"] = rng.random() < 0.8
    elif op in ("insert", "scatter"):
        c["n"] = log_int(48, 320)
        c["slices"] = log_int(8, min(1000, int(40e6 / (c["n"] * c["n"]))))
        c["half_width"] = rng.choice([1.0, 2.0, 4.0, 6.0])
        c["weights"] = rng.random() < 0.8
    elif op == "insert_extract":
        c["n"] = log_int(48, 256)
        c["slices"] = log_int(16, 2000)
        c["outputs"] = log_int(4, 64)
        c["weights"] = rng.random() < 0.8
    elif op == "batch":
        c["n"] = log_int(96, 384)
        c["slices"] = log_int(100, 4000)
        c["outputs"] = log_int(4, 60)
        return c
    else:
        c["n"] = log_int(48, 250)
        c["slices"] = 1
        c["remap"] = rng.choice(["hc2h", "h2h"])
        return c
    # Even sizes serve most boxes, odd ones come from cropped data.
    if rng.random() < 0.3 and op != "reconstruct":
        c["size"] = max(16, int(c["n"] * rng.uniform(0.75, 1.0)))
    c["cutoff"] = rng.choice([0.5, 0.5, 0.45, 0.3])
    c["rotation"] = rng.choice(["matrix", "matrix", "quaternion"])
    c["scaling"] = rng.random() < 0.2
    return c


# ---------------------------------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------------------------------
def _full(case: dict) -> dict:
    return {**DEFAULTS, **case}


def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _indices(n: int, centered: bool):
    i = torch.arange(n, device="cuda")
    return i - n // 2 if centered else torch.where(i < (n + 1) // 2, i, i - n)


def _norm(shape: tuple, centered: bool):
    """|fftfreq| over an rfft grid of the logical `shape` (the last dimension is the half one)."""
    total = None
    for axis, n in enumerate(shape):
        last = axis == len(shape) - 1
        f = (torch.arange(n // 2 + 1, device="cuda") if last else _indices(n, centered)).float() / n
        f = f.square().reshape([-1 if k == axis else 1 for k in range(len(shape))])
        total = f if total is None else total + f
    return total.sqrt()


def _spectra(g, shape: tuple, centered: bool, envelope, real: bool):
    """rfft of white noise (unit variance per frequency, Hermitian as spectra of real data are) over the
    dimensions of `shape` but the first, times `envelope`; or its real part."""
    axes = tuple(range(1, len(shape)))
    v = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"), dim=axes, norm="ortho")
    if centered:
        v = torch.fft.fftshift(v, dim=axes[:-1])
    v.mul_(envelope)
    return v.real.contiguous() if real else v.contiguous()


def _volume(g, n: int, centered: bool, real: bool):
    return _spectra(g, (1, n, n, n), centered, 1 / _norm((n, n, n), centered).clamp_min(1 / 64), real)


def _slices(g, count: int, n: int, centered: bool, real: bool):
    envelope = torch.exp(-25 * _norm((n, n), centered).square())
    out = torch.empty((count, 1, n, n // 2 + 1), dtype=torch.float32 if real else torch.complex64, device="cuda")
    for b in range(0, count, 512):
        out[b:b + 512, 0] = _spectra(g, (min(512, count - b), n, n), centered, envelope, real)
    return out


def _rotations(count: int, seed: int, kind: str):
    q = random_quaternions(count, seed=seed)
    if kind == "quaternion":
        return torch.from_numpy(q.astype(np.float32)).cuda()
    return fp.pack_rotations(torch.from_numpy(quaternion_to_matrix(q).astype(np.float32)).cuda())


def _scalings(g, count: int):
    """Small anisotropic magnification corrections, one 2x2 matrix per slice."""
    eye = torch.eye(2, device="cuda").expand(count, 2, 2)
    return (eye + 0.02 * torch.randn((count, 2, 2), generator=g, device="cuda")).contiguous()


def _boxes(c: dict, seed: int) -> list[tuple]:
    """Of a batch: (volume, box, slices) of each request; four volumes of 1/3 to all of the largest box."""
    rng = np.random.default_rng([c["n"], c["slices"], c["outputs"]])
    sizes = [max(16, int(c["n"] * f)) for f in (1 / 3, 1 / 2, 2 / 3, 1)]
    counts = rng.lognormal(0, 0.5, c["outputs"])
    counts = np.maximum(1, counts / counts.sum() * c["slices"]).astype(int)
    return [(i % 4, sizes[i % 4], int(k)) for i, k in enumerate(counts)]


def prepare(case: dict, seed: int) -> dict:
    c = _full(case)
    g, op, n = _generator(seed), c["op"], c["n"]
    size = c["size"] or n
    real = c["kind"] == "r2r"
    out_type = torch.complex64 if c["kind"] == "c2c" else torch.float32
    in_centered, out_centered = c["remap"].startswith("hc"), c["remap"].endswith("hc")
    state = {"case": c}
    if op == "batch":
        volumes = [_volume(g, max(16, int(n * f)), in_centered, False) for f in (1 / 3, 1 / 2, 2 / 3, 1)]
        requests = []
        for k, (which, box, count) in enumerate(_boxes(c, seed)):
            out = torch.zeros((count, 1, box, box // 2 + 1), dtype=torch.complex64, device="cuda")
            requests.append(ExtractRequest(volume=volumes[which], volume_shape=(1, box, box, box), slice=out,
                                           slice_shape=(count, 1, box, box),
                                           fwd_rotation=_rotations(count, seed + 100 + k, "matrix")))
        state.update(requests=requests, batch=ExtractBatch(c["remap"], requests))
        return state
    if op == "reconstruct":
        weights = torch.rand((1, n, n, n // 2 + 1), generator=g, device="cuda").mul_(40)
        state.update(values=_volume(g, n, in_centered, False).mul_(weights), weights=weights)
        return state
    count = c["slices"]
    state["rotation"] = _rotations(count, seed + 1, c["rotation"])
    state["scaling"] = _scalings(g, count) if c["scaling"] else None
    volume_shape, slice_shape = (1, n, n, n), (count, 1, size, size)
    if op == "extract":
        state["input"] = _volume(g, n, in_centered, real)
        state["output"] = torch.zeros((count, 1, size, size // 2 + 1), dtype=out_type, device="cuda")
        state["output_weight"] = (torch.zeros(state["output"].shape, device="cuda") if c["weights"] else None)
        state["shapes"] = (volume_shape, slice_shape)
        return state
    state["input"] = _slices(g, count, size, in_centered, real)
    state["input_weight"] = None
    if op == "insert_extract":
        made = c["outputs"]
        state["output"] = torch.zeros((made, 1, size, size // 2 + 1), dtype=out_type, device="cuda")
        state["rotation2"] = _rotations(made, seed + 2, c["rotation"])
        state["shapes"] = (slice_shape, (made, 1, size, size))
    else:
        state["output"] = torch.zeros((1, n, n, n // 2 + 1), dtype=out_type, device="cuda")
        state["shapes"] = (slice_shape, volume_shape)
    state["output_weight"] = torch.zeros(state["output"].shape, device="cuda") if c["weights"] else None
    return state


def _insertion_window(c: dict) -> fp.WindowedSinc | None:
    if c["half_width"] <= 1:
        return None
    return fp.WindowedSinc(1 / c["n"], c["half_width"] / c["n"])


# ---------------------------------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------------------------------
def run(state: dict):
    c = state["case"]
    op = c["op"]
    if op == "batch":
        state["batch"].run()
        return [r.slice for r in state["requests"]]
    if op == "reconstruct":
        return reconstruct(state["values"], state["weights"], (1, c["n"], c["n"], c["n"]),
                           centered=c["remap"].startswith("hc"))
    shape_in, shape_out = state["shapes"]
    out, out_w = state["output"], state["output_weight"]
    if op == "extract":
        w = fp.WindowedSinc(1 / c["n"], c["w_width"] / c["n"]) if c["w_width"] > 1 else None
        fp.extract_central_slices_3d(c["remap"], state["input"], None, shape_in, out, out_w, shape_out,
                                     state["scaling"], state["rotation"], interp=c["interp"], w_windowed_sinc=w,
                                     fftfreq_cutoff=c["cutoff"])
    elif op == "rasterize":
        fp.rasterize_central_slices_3d(c["remap"], state["input"], None, shape_in, out, out_w, shape_out,
                                       state["scaling"], state["rotation"], fftfreq_cutoff=c["cutoff"])
    elif op in ("insert", "scatter"):
        call = fp.insert_central_slices_3d if op == "insert" else fp.insert_central_slices_3d_scatter
        call(c["remap"], state["input"], None, shape_in, out, out_w, shape_out, state["scaling"],
             state["rotation"], interp=c["interp"], windowed_sinc=_insertion_window(c), fftfreq_cutoff=c["cutoff"])
    else:
        fp.insert_and_extract_central_slices_3d(c["remap"], state["input"], None, shape_in, out, out_w, shape_out,
                                                state["scaling"], state["rotation"], None, state["rotation2"],
                                                interp=c["interp"], fftfreq_cutoff=c["cutoff"])
    return (out, out_w) if out_w is not None else out


def work(case: dict) -> dict:
    """Bytes: every input read once, every output written once (insertions also read their grids).
    Operations: of the interpolation sums (and window evaluations) of the samples inside the cutoff."""
    c = _full(case)
    n, size = c["n"], c["size"] or c["n"]
    voxels = n * n * (n // 2 + 1)
    read = 4 if c["kind"] == "r2r" else 8
    wrote = 8 if c["kind"] == "c2c" else 4
    inside = math.pi * (c["cutoff"] * size) ** 2 / 2          # pixels of one slice within the cutoff
    pixels = c["slices"] * (size * (size // 2 + 1))
    weight = 4 if c["weights"] else 0
    op = c["op"]
    if op == "batch":
        boxes = _boxes(c, 0)
        pix = sum(k * b * (b // 2 + 1) for _, b, k in boxes)
        vox = sum(b * b * (b // 2 + 1) for b in {w: b for w, b, _ in boxes}.values())
        return {"bytes": 8 * (pix + vox), "flops": 32 * 0.78 * pix}
    if op == "reconstruct":
        return {"bytes": 12 * voxels + 4 * n ** 3, "flops": 2.5 * n ** 3 * math.log2(n ** 3)}
    if op == "extract":
        samples = max(1, 2 * math.ceil(c["w_width"]) - 1)
        taps = WINDOW_SIZE[c["interp"]] ** 3 * samples
        return {"bytes": read * voxels + (wrote + weight) * pixels + 48 * c["slices"],
                "flops": 4 * taps * inside * c["slices"]}
    if op == "rasterize":
        return {"bytes": read * pixels + 2 * (wrote + weight) * voxels + 48 * c["slices"],
                "flops": 8 * 6 * inside * c["slices"]}
    if op == "insert_extract":
        made = c["outputs"]
        # a slice passes within one voxel of a pixel of radius r with probability 1 / r (r in voxels)
        pairs = made * c["slices"] * math.pi * c["cutoff"] * size
        return {"bytes": read * pixels + (wrote + weight) * made * size * (size // 2 + 1) + 48 * (c["slices"] + made),
                "flops": 40 * pairs}
    pairs = c["slices"] * math.pi * (c["cutoff"] * n) ** 2 / 2 * 2 * c["half_width"]
    return {"bytes": read * pixels + 2 * (wrote + weight) * voxels + 48 * c["slices"], "flops": 40 * pairs}


def tolerance(case: dict):
    """Single-precision coordinates of up to a few hundred samples are uncertain by about 1e-5 of a
    sample, which the interpolation of noise turns into a relative error of 1e-6 to 6e-6 (measured
    against double precision over these ranges); sums in another order add 1e-7."""
    return {"rel": 2e-5}


# ---------------------------------------------------------------------------------------------------
# Double precision, from the definitions.
# ---------------------------------------------------------------------------------------------------
def _parts(rotation, dtype, dims: int):
    """The numbers of packed matrices or quaternions (z, y, x, w), each to broadcast over `dims` dimensions."""
    return [p.to(dtype).reshape(p.shape + (1,) * dims) for p in rotation.unbind(-1)]


def _rotate(parts, v):
    """`v`: three broadcastable tensors (z, y, x). Products and sums in the order of the definition, so
    that in single precision they round as it does."""
    if len(parts) == 12:
        m = parts
        return [(m[3 * r] * v[0] + m[3 * r + 1] * v[1]) + m[3 * r + 2] * v[2] for r in range(3)]
    z, y, x, w = parts
    v0, v1, v2 = v
    s0 = (w * v2 + y * v0) - z * v1
    s1 = (w * v1 + z * v2) - x * v0
    s2 = (w * v0 + x * v1) - y * v2
    return [v0 + 2 * (x * s1 - y * s0), v1 + 2 * (z * s0 - x * s2), v2 + 2 * (y * s2 - z * s1)]


def _scale(m, f0, f1):
    """`m`: the four numbers of 2x2 matrices, or None."""
    if m is None:
        return f0, f1
    return m[0] * f0 + m[1] * f1, m[2] * f0 + m[3] * f1


def _over(i, n: int, dtype):
    """i / n, rounded once (a division by a Python number may be a product with its reciprocal)."""
    return i.to(dtype) / torch.full((), n, dtype=dtype, device="cuda")


def _slice_to_grid(size, centered, scaling, rotation, dtype):
    """3-D frequencies (z, y, x) of the pixels of some slices, each (slices, size, size // 2 + 1)."""
    f0 = _over(_indices(size, centered), size, dtype)[None, :, None]
    f1 = _over(torch.arange(size // 2 + 1, device="cuda"), size, dtype)[None, None, :]
    f0, f1 = torch.broadcast_tensors(f0, f1)
    f0, f1 = _scale(None if scaling is None else _parts(scaling.reshape(-1, 4), dtype, 2), f0, f1)
    return _rotate(_parts(rotation, dtype, 2), [torch.zeros_like(f0), f0, f1])


def _groups(count: int, size: int):
    """Ranges of slices of about two million pixels."""
    step = max(1, (2 << 20) // (size * (size // 2 + 1)))
    return [slice(b, min(b + step, count)) for b in range(0, count, step)]


def _inside(f, cutoff):
    return (f[0] * f[0] + f[1] * f[1]) + f[2] * f[2] <= torch.tensor(cutoff, dtype=torch.float32).square().item()


def _window(f, sinc, blackman):
    x = f * (math.pi / sinc)
    s = torch.where(x == 0, torch.ones_like(x), torch.sin(x) / torch.where(x == 0, torch.ones_like(x), x))
    b = f * (math.pi / blackman)
    return s * (0.42 + 0.5 * torch.cos(b) + 0.08 * torch.cos(2 * b))


def _tap_weights(t, interp):
    """Weights of the taps around a sample at fraction `t` past the tap before it, one per tap."""
    if interp == "linear":
        return [1 - t, t]
    size = WINDOW_SIZE[interp]
    if interp == "cubic":
        def near(d):
            return ((1.5 * d - 2.5) * d) * d + 1

        def far(d):
            return ((-0.5 * d + 2.5) * d - 4) * d + 2
        return [far(1 + t), near(t), near(1 - t), far(2 - t)]
    centre = size // 2 - 1
    ws = []
    for i in range(size):
        y = math.pi / 4 * (i - centre - t)
        at = y.abs() < 1e-12
        ws.append((-1) ** i * torch.where(at, torch.ones_like(y), torch.sin(y) / torch.where(at, torch.ones_like(y), y * y)))
    # on a tap (fraction 0 or 1) the sample is that tap
    total = sum(ws)
    out = []
    for i, w in enumerate(ws):
        w = w / total
        w = torch.where(t < 1e-7, torch.full_like(w, float(i == centre)), w)
        out.append(torch.where(t > 1 - 1e-7, torch.full_like(w, float(i == centre + 1)), w))
    return out


def _interpolate(grid, centered, sizes, q, interp):
    """Samples of the rfft `grid` (dimensions `sizes`, double precision) at `q`, in samples from DC."""
    early = WINDOW_SIZE[interp] <= 2
    flip = torch.zeros_like(q[-1], dtype=torch.bool)
    if early:
        flip = q[-1] < 0
        q = [torch.where(flip, -a, a) for a in q]
    base = [torch.floor(a) for a in q]
    ws = [_tap_weights(a - b, interp) for a, b in zip(q, base)]
    base = [b.long() for b in base]
    start = -((WINDOW_SIZE[interp] - 1) // 2)
    flat, total = grid.reshape(-1), 0
    dims = len(q)
    for tap in np.ndindex(*([WINDOW_SIZE[interp]] * dims)):
        at = [b + start + k for b, k in zip(base, tap)]
        weight = ws[0][tap[0]]
        for axis in range(1, dims):
            weight = weight * ws[axis][tap[axis]]
        mirrored = at[-1] < 0
        if not early:
            at = [torch.where(mirrored, -a, a) for a in at]
        good = (at[-1] >= 0) & (at[-1] <= sizes[-1] // 2)
        index = 0
        for a, n in zip(at[:-1], sizes[:-1]):
            good &= (a >= -(n // 2)) & (a <= (n - 1) // 2)
            index = index * n + (a + n // 2 if centered else torch.where(a < 0, a + n, a))
        index = index * (sizes[-1] // 2 + 1) + at[-1]
        v = flat[torch.where(good, index, 0)]
        if v.is_complex() and not early:
            v = torch.where(mirrored, v.conj(), v)
        total = total + torch.where(good, v * weight, torch.zeros_like(v))
    if total.is_complex():
        total = torch.where(flip, total.conj(), total)
    return total


def _double(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _exact_extract(c, volume, rotation, scaling, size, count):
    n = c["n"]
    in_centered, out_centered = c["remap"].startswith("hc"), c["remap"].endswith("hc")
    grid = _double(volume)
    values, weights = [], []
    steps = range(1) if c["w_width"] <= 1 else range(-(math.ceil(c["w_width"]) - 1), math.ceil(c["w_width"]))
    for b in _groups(count, size):
        sc = None if scaling is None else scaling[b]
        near = _slice_to_grid(size, out_centered, sc, rotation[b], torch.float32)
        f = _slice_to_grid(size, out_centered, sc, rotation[b], torch.float64)
        value, weight = 0, 0
        for w in steps:
            off = w / n
            keep = _inside([near[0] + torch.tensor(w / n, dtype=torch.float32).item(), near[1], near[2]], c["cutoff"])
            at = [(a + (off if k == 0 else 0)) * n for k, a in enumerate(f)]
            v = _interpolate(grid, in_centered, (n, n, n), at, c["interp"])
            if c["kind"] == "c2r":
                v = v.real.square() + v.imag.square()
            factor = keep.double()
            if c["w_width"] > 1:
                factor = factor * _window(torch.tensor(off, dtype=torch.float64, device="cuda"), 1 / n, c["w_width"] / n)
            value, weight = value + v * factor, weight + factor
        values.append(value)
        weights.append(weight)
    return torch.cat(values)[:, None], torch.cat(weights)[:, None]


def _exact_rasterize(c, slices, rotation, scaling, size):
    n = c["n"]
    wp = n // 2 + 1
    in_centered, out_centered = c["remap"].startswith("hc"), c["remap"].endswith("hc")
    out = torch.zeros(n * n * wp, dtype=_double(slices[:0]).dtype, device="cuda")
    out_w = torch.zeros(n * n * wp, dtype=torch.float64, device="cuda")

    def index_of(a):
        i = a + n // 2 if out_centered else torch.where(a < 0, a + n, a)
        return i, (i >= 0) & (i < n)

    def put(z, y, x, v, k):
        (iz, gz), (iy, gy) = index_of(z), index_of(y)
        good = gz & gy & (x >= 0) & (x < wp)
        at = torch.where(good, (iz * n + iy) * wp + x, 0)
        k = torch.where(good, k, torch.zeros_like(k))
        if v.is_complex():  # two real sums: complex atomics are slow
            torch.view_as_real(out)[:, 0].index_add_(0, at, v.real * k)
            torch.view_as_real(out)[:, 1].index_add_(0, at, v.imag * k)
        else:
            out.index_add_(0, at, v * k)
        out_w.index_add_(0, at, k)

    for b in _groups(slices.shape[0], size):
        sc = None if scaling is None else scaling[b]
        keep = _inside(_slice_to_grid(size, in_centered, sc, rotation[b], torch.float32), c["cutoff"])
        f = [a[keep] for a in _slice_to_grid(size, in_centered, sc, rotation[b], torch.float64)]
        v = _double(slices[b, 0])[keep]
        flip = f[2] < 0
        q = [torch.where(flip, -a, a) * n for a in f]
        if v.is_complex():
            v = torch.where(flip, -v, v)  # the sign changes, the value is not conjugated
        base = [torch.floor(a).long() for a in q]
        t = [a - o for a, o in zip(q, base)]
        plane = base[2] == 0
        for dz in range(2):
            for dy in range(2):
                k = (t[0] if dz else 1 - t[0]) * (t[1] if dy else 1 - t[1])
                for dx in range(2):
                    put(base[0] + dz, base[1] + dy, base[2] + dx, v, k * (t[2] if dx else 1 - t[2]))
                mirror = v[plane].conj() if v.is_complex() else v[plane]
                put(-(base[0] + dz)[plane], -(base[1] + dy)[plane], base[2][plane], mirror, (k * (1 - t[2]))[plane])
    shape = (1, n, n, wp)
    return out.reshape(shape), out_w.reshape(shape)


def _exact_insert(c, slices, rotation, scaling, size):
    n = c["n"]
    in_centered, out_centered = c["remap"].startswith("hc"), c["remap"].endswith("hc")
    sinc, blackman = 1 / n, max(c["half_width"], 1.0) / n
    slices = _double(slices)
    zy, x = _indices(n, out_centered), torch.arange(n // 2 + 1, device="cuda")
    single = [_over(zy, n, torch.float32)[:, None, None], _over(zy, n, torch.float32)[None, :, None],
              _over(x, n, torch.float32)[None, None, :]]
    inside = _inside(single, c["cutoff"]).reshape(-1).nonzero()[:, 0]
    iz, iy, ix = inside // (n * (n // 2 + 1)), inside // (n // 2 + 1) % n, inside % (n // 2 + 1)
    f = [zy.double()[iz] / n, zy.double()[iy] / n, x.double()[ix] / n]
    out = torch.zeros(n * n * (n // 2 + 1), dtype=slices.dtype, device="cuda")
    out_w = torch.zeros(out.shape, dtype=torch.float64, device="cuda")
    for b in range(slices.shape[0]):
        r = _parts(rotation[b], torch.float64, 0)
        near = (_rotate(r, f)[0].abs() <= blackman).nonzero()[:, 0]
        g = _rotate(r, [a[near] for a in f])
        f0, f1 = _scale(None if scaling is None else _parts(scaling[b].reshape(4), torch.float64, 0), g[1], g[2])
        k = _window(g[0], sinc, blackman)
        v = _interpolate(slices[b, 0], in_centered, (size, size), [f0 * size, f1 * size], c["interp"])
        out[inside[near]] += v * k  # a voxel appears once per slice
        out_w[inside[near]] += k
    shape = (1, n, n, n // 2 + 1)
    return out.reshape(shape), out_w.reshape(shape)


def _exact_insert_extract(c, slices, rotation, scaling, rotation2, size):
    in_centered, out_centered = c["remap"].startswith("hc"), c["remap"].endswith("hc")
    slices, count = _double(slices), slices.shape[0]
    flat = slices.reshape(count, -1)
    sinc = blackman = 1 / size
    axes = torch.eye(3, dtype=torch.float64, device="cuda")
    rows = torch.stack(_rotate(_parts(rotation, torch.float64, 1), [a[None] for a in axes]), 1)  # (count, 3, 3)
    values, weights = [], []
    wp = size // 2 + 1
    for b in range(rotation2.shape[0]):
        near, far = (_slice_to_grid(size, out_centered, None, rotation2[b:b + 1], t)
                     for t in (torch.float32, torch.float64))
        keep = _inside(near, c["cutoff"])[0]
        g = torch.stack([a[0][keep] for a in far])
        i, p = ((rows[:, 0] @ g).abs() < blackman).nonzero(as_tuple=True)
        gp = g[:, p]
        fz, f0, f1 = ((rows[i, k] * gp.T).sum(1) for k in range(3))
        if scaling is not None:
            s = scaling.double()[i]
            f0, f1 = s[:, 0, 0] * f0 + s[:, 0, 1] * f1, s[:, 1, 0] * f0 + s[:, 1, 1] * f1
        k = _window(fz, sinc, blackman)
        q0, q1 = f0 * size, f1 * size
        flip = q1 < 0
        q0, q1 = torch.where(flip, -q0, q0), torch.where(flip, -q1, q1)
        b0, b1 = torch.floor(q0).long(), torch.floor(q1).long()
        v = torch.zeros(i.shape, dtype=slices.dtype, device="cuda")
        for d0 in range(2):
            for d1 in range(2):
                a0, a1 = b0 + d0, b1 + d1
                w = (q0 - b0 if d0 else 1 - (q0 - b0)) * (q1 - b1 if d1 else 1 - (q1 - b1))
                good = (a0 >= -(size // 2)) & (a0 <= (size - 1) // 2) & (a1 <= size // 2)
                row = a0 + size // 2 if in_centered else torch.where(a0 < 0, a0 + size, a0)
                v += torch.where(good, flat[i, torch.where(good, row * wp + a1, 0)] * w, torch.zeros_like(v))
        v = torch.where(flip, v.conj(), v) if v.is_complex() else v
        value = torch.zeros((size, wp), dtype=slices.dtype, device="cuda")
        weight = torch.zeros((size, wp), dtype=torch.float64, device="cuda")
        sums = torch.zeros(g.shape[1], dtype=torch.float64, device="cuda")
        if v.is_complex():
            parts = [sums.clone().index_add_(0, p, a * k) for a in (v.real, v.imag)]
            value[keep] = torch.complex(*parts)
        else:
            value[keep] = sums.clone().index_add_(0, p, v * k)
        weight[keep] = sums.index_add_(0, p, k)
        values.append(value)
        weights.append(weight)
    return torch.stack(values)[:, None], torch.stack(weights)[:, None]


def _exact_reconstruct(c, values, weights):
    n = c["n"]
    centered = c["remap"].startswith("hc")
    spectrum = _double(values)[0] / weights[0].double().clamp_min(1.0)
    if centered:
        spectrum = torch.roll(spectrum, (-(n // 2), -(n // 2)), (0, 1))
    k, x = _indices(n, False).double(), torch.arange(n // 2 + 1, device="cuda").double()
    turns = (n // 2) / n * (k[:, None, None] + k[None, :, None] + x[None, None, :])
    spectrum = spectrum * torch.exp(-2j * math.pi * (turns - turns.round()))
    real = torch.fft.irfftn(spectrum, s=(n, n, n))
    d = ((torch.arange(n, device="cuda").double() - n / 2) / n).square()
    r = math.pi * (d[:, None, None] + d[None, :, None] + d[None, None, :]).sqrt()
    return (real / torch.sinc(r / math.pi).square())[None]


def exact(case: dict, seed: int):
    c = _full(case)
    size = c["size"] or c["n"]
    pixels = c["slices"] * size * (size // 2 + 1)
    if c["op"] == "extract" and pixels * WINDOW_SIZE[c["interp"]] ** 3 * max(1.0, 2 * c["w_width"] - 1) > 6e9:
        return None  # minutes of elementwise passes
    state = prepare(case, seed)
    if c["op"] == "reconstruct":
        return _exact_reconstruct(c, state["values"], state["weights"])
    if c["op"] == "batch":
        got = []
        for r in state["requests"]:
            box, count = r.volume_shape[1], r.slice_shape[0]
            got.append(_exact_extract({**c, "n": box}, r.volume, r.fwd_rotation, None, box, count)[0])
        return got
    if c["op"] == "extract":
        got = _exact_extract(c, state["input"], state["rotation"], state["scaling"], size, c["slices"])
    elif c["op"] == "rasterize":
        got = _exact_rasterize(c, state["input"], state["rotation"], state["scaling"], size)
    elif c["op"] == "insert_extract":
        got = _exact_insert_extract(c, state["input"], state["rotation"], state["scaling"], state["rotation2"], size)
    else:
        got = _exact_insert(c, state["input"], state["rotation"], state["scaling"], size)
    return got if c["weights"] else got[0]
