"""GPU kernels at the edges of their tiles and dispatch rules, against the oracle (relative L2 1e-5, the
tolerance of the same call in test_gpu_parity.py; 1e-4 for the rasterizer's atomic sums)."""
import numpy as np
import pytest

from cases import build, clone, default_case, rel_l2
from oracle.oracle import FpOracle

pytestmark = pytest.mark.gpu


def _check(case, tol, copies=None, **kw):
    """`copies`: how many pair copies the call has to make (None: not looked at)."""
    import gpu_run
    call = build(case)
    if copies is not None:
        assert gpu_run.scratch_wanted(lambda: gpu_run.run(clone(call), **kw))[0] == copies
    ref = clone(call)
    assert FpOracle().run(ref, 8) == 0
    out, out_w = gpu_run.run(clone(call), **kw)
    assert rel_l2(out, ref.out) <= tol
    if ref.out_w is not None:
        assert rel_l2(out_w, ref.out_w) <= tol


# Warp patches of 4x8 pixels that the slice fills partly, cells across x = 0 and the edges of the volume
# (cutoff beyond 0.5), every window size, both value kinds, input weights, the w-window.
@pytest.mark.parametrize("interp", ["cubic", "cubic_bspline", "lanczos4", "lanczos6", "lanczos8"])
@pytest.mark.parametrize("kw", [
    dict(n=9, slice_n=9, remap="h2h", cutoff=0.8),
    dict(n=33, slice_n=21, remap="hc2hc", in_w=True, out_w=True),
    dict(n=26, slice_n=17, remap="h2hc", in_dt="f32", out_dt="f32", cutoff=0.7, out_w=True),
    dict(n=24, remap="hc2h", w_sinc=(0.05, 0.12), out_w=True, in_w=True),
], ids=["tiny", "weights", "real", "w-window"])
def test_window_extraction(interp, kw):
    _check(default_case("extract", interp=interp, nslices=3, seed=701, **kw), 1e-5)


# A slice whose rotation is NaN: with a w-window every sample passes the cutoff test (it excludes what is
# larger), so the slice's values and weights are NaN, whatever the interpolation, and the others are not.
@pytest.mark.parametrize("interp", ["nearest", "linear", "cubic", "cubic_bspline", "lanczos4", "lanczos6", "lanczos8"])
@pytest.mark.parametrize("dt", ["c32", "f32"])
def test_nan_rotation_with_w_window(interp, dt):
    import gpu_run
    call = build(default_case("extract", interp=interp, n=24, nslices=3, remap="hc2h", in_dt=dt, out_dt=dt, in_w=True,
                              out_w=True, w_sinc=(0.05, 0.12), seed=709))
    call.rot[1] = np.nan
    out, out_w = gpu_run.run(call)
    if interp != "nearest":  # takes the nearest voxel without weights
        assert np.isnan(out[1]).all() and np.isnan(out_w[1]).all()
    assert np.isfinite(out[[0, 2]]).all() and np.isfinite(out_w[[0, 2]]).all()


# Run lengths of 1, 2, 4, 8 and 16 rows (148 SMs x 1024 threads decide), the last run of a column shorter.
@pytest.mark.parametrize("nslices", [7, 400, 800, 1600, 3200])
def test_rasterize_run_lengths(nslices):
    _check(default_case("rasterize", n=40, nslices=nslices, remap="h2hc", out_w=True, seed=702), 1e-4)


# The planes that a pixel's z samples share: more samples than planes of the volume, offsets outside it, a
# window wider than the table, odd sizes, power spectra; from a pair copy and from the volume.
@pytest.mark.parametrize("copies", [0, 1])
@pytest.mark.parametrize("kw", [dict(n=16, w_sinc=(0.05, 0.9), cutoff=0.9, nslices=520), dict(n=64, w_sinc=(0.1, 0.6), cutoff=0.7, nslices=160),
                                dict(n=17, w_sinc=(-1.0, 0.2), remap="h2h", nslices=2000),
                                dict(n=20, w_sinc=(-1.0, 0.15), out_dt="f32", nslices=2000)],
                         ids=["beyond", "long", "odd", "power"])
def test_w_window_planes(kw, copies):
    case = default_case("extract", **{"remap": "hc2h", "out_w": True, "seed": 703, **kw})
    if not copies:
        case["nslices"] = 8
    _check(case, 1e-5, copies)


# LINEAR insertion from Mat33 rotations: bricks that the volume fills partly, more slices than one pass of
# the list, both layouts, value kinds, input weights, windows from one voxel to wider than the volume.
@pytest.mark.parametrize("scatter", [False, True], ids=["gather", "scatter"])
@pytest.mark.parametrize("kw", [dict(n=9, nslices=300, out_w=True), dict(n=17, nslices=40, sinc=(0.06, 0.4), remap="hc2hc"),
                                dict(n=20, nslices=30, slice_n=15, in_w=True, out_w=True, remap="h2hc", cutoff=0.8),
                                dict(n=16, nslices=20, in_dt="f32", out_dt="f32", in_w=True, out_w=True, sinc=(-1.0, 1.5)),
                                dict(n=24, nslices=270, in_dt="c32", out_dt="f32", remap="h2h", sinc=(-1.0, 0.2))],
                         ids=["small", "wide", "weights", "real", "power"])
def test_linear_insertion(kw, scatter):
    _check(default_case("insert", **{"seed": 704, **kw}), 1e-5, scatter=scatter)


# The same for the gather form by packed pairs of voxels, which takes launches of many 8^3 bricks: 320 for one
# slice, 320 s^(2/3) for s, 12,000 for any number. Its smallest launches, partly filled bricks on every
# axis, a second pass of the list (256 slices each), and the other options as above; and the general
# kernel just below each line.
@pytest.mark.parametrize("linear,kw", [
    (True, dict(n=64, nslices=1, out_w=True)), (False, dict(n=56, nslices=1, out_w=True)),
    (True, dict(n=85, nslices=3, slice_n=70, in_w=True, out_w=True, remap="h2hc", cutoff=0.8)),
    (False, dict(n=72, nslices=3, slice_n=70, in_w=True, out_w=True, remap="h2hc", cutoff=0.8)),
    (True, dict(n=84, nslices=3, in_dt="f32", out_dt="f32", in_w=True, out_w=True, sinc=(-1.0, 1.5))),
    (True, dict(n=97, nslices=4, in_dt="c32", out_dt="f32", remap="h2h", sinc=(-1.0, 0.2))),
    (True, dict(n=131, nslices=17, sinc=(0.01, 6 / 131), remap="hc2hc")),
    (True, dict(n=227, nslices=260, remap="hc2hc")), (False, dict(n=217, nslices=260, remap="hc2hc"))],
    ids=["one", "one-below", "weights", "weights-below", "real", "power", "wide", "passes", "passes-below"])
def test_linear_insertion_kernel(linear, kw):
    bricks = ((kw["n"] + 7) // 8) ** 2 * ((kw["n"] // 2 + 8) // 8)
    assert linear == (bricks >= 12000 or bricks ** 3 >= 320 ** 3 * kw["nslices"] ** 2)
    _check(default_case("insert", **{"seed": 707, **kw}), 1e-5)


# In-slice coordinates past the range of the integers: no tap of the slice is read, as for coordinates that are
# outside it by less. A slice scaled by 1e15 adds what one scaled by 1e7 adds; one whose in-plane matrix rows are
# infinite leaves the voxels and pixels outside its slab as they are.
@pytest.mark.parametrize("interp", ["nearest", "linear", "cubic", "cubic_bspline", "lanczos4", "lanczos6", "lanczos8"])
@pytest.mark.parametrize("func", ["insert", "scatter", "insert_extract"])
@pytest.mark.parametrize("kw", [dict(), dict(rot="quat"), dict(sinc=(0.05, 0.3)), dict(in_dt="f32", out_dt="f32", in_w=True, out_w=True)],
                         ids=["thin", "quat", "thick", "real"])
def test_coordinates_past_the_integers(interp, func, kw):
    import gpu_run
    call = build(default_case(func.replace("scatter", "insert"), interp=interp, n=24, nslices=12, remap="h2h", scale=True,
                              seed=712, **kw))
    scatter = func == "scatter"
    outs = []
    for factor in (1e7, 1e15):
        c = clone(call)
        c.scale = call.scale.copy()
        c.scale[5] *= np.float32(factor)
        outs.append(gpu_run.run(c, scatter=scatter)[0])
    assert np.isfinite(outs[0]).all() and np.abs(outs[0]).max() > 0
    assert rel_l2(outs[1], outs[0]) <= 1e-6 if scatter else np.array_equal(outs[0], outs[1])
    if call.rot.shape[1:] == (3, 3) and interp != "nearest":  # which takes a voxel for NaN coordinates (inf * 0)
        c = clone(call)
        c.scale, c.rot = None, call.rot.copy()
        base = clone(c)
        base.rot[5, 1:] *= np.float32(1e7)
        outs = [gpu_run.run(base, scatter=scatter)[0]]
        c.rot = call.rot.copy()
        c.rot[5, 1:] = np.inf
        outs.append(gpu_run.run(c, scatter=scatter)[0])
        same = np.isfinite(outs[1])
        assert same.any() and rel_l2(outs[1][same], outs[0][same]) <= (1e-6 if scatter else 0)


# The pairs of insert_and_extract by the queue (LINEAR matrices two per lane, else one) and by walking: fewer
# pairs than a half, halves that fill exactly and by many slices, a second pass of the input slices (4096
# each), windows over the whole slice, w offsets, every value kind; slabs on either side of each form's
# width (5, 2 and 1.5 pixels), and 8 and fewer slices.
@pytest.mark.parametrize("kw", [dict(n=12, nslices=1, nout=2), dict(n=10, nslices=4200, nout=1, out_w=True),
                                dict(n=33, nslices=64, nout=3, sinc=(0.03, 1.0), out_w=True, in_w=True),
                                dict(n=33, nslices=64, nout=3, sinc=(0.03, 0.14), out_w=True, in_w=True),
                                dict(n=20, nslices=40, nout=3, rot="quat", scale=True, sinc=(0.02, 0.2), out_w=True),
                                dict(n=20, nslices=40, nout=3, rot="quat", scale=True, sinc=(0.02, 0.09), out_w=True),
                                dict(n=10, nslices=4200, nout=1, rot="quat", out_w=True),
                                dict(n=20, nslices=40, nout=2, sinc=(0.02, 0.1), w_sinc=(0.05, 0.2), out_w=True),
                                dict(n=18, nslices=40, nout=2, in_dt="f32", out_dt="f32", interp="nearest"),
                                dict(n=18, nslices=40, nout=2, in_dt="f32", out_dt="f32", interp="nearest", sinc=(0.06, 0.3))],
                         ids=["few", "passes", "wide", "thick", "general", "general-thin", "general-passes", "w-window",
                              "nearest", "nearest-wide"])
def test_pair_queue(kw):
    _check(default_case("insert_extract", **{"remap": "h2h", "seed": 705, **kw}), 1e-5)


@pytest.mark.parametrize("interp", ["cubic", "cubic_bspline", "lanczos4", "lanczos6", "lanczos8"])
@pytest.mark.parametrize("kw", [dict(nslices=70, rot="quat"), dict(nslices=8, in_w=True), dict(nslices=7),
                                dict(nslices=40, sinc=(0.05, 0.3), in_w=True), dict(nslices=40, in_dt="f32", out_dt="f32"),
                                dict(nslices=40, w_sinc=(0.05, 0.12), out_dt="f32")],
                         ids=["quat", "eight", "seven", "wide", "real", "w-window"])
def test_pair_queue_windows(interp, kw):
    _check(default_case("insert_extract", n=22, nout=3, remap="h2h", out_w=True, seed=708, interp=interp, **kw), 1e-5)


# More tiles than are taken slice by slice (592): by place, rows alternately below and above the origin's, odd
# and even numbers of rows, both layouts; and launches of many tiles that meet few slices each.
@pytest.mark.parametrize("remap", ["h2h", "h2hc"])
@pytest.mark.parametrize("kw", [dict(n=33, nout=110, nslices=30), dict(n=49, nout=80, nslices=200, rot="quat"),
                                dict(n=64, nout=110, nslices=20), dict(n=64, nout=110, nslices=22, interp="nearest")],
                         ids=["odd", "even", "few", "enough"])
def test_tile_order(kw, remap):
    _check(default_case("insert_extract", **{"remap": remap, "out_w": True, "seed": 711, **kw}), 1e-5)


# LINEAR extraction: several slices per CTA with a shorter last group, rows past the slice, cells at the
# edges of the volume and the non-centered wrap; over a pair copy, from the volume with four pixels per thread
# (1.52 M pixels, 1.82 M with input weights, 1.22 M real) and with one.
@pytest.mark.parametrize("remap", ["h2h", "hc2hc"])
@pytest.mark.parametrize("copies,kw", [(1, dict(n=20, nslices=9700)), (0, dict(n=20, nslices=1030)),
                                       (1, dict(n=21, slice_n=70, nslices=841, target=(1, 70, 70, 70), cutoff=0.9)),
                                       (0, dict(n=21, slice_n=70, nslices=610, target=(1, 70, 70, 70), cutoff=0.9)),
                                       (0, dict(n=21, slice_n=70, nslices=513, target=(1, 70, 70, 70), cutoff=0.9)),
                                       (1, dict(n=40, nslices=2600, out_dt="f32", out_w=True)),
                                       (0, dict(n=40, nslices=1830, out_dt="f32", out_w=True)),
                                       (0, dict(n=40, nslices=800, out_dt="f32", out_w=True)),
                                       (0, dict(n=64, nslices=870, in_w=True, out_w=True)),
                                       (0, dict(n=64, nslices=301, in_w=True, out_w=True)),
                                       (0, dict(n=40, nslices=1450, in_dt="f32", out_dt="f32")),
                                       (0, dict(n=40, nslices=800, in_dt="f32", out_dt="f32"))],
                         ids=["pairs", "small", "beyond-pairs", "beyond", "beyond-small", "power-pairs", "power", "power-small",
                              "weights", "weights-small", "real", "real-small"])
def test_linear_extraction_groups(kw, copies, remap):
    _check(default_case("extract", remap=remap, seed=706, **kw), 1e-5, copies)


# The rule on making a pair copy (two pixels per voxel, 2^21 pixels), its padded strides, and requests of a
# batch that read their volume in grids of their own: the same bits with and without the copy, in every layout
# and with every form of the coordinates and outputs that a copy serves.
def _with_and_without_pair_copy(n, size, count, remap="hc2h", form="plain"):
    import gpu_run
    import torch
    from noa_b200 import fourier_project as fp, synthetic
    from noa_b200.batch import ExtractBatch, ExtractRequest
    q = synthetic.random_quaternions(count, seed=count)
    rot = torch.from_numpy(q.astype(np.float32)).cuda() if form == "quaternion" else \
        fp.pack_rotations(torch.from_numpy(synthetic.quaternion_to_matrix(q).astype(np.float32)).cuda())
    vol = synthetic.make_volume(n, seed=n)  # centered
    if remap.startswith("h2"):
        vol = np.ascontiguousarray(np.fft.ifftshift(vol, axes=(1, 2)))
    vol = torch.from_numpy(vol).cuda()
    scale = torch.from_numpy(synthetic.scale_matrices(count, (1.0, 1.0), seed=5, jitter=0.05).astype(np.float32)).cuda() \
        if form == "scaled" else None
    kw = {"curved": dict(ews_radius=(45.0, 60.0)), "cutoff": dict(fftfreq_cutoff=0.8)}.get(form, {})
    shape, slices = (1, n, n, n), (count, 1, size, size)
    dt = torch.float32 if form == "power" else torch.complex64
    outs = [torch.empty((count, 1, size, size // 2 + 1), dtype=dt, device="cuda") for _ in range(3)]
    weights = [torch.empty(outs[0].shape, device="cuda") if form == "weights" else None for _ in range(3)]

    def extract(k):
        fp.extract_central_slices_3d(remap, vol, None, shape, outs[k], weights[k], slices, scale, rot, **kw)
    extract(0)
    assert gpu_run.scratch_wanted(lambda: extract(1))[0] == 1
    batch = ExtractBatch(remap, [ExtractRequest(volume=vol, volume_shape=shape, slice=outs[2], slice_shape=slices,
                                                slice_weight=weights[2], inv_scaling=scale, fwd_rotation=rot)],
                         autotune=False, **kw)
    batch.run()
    torch.cuda.synchronize()
    assert batch.info()["n_direct"] == 1
    assert outs[0].abs().max().item() > 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    if form == "weights":
        assert torch.equal(weights[0], weights[1]) and torch.equal(weights[0], weights[2])
    batch.close()


@pytest.mark.parametrize("n,size,count", [(33, 33, 4000), (64, 64, 1100), (96, 95, 470), (40, 200, 110), (128, 128, 400)])
def test_extraction_with_and_without_pair_copy(n, size, count):
    _with_and_without_pair_copy(n, size, count)


@pytest.mark.parametrize("remap", ["h2h", "h2hc", "hc2h", "hc2hc"])
@pytest.mark.parametrize("form", ["plain", "power", "weights", "quaternion", "scaled", "curved", "cutoff"])
def test_forms_with_and_without_pair_copy(form, remap):
    _with_and_without_pair_copy(33, 33, 4000, remap, form)
    _with_and_without_pair_copy(40, 51, 1600, remap, form)
