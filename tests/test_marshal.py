"""The native marshalling fills the structures that the ctypes path fills, and refuses what it refuses (CPU)."""
import ctypes as C
import os
import subprocess
import sysconfig

import numpy as np
import pytest
import torch

from noa_b200 import build
from noa_b200 import fourier_project as fp

pytestmark = pytest.mark.skipif(fp._native() is None, reason="built without Python headers")

_P = C.c_void_p
_ENTRY = {n: C.CFUNCTYPE(C.c_int, C.c_int32, *([_P] * (8 + n))) for n in (2, 4)}


def _bytes(address, struct):
    return None if not address else C.string_at(address, C.sizeof(struct))


def _seen(monkeypatch, native, call, n_transforms):
    """What the entry point gets from `call`, by value."""
    got = []

    def entry(remap, *p):
        got.append((remap, [_bytes(p[i], fp.NbArray) for i in (0, 1, 3, 4)],
                    [_bytes(p[i], C.c_int64 * 4) for i in (2, 5)],
                    [_bytes(p[6 + i], fp.NbTransform) for i in range(n_transforms)],
                    _bytes(p[6 + n_transforms], fp.NbOptions), p[7 + n_transforms]))
        return 0

    function = _ENTRY[n_transforms](entry)
    with monkeypatch.context() as m:
        if native:
            m.setattr(fp, "_address", lambda name: C.cast(function, _P).value)
        else:
            m.setattr(fp, "_native", lambda: None)
            m.setattr(fp, "lib", lambda: type("Lib", (), {"__getattr__": lambda self, name: function}, )())
            m.setattr(fp, "_default_options", lambda: fp.NbOptions(interp=1))
        call()
    return got


_vol = torch.zeros((1, 8, 8, 5), dtype=torch.complex64)
_out = torch.zeros((3, 1, 8, 9), dtype=torch.float32)[..., ::2]
_w = torch.zeros((3, 1, 8, 5))
_rot, _quat, _scale = torch.eye(3).repeat(3, 1, 1), torch.zeros((3, 4)), torch.zeros((3, 2, 2))
_packed = fp.pack_rotations(_rot)


@pytest.mark.parametrize("volume", [_vol, 2.5, 3, 1 + 2j, np.float64(4.0)], ids=str)
@pytest.mark.parametrize("weight", [_w, None])
@pytest.mark.parametrize("rotation", [_packed, _quat, np.eye(3), (0, 0, 0, 1)], ids=["mat33", "quat", "one", "inline"])
@pytest.mark.parametrize("kw", [{}, dict(interp="lanczos8", fftfreq_cutoff=1, ews_radius=3.5, target_shape=[1, 9, 9, 9, 7]),
                                dict(interp=101, w_windowed_sinc=fp.WindowedSinc(0.1, 1), ews_radius=np.array([1.0, 2.0]))],
                         ids=["default", "options", "more"])
def test_same_structures(monkeypatch, volume, weight, rotation, kw):
    for scaling in (None, _scale, np.eye(2)):
        def call():
            fp.extract_central_slices_3d("hc2h", volume, None, (1, 8, 8, 8), _out, weight, torch.Size((3, 1, 8, 8)), scaling,
                                         rotation, stream=77, **kw)
        a, b = _seen(monkeypatch, True, call, 2), _seen(monkeypatch, False, call, 2)
        assert a == b and len(a) == 1


def _call_with(**kw):
    fp.extract_central_slices_3d("hc2h", _vol, None, (1, 8, 8, 8), _out, None, (3, 1, 8, 8), None, _packed, stream=3, **kw)


def _same(monkeypatch, call):
    """What both ways make of `call`: the structures, or the class of the error."""
    results = []
    for native in (True, False):
        try:
            results.append(_seen(monkeypatch, native, call, 2))
        except Exception as e:
            results.append(type(e))
    return results


@pytest.mark.parametrize("radius,accepted", [
    (0, True), (3.5, True), (True, True), (np.float32(3), True), (np.int64(4), True), ((1, 2), True), ([1.5, 2], True),
    ((1, 2, 3), True), (np.array([1.0, 2.0]), True), (torch.tensor([1.0, 2.0]), True), ("3", True), ({0: 1, 1: 2}, True),
    ((1,), False), ([], False), (np.array(3.0), False), (torch.tensor(3.0), False), ("ab", False), (None, False)], ids=repr)
def test_same_ews_radius(monkeypatch, radius, accepted):
    a, b = _same(monkeypatch, lambda: _call_with(ews_radius=radius))
    assert a == b and isinstance(a, list) == accepted


@pytest.mark.parametrize("target,accepted", [
    (lambda: (1, 8, 8, 8), True), (lambda: [1, 8, 8, 8, 9], True), (lambda: torch.Size((1, 8, 8, 8)), True),
    (lambda: np.array([1, 8, 8, 8]), True), (lambda: torch.tensor([1, 8, 8, 8, 8]), True), (lambda: {3: 4, 2: 3, 1: 2, 0: 1}, True),
    (lambda: "1888", True), (lambda: {1: 0, 8: 0, 9: 0, 7: 0}, False), (lambda: (x for x in (1, 8, 8, 8)), False),
    (lambda: {1, 2, 3, 4}, False), (lambda: (1, 8, 8), False), (lambda: 8, False)])
def test_same_target_shape(monkeypatch, target, accepted):
    a, b = _same(monkeypatch, lambda: _call_with(target_shape=target()))
    assert a == b and isinstance(a, list) == accepted


@pytest.mark.parametrize("big", [2 ** 63, 2 ** 64 + 8, 2 ** 70, -2 ** 63, -2 ** 63 - 1, 2 ** 32 + 1, -1])
def test_same_integers_beyond_the_structures(monkeypatch, big):
    def call():
        fp.extract_central_slices_3d("hc2h", _vol, None, (1, big, 8, 8), _out, None, (3, 1, 8, big), None, _packed,
                                     stream=big, target_shape=(1, big, 8, 8), interp=big)
    a, b = _same(monkeypatch, call)
    assert a == b and isinstance(a, list)


def test_same_structures_of_both_sides(monkeypatch):
    def call():
        fp.insert_and_extract_central_slices_3d(
            "h2h", _w, 2.0, (3, 1, 8, 8), _out, _w, np.array([3, 1, 8, 8]), _scale, _packed, None, _quat,
            input_windowed_sinc=fp.WindowedSinc(0.2, 0.3), add_to_output=np.bool_(True), correct_weights=0, stream=5)
    a, b = _seen(monkeypatch, True, call, 4), _seen(monkeypatch, False, call, 4)
    assert a == b and len(a) == 1


@pytest.mark.parametrize("change", [dict(volume=_vol[0]), dict(volume=torch.zeros((1, 8, 8, 5), dtype=torch.int32)),
                                    dict(rotation=None), dict(rotation=np.zeros((2, 3))), dict(rotation=_quat.double()),
                                    dict(rotation=torch.zeros((3, 5))), dict(shape=(1, 8, 8, 8, 8)), dict(interp="none"),
                                    dict(target_shape=(1, 2)), dict(volume="x"), dict(remap="h2x"), dict(interp=None)],
                         ids=str)
def test_same_refusals(monkeypatch, change):
    a = dict(volume=_vol, rotation=_packed, shape=(1, 8, 8, 8), interp="linear", target_shape=None, remap="hc2h")
    a.update(change)

    def call():
        fp.extract_central_slices_3d(a["remap"], a["volume"], None, a["shape"], _out, None, (3, 1, 8, 8), None, a["rotation"],
                                     interp=a["interp"], target_shape=a["target_shape"], stream=0)
    errors = []
    for native in (True, False):
        with pytest.raises(Exception) as e:
            _seen(monkeypatch, native, call, 2)
        errors.append((type(e.value), getattr(e.value, "code", None)))
    assert errors[0] == errors[1]


def test_the_module_is_of_this_interpreter():
    """Its name carries the ABI tag, so a module that another Python built beside the library is not loaded."""
    assert fp._MARSHAL_PATH.endswith("/_marshal" + sysconfig.get_config_var("EXT_SUFFIX"))
    assert build.MARSHAL == os.path.basename(fp._MARSHAL_PATH)


def test_a_module_that_does_not_load_leaves_ctypes(monkeypatch, tmp_path):
    path = tmp_path / build.MARSHAL
    path.write_bytes(b"not an extension")
    monkeypatch.setattr(fp, "_MARSHAL_PATH", str(path))
    monkeypatch.setattr(fp, "_native_module", [])
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert fp._native() is None
    assert fp._native() is None  # decided once, without another warning


def test_a_module_that_does_not_compile_leaves_the_library_build_going(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "LIBDIR", str(tmp_path))
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: subprocess.CompletedProcess(a, 1, "", "no compiler"))
    with pytest.warns(RuntimeWarning, match="no compiler"):
        build._build_marshal()


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_current_stream_without_torchs_private_functions(monkeypatch, missing):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 11, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), {"cuda_stream": 12}))
    assert fp._stream_ptr(None) == 11
    monkeypatch.delattr(torch._C, missing)
    assert fp._stream_ptr(None) == 12
