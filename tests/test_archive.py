"""The library's archive writer and reader (csrc/archive.cu) against numpy, zipfile and the same records
packed in Python: sizes around the words and blocks its checksum folds."""

from __future__ import annotations

import io
import zipfile

import numpy as np
import pytest

from turboquant_pro_b200 import _lib, kv_blob


def _bytes(n, seed=0):
    return np.random.default_rng(seed + n).integers(0, 256, n, dtype=np.uint8)


@pytest.mark.parametrize("sizes", [[*range(20)], [*range(60, 84)], [127, 128, 129, 191, 192, 193, 255, 256],
                                   [4095, 4096, 4111, 65536, 100003]])
def test_bytes_of_savez(sizes, monkeypatch):
    arrays = {f"k.{n}": _bytes(n) for n in sizes}
    buf = io.BytesIO()
    np.savez(buf, **arrays)
    blob = kv_blob._write_native(_lib.load(), arrays)
    assert blob == buf.getvalue()
    assert zipfile.ZipFile(io.BytesIO(blob)).testzip() is None  # zlib's checksum of every member
    for copy in (True, False):
        back = kv_blob._read_native(_lib.load(), blob, 1 << 30, copy)
        assert list(back) == list(arrays) and all(np.array_equal(back[k], arrays[k]) for k in arrays)
    monkeypatch.setattr(kv_blob, "_native", lambda: None)
    assert kv_blob._write_npz(arrays) == blob
    assert all(np.array_equal(a, arrays[k]) for k, a in kv_blob._read_npz(blob, 1 << 30).items())


def test_forms_and_damage():
    arrays = {"a": np.arange(30, dtype=np.float32).reshape(1, 5, 6), "b": np.zeros((0, 3), np.int32),
              "c": np.float16([[1.5]]), "d": _bytes(300)}
    blob = kv_blob._write_native(_lib.load(), arrays)
    back = kv_blob._read_native(_lib.load(), blob, 1 << 20, True)
    for k, a in arrays.items():
        assert back[k].dtype == a.dtype and back[k].shape == a.shape and np.array_equal(back[k], a)
        assert back[k].flags.writeable
    assert kv_blob._read_native(_lib.load(), blob, 100, True) is None  # above the limit
    for at in range(0, len(blob), 7):
        bad = bytearray(blob)
        bad[at] ^= 0x40
        got = kv_blob._read_native(_lib.load(), bytes(bad), 1 << 20, True)
        # a field that neither reader looks at (times, versions, attributes, the repeated sizes) changes nothing
        assert got is None or all(np.array_equal(got[k], a) for k, a in arrays.items())
    for n in range(0, len(blob), 11):
        assert kv_blob._read_native(_lib.load(), blob[:n], 1 << 20, True) is None
    many = kv_blob._write_native(_lib.load(), {str(i): _bytes(3) for i in range(70)})
    assert kv_blob._read_native(_lib.load(), many, 1 << 20, True) is None  # (left to numpy)
    with np.load(io.BytesIO(many)) as z:
        assert len(z.files) == 70


def test_prototypes_of_other_packages_are_left_alone():
    """ctypes.pythonapi is shared by the whole process: its attributes are neither changed nor relied on."""
    import ctypes

    shared = ctypes.pythonapi.PyBytes_FromStringAndSize
    before = shared.restype, shared.argtypes
    assert before != (ctypes.py_object, [ctypes.c_void_p, ctypes.c_ssize_t])
    arrays = {"a": np.arange(1000, dtype=np.int32)}
    want = kv_blob._write_npz(arrays)
    try:
        shared.restype, shared.argtypes = ctypes.c_int, [ctypes.c_char_p, ctypes.c_int]
        assert kv_blob._write_npz(arrays) == want
    finally:
        shared.restype, shared.argtypes = before
