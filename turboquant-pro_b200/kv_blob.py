"""One compressed KV block as a self-describing byte string (codec ``tqp-kv-npz/1``).

The reference's vLLM connector stores a (request, layer) block as one ``.npz`` archive: the
arrays of the key and value containers under ``k.*`` / ``v.*`` plus a JSON header with the
scalars (``connectors/vllm_v1.py:67``, ``:113-196``).  This module writes and reads that
layout for blocks exported from the GPU context (``KVContext.export_block``), so blocks
produced here can be consumed by the reference and the other way round.  No pickle is
involved in either direction; the reader refuses what it does not know instead of guessing
(codec string, size limits, dtype whitelist), as the reference's reader does.

``block_from_parsed`` turns a parsed blob back into the arrays ``KVContext.import_block``
takes, so a stored block goes into device pages without passing through dense tensors.
"""

from __future__ import annotations

import contextlib
import ctypes
import functools
import io
import json
import math
import re
import struct
import zlib

import numpy as np

CODEC = "tqp-kv-npz/1"
_OK_DTYPES = {"uint8", "int8", "int16", "int32", "int64", "float16", "float32", "float64", "bool"}

__all__ = ["CODEC", "block_to_blob", "blob_to_block", "block_from_parsed"]


@functools.lru_cache(maxsize=64)
def _allowed(dtype) -> bool:
    return str(dtype) in _OK_DTYPES


def _tuple(v):
    return {"__tuple__": [int(x) for x in v]}


def _dtype(name):
    return {"__dtype__": str(np.dtype(name))}


def block_to_blob(block: dict, *, key_mode: str = "nf4_asym", zero_point: str = "calibrated",
                  mean_mask=None, rope_theta: float | None = None, position_start: int = 0,
                  dtype: str = "float32") -> bytes:
    """Serialise one exported cold block.

    ``block`` is the dict of ``KVContext.export_block`` (reference container layout:
    bit-reversed packed key nibbles, LSB-first packed value codes, ``(1, H, D)`` key scale
    and mean, flat int32 outlier indices with float16 values, ``(1, H, S)`` value norms).
    ``key_mode`` / ``zero_point`` say how the key scalars are to be named and which of them
    the format stores: uniform keys as ``scale`` / ``zero`` ``(1, H, 1, D)``; symmetric NF4
    without a mean; the ``sparse`` zero-point with the means of the ``mean_mask`` channels
    only; the ``bias`` zero-point with none (``rope_theta`` and ``position_start`` let the
    reader recompute it).  ``dtype`` is the element type the tokens had.
    """
    shape = tuple(int(x) for x in block["shape"])
    k_arr: dict[str, np.ndarray] = {"indices": np.ascontiguousarray(block["key_indices"])}
    k_sc = {"scale": None, "zero": None, "bits": int(block["key_bits"]), "shape": _tuple(shape),
            "packed": True, "levels": None, "original_dtype": _dtype("float32"),
            "zp_mode": "calibrated", "rope_theta": None, "position_start": int(position_start)}
    scale, mean = np.asarray(block["nf4_scale"]), np.asarray(block["nf4_mean"])
    if key_mode == "uniform":
        del k_sc["scale"], k_sc["zero"]
        k_arr["scale"] = np.ascontiguousarray(scale[:, :, None, :])
        k_arr["zero"] = np.ascontiguousarray(mean[:, :, None, :])
        k_sc["nf4_scale"] = k_sc["nf4_mean"] = None
    else:
        k_arr["nf4_scale"] = np.ascontiguousarray(scale)
        if key_mode == "nf4":
            k_sc["nf4_mean"] = None
        elif zero_point == "sparse":
            if mean_mask is None or rope_theta is None:
                raise ValueError("the sparse zero-point needs mean_mask and rope_theta")
            k_arr["nf4_mean"] = np.ascontiguousarray(mean[:, :, np.asarray(mean_mask, bool)])
            k_sc["zp_mode"], k_sc["rope_theta"] = "sparse", float(rope_theta)
        elif zero_point == "bias":
            if rope_theta is None:
                raise ValueError("the bias zero-point needs rope_theta")
            k_sc["nf4_mean"] = None
            k_sc["zp_mode"], k_sc["rope_theta"] = "bias", float(rope_theta)
        else:
            k_arr["nf4_mean"] = np.ascontiguousarray(mean)
    if block.get("outlier_idx") is not None:
        k_arr["outlier_idx"] = np.ascontiguousarray(block["outlier_idx"], dtype=np.int32)
        k_arr["outlier_val"] = np.ascontiguousarray(block["outlier_val"]).view(np.float16)
    else:
        k_sc["outlier_idx"] = k_sc["outlier_val"] = None
    v_arr = {"indices": np.ascontiguousarray(block["value_indices"]),
             "norms": np.ascontiguousarray(block["value_norms"], dtype=np.float32)}
    v_sc = {"bits": int(block["value_bits"]), "original_dtype": _dtype("float32"),
            "packed": True, "n_values": int(np.prod(shape)), "shape": _tuple(shape)}
    header = {"codec": CODEC, "shape": list(shape), "dtype": str(dtype),
              "num_tokens": shape[2], "head_dim": shape[3], "n_heads": shape[1],
              "key_scalars": k_sc, "value_scalars": v_sc}
    return _write_npz({"__header__": np.frombuffer(json.dumps(header).encode(), dtype=np.uint8),
                       **{f"k.{n}": a for n, a in k_arr.items()},
                       **{f"v.{n}": a for n, a in v_arr.items()}})


# ---- the archive ---------------------------------------------------------------------------
# A blob is what np.savez writes: a zip archive of stored (uncompressed) .npy members.  zipfile and
# the .npy header parser spend several times longer on the nine small headers of a block than the
# checksums and copies of its 280 KB take, so the plain form is written and read by the record
# layouts of the zip format (PKWARE's APPNOTE, 4.3): by the library's csrc/archive.cu, in Python
# where the library has not been built.  Everything else is left to numpy.
_LOCAL = struct.Struct("<4s5H3L2H")       # local file header
_CENTRAL = struct.Struct("<4s6H3L5H2L")   # central directory entry
_END = struct.Struct("<4s4H2LH")          # end of central directory
_ZIP64 = struct.Struct("<2H2Q")           # extra field with 64-bit sizes
_MEMBERS = 64                             # most members the library is asked for
_NPY = re.compile(rb"\{'descr': '([<|][a-z][0-9]+)', 'fortran_order': False, "
                  rb"'shape': \(((?:[0-9]+,(?: [0-9]+,)*(?: [0-9]+)?)?)\), \} *\n")


@functools.lru_cache(maxsize=256)
def _npy_header(descr: str, shape: tuple) -> bytes:
    buf = io.BytesIO()
    np.lib.format.write_array_header_1_0(
        buf, {"descr": descr, "fortran_order": False, "shape": shape})
    return buf.getvalue()


@functools.lru_cache(maxsize=256)
def _npy_parse(head: bytes):
    """Element type and shape a .npy header (magic and length included) gives, ``None`` for another
    form than the plain one."""
    head = _NPY.fullmatch(head[10:])
    if head is None:
        return None
    shape = tuple(int(x) for x in head[2].split(b",") if x.strip())
    try:
        dtype = np.dtype(head[1].decode())
    except TypeError:
        return None
    return None if dtype.hasobject else (dtype, shape)


@functools.lru_cache(maxsize=1)
def _native():
    """The built library, ``None`` where there is none."""
    from . import _lib

    try:
        return _lib.load()
    except (RuntimeError, OSError, AttributeError):
        return None


# (a function object of its own: the attributes of ctypes.pythonapi belong to the whole process)
_new_bytes = ctypes.PYFUNCTYPE(ctypes.py_object, ctypes.c_void_p, ctypes.c_ssize_t)(
    ("PyBytes_FromStringAndSize", ctypes.pythonapi))


def _address(a) -> int:
    return a.__array_interface__["data"][0]


def _write_native(lib, arrays: dict) -> bytes:
    text, parts, size = [], [], _END.size
    for name, a in arrays.items():
        file, head = (name + ".npy").encode("ascii"), _npy_header(a.dtype.str, a.shape)
        text += [file, head]
        parts += [len(file), len(head), _address(a), a.nbytes]
        size += _LOCAL.size + _ZIP64.size + _CENTRAL.size + 2 * len(file) + len(head) + a.nbytes
    out = _new_bytes(None, size)  # (filled before anyone else sees it)
    if lib.tq_npz_write(len(arrays), (ctypes.c_int64 * len(parts))(*parts), b"".join(text),
                        ctypes.cast(ctypes.c_char_p(out), ctypes.c_void_p), size) != size:
        raise RuntimeError("the archive could not be written")
    return out


def _read_native(lib, blob, max_bytes: int, copy: bool):
    raw = np.frombuffer(blob, dtype=np.uint8)
    table = (ctypes.c_int64 * (6 * _MEMBERS))()
    view, members, used = memoryview(raw), {}, 0
    for i in range(lib.tq_npz_read(_address(raw), raw.size, _MEMBERS, table)):
        name_at, n_name, head_at, n_head, at, n = table[6 * i:6 * i + 6]
        file = bytes(view[name_at:name_at + n_name])
        form = _npy_parse(bytes(view[head_at:head_at + n_head]))
        used += n_head + n
        if form is None or not file.isascii() or not file.endswith(b".npy") or used > max_bytes \
                or form[0].itemsize * math.prod(form[1]) != n:
            return None
        name = file[:-4].decode()
        if name in members:
            return None
        a = raw[at:at + n].view(form[0]).reshape(form[1])
        members[name] = a if form[0] == np.uint8 and not copy else a.copy()
    return members or None


def _write_npz(arrays: dict) -> bytes:
    """The bytes np.savez writes for these arrays."""
    if any(a.dtype.hasobject or not a.flags.c_contiguous for a in arrays.values()) \
            or sum(a.nbytes for a in arrays.values()) >= 1 << 30:
        buf = io.BytesIO()
        np.savez(buf, **arrays)
        return buf.getvalue()
    if (lib := _native()) is not None:
        return _write_native(lib, arrays)
    out, central, at = [], [], 0
    for name, a in arrays.items():
        file = (name + ".npy").encode("ascii")
        head = _npy_header(a.dtype.str, a.shape)
        data = a.reshape(-1).view(np.uint8) if a.size else b""
        crc = zlib.crc32(data, zlib.crc32(head))
        size = len(head) + a.nbytes
        # version 4.5 (64-bit sizes in the extra field), stored, dated 1980-01-01
        local = _LOCAL.pack(b"PK\3\4", 45, 0, 0, 0, 33, crc, 0xFFFFFFFF, 0xFFFFFFFF, len(file), 20)
        out += [local, file, _ZIP64.pack(1, 16, size, size), head, data]
        # (written on a Unix system, readable and writable by the owner)
        central += [_CENTRAL.pack(b"PK\1\2", 3 << 8 | 45, 45, 0, 0, 0, 33, crc, size, size,
                                  len(file), 0, 0, 0, 0, 0o600 << 16, at), file]
        at += _LOCAL.size + len(file) + _ZIP64.size + size
    n_central = sum(len(c) for c in central)
    end = _END.pack(b"PK\5\6", 0, 0, len(arrays), len(arrays), n_central, at, 0)
    return b"".join(out + central + [end])


def _read_npz(blob: bytes, max_bytes: int, copy: bool = True):
    """The members of an archive of the plain form above, ``{name: array}``; ``None`` for any other
    one (and for one that is damaged): numpy then reads it, or says what is wrong.  Without ``copy``
    the members of bytes may be views of the blob."""
    if len(blob) < _END.size:
        return None
    if (lib := _native()) is not None:
        return _read_native(lib, blob, max_bytes, copy)
    end = len(blob) - _END.size
    sig, disk, disk_c, here, total, n_central, first, comment = _END.unpack_from(blob, end)
    if sig != b"PK\5\6" or disk or disk_c or here != total or comment or first + n_central != end:
        return None
    view, members, at, used = memoryview(blob), {}, first, 0
    for _ in range(total):
        if at + _CENTRAL.size > end:
            return None
        (sig, _, _, flags, method, _, _, crc, packed, size, n_file, n_extra, n_comment, _, _, _,
         local) = _CENTRAL.unpack_from(blob, at)
        file = bytes(view[at + _CENTRAL.size:at + _CENTRAL.size + n_file])
        at += _CENTRAL.size + n_file
        if sig != b"PK\1\2" or flags or method or packed != size or size == 0xFFFFFFFF or n_extra \
                or n_comment or not file.isascii() or not file.endswith(b".npy") or at > end \
                or local + _LOCAL.size > first:
            return None
        (sig, _, flags, method, _, _, crc_l, _, _, n_file_l, n_extra_l) = _LOCAL.unpack_from(blob, local)
        start = local + _LOCAL.size
        if sig != b"PK\3\4" or flags or method or crc_l != crc \
                or bytes(view[start:start + n_file_l]) != file:
            return None
        start += n_file_l + n_extra_l
        if start + size > first or size < 10:
            return None
        data = view[start:start + size]
        n_head = int.from_bytes(data[8:10], "little")
        if bytes(data[:8]) != b"\x93NUMPY\x01\x00" or 10 + n_head > size or zlib.crc32(data) != crc:
            return None
        form = _npy_parse(bytes(data[:10 + n_head]))
        if form is None or form[0].itemsize * math.prod(form[1]) != size - 10 - n_head:
            return None
        dtype, shape = form
        name = file[:-4].decode()
        used += size
        if name in members or used > max_bytes:
            return None
        members[name] = np.frombuffer(data[10 + n_head:], dtype=dtype).reshape(shape).copy()
    return members if at == end else None


def _scalars(d: dict) -> dict:
    out = {}
    for name, v in d.items():
        if isinstance(v, dict) and "__dtype__" in v:
            out[name] = np.dtype(v["__dtype__"])
        elif isinstance(v, dict) and "__tuple__" in v:
            out[name] = tuple(v["__tuple__"])
        else:
            out[name] = v
    return out


def blob_to_block(blob: bytes, max_bytes: int = 1 << 30) -> dict:
    """Parse one blob: ``{"header": {...}, "key": {field: array or scalar}, "value": {...}}``.

    Raises ``ValueError`` for a blob or a decompressed payload above ``max_bytes``, for a
    codec string other than ``tqp-kv-npz/1`` and for array dtypes outside the numeric
    whitelist (object arrays cannot be loaded at all: ``allow_pickle=False``).
    """
    return _parse(blob, max_bytes)


def _parse(blob: bytes, max_bytes: int = 1 << 30, copy: bool = True) -> dict:
    if len(blob) > max_bytes:
        raise ValueError(f"blob exceeds max_bytes ({len(blob)} > {max_bytes})")
    members = _read_npz(blob, max_bytes, copy)
    with contextlib.nullcontext(members) if members is not None else \
            np.load(io.BytesIO(blob), allow_pickle=False) as z:
        names = list(z) if members is not None else z.files
        if "__header__" not in names:
            raise ValueError("not a KV block blob: no header")
        header = json.loads(bytes(z["__header__"]).decode())
        if header.get("codec") != CODEC:
            raise ValueError(f"unknown record codec {header.get('codec')!r}; this reader "
                             f"handles {CODEC!r} only")
        total = 0
        key, value = {}, {}
        for name in names:
            if name == "__header__":
                continue
            a = z[name]
            if not _allowed(a.dtype):
                raise ValueError(f"dtype {a.dtype} of {name} is not allowed")
            total += a.nbytes
            if total > max_bytes:
                raise ValueError("decompressed size exceeds max_bytes")
            if name.startswith("k."):
                key[name[2:]] = a
            elif name.startswith("v."):
                value[name[2:]] = a
            else:
                raise ValueError(f"unexpected member {name!r}")
    key.update(_scalars(header["key_scalars"]))
    value.update(_scalars(header["value_scalars"]))
    meta = {k: header[k] for k in ("codec", "shape", "dtype", "num_tokens", "head_dim", "n_heads")}
    meta["shape"] = tuple(meta["shape"])
    return {"header": meta, "key": key, "value": value}


def block_from_parsed(parsed: dict, *, key_mode: str = "nf4_asym", mean_mask=None,
                      bias_means=None, geom=None) -> dict:
    """The arrays of ``KVContext.import_block`` from the result of :func:`blob_to_block`.

    The key scalars are brought back to one full ``(1, H, D)`` scale and zero-point: the
    uniform grid's ``scale`` / ``zero``; symmetric NF4 with zeros; the ``sparse`` zero-point
    scattered to the ``mean_mask`` channels; the ``bias`` zero-point from ``bias_means``
    ``(H, D)`` (the blob stores none: the reader recomputes it from the model's k-bias, the
    block's first position and ``rope_theta``).  ``geom`` ``(H, S, D, value_bits)``, when given,
    is checked against the blob's header.
    """
    key, value, meta = parsed["key"], parsed["value"], parsed["header"]
    _, h, s, d = meta["shape"]
    if geom is not None and (h, s, d, int(value["bits"])) != tuple(geom):
        raise ValueError(f"blob holds a block of (H, S, D, value_bits) = "
                         f"{(h, s, d, int(value['bits']))}, the context expects {tuple(geom)}")
    if int(key["bits"]) != 4 or not key.get("packed", True) or not value.get("packed", True):
        raise ValueError("only packed blocks with 4-bit keys can be imported")
    uniform = "scale" in key and key.get("nf4_scale") is None
    if uniform != (key_mode == "uniform"):
        raise ValueError("the blob's key grid differs from the context's key_mode")
    if uniform:
        scale = np.asarray(key["scale"], np.float32).reshape(1, h, d)
        mean = np.asarray(key["zero"], np.float32).reshape(1, h, d)
    else:
        scale = np.asarray(key["nf4_scale"], np.float32).reshape(1, h, d)
        zp = key.get("zp_mode", "calibrated")
        stored = key.get("nf4_mean")
        if key_mode == "nf4":
            if stored is not None:
                raise ValueError("the blob holds key means, the context is symmetric NF4")
            mean = np.zeros((1, h, d), np.float32)
        elif zp == "sparse":
            if mean_mask is None:
                raise ValueError("a sparse zero-point needs the context's channel mask")
            mask = np.asarray(mean_mask, bool)
            stored = np.asarray(stored, np.float32)
            if stored.shape[-1] != int(mask.sum()):
                raise ValueError("the blob's sparse means do not match the channel mask")
            mean = np.zeros((1, h, d), np.float32)
            mean[:, :, mask] = stored.reshape(1, h, -1)
        elif zp == "bias":
            if bias_means is None:
                raise ValueError("a bias zero-point stores no means: pass bias_means")
            mean = np.asarray(bias_means, np.float32).reshape(1, h, d)
        else:
            if stored is None:
                raise ValueError("the blob holds no key means, the context expects them")
            mean = np.asarray(stored, np.float32).reshape(1, h, d)
    oidx = key.get("outlier_idx")
    return {
        "key_indices": np.asarray(key["indices"], np.uint8), "nf4_scale": scale, "nf4_mean": mean,
        "outlier_idx": None if oidx is None else np.asarray(oidx, np.int32),
        "outlier_val": None if oidx is None else np.asarray(key["outlier_val"]),
        "value_indices": np.asarray(value["indices"], np.uint8),
        "value_norms": np.asarray(value["norms"], np.float32),
        "shape": (1, h, s, d), "key_bits": 4, "value_bits": int(value["bits"]),
    }
