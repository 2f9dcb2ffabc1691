"""PNG export (z2d's png_exporter, src/export_png.zig) through the GPU
encoder: z2dgpu_png_encode / z2dgpu_png_scanlines."""
from __future__ import annotations

import ctypes as C
from typing import Optional

from . import abi
from .native import check, default_context, Context


def encode(surface, color_profile: Optional[str] = None, ctx: Optional[Context] = None) -> bytes:
    """The PNG file writeToPNGFile would write for `surface` (host or
    device memory); color_profile None, "linear" or "srgb"."""
    ctx = ctx or default_context()
    out = C.POINTER(C.c_uint8)()
    n = C.c_size_t()
    s = surface.to_abi() if hasattr(surface, "to_abi") else surface
    check(ctx.lib.z2dgpu_png_encode(ctx.handle, C.byref(s), abi.PROFILE[color_profile], C.byref(out), C.byref(n)))
    try:
        return C.string_at(out, n.value)
    finally:
        ctx.lib.z2dgpu_free(out)


# a bytes object of n bytes to be filled by its creator
_new_bytes = C.pythonapi.PyBytes_FromStringAndSize
_new_bytes.restype = C.py_object
_new_bytes.argtypes = [C.c_char_p, C.c_ssize_t]
_bytes_data = C.pythonapi.PyBytes_AsString
_bytes_data.restype = C.c_void_p
_bytes_data.argtypes = [C.py_object]


def scanlines(surface, color_profile: Optional[str] = None, ctx: Optional[Context] = None) -> bytes:
    """The PNG's uncompressed image data: per row a 0 filter byte and the
    encoded pixels."""
    ctx = ctx or default_context()
    s = surface.to_abi() if hasattr(surface, "to_abi") else surface
    profile = abi.PROFILE[color_profile]
    n = C.c_size_t()
    check(ctx.lib.z2dgpu_png_scanlines_into(ctx.handle, C.byref(s), profile, None, 0, C.byref(n)))
    out = _new_bytes(None, n.value)
    check(ctx.lib.z2dgpu_png_scanlines_into(ctx.handle, C.byref(s), profile, _bytes_data(out), len(out), C.byref(n)))
    return out


def write_to_png_file(surface, filename: str, color_profile: Optional[str] = None,
                      ctx: Optional[Context] = None) -> None:
    """png_exporter.writeToPNGFile (src/export_png.zig:56-87)."""
    with open(filename, "wb") as f:
        f.write(encode(surface, color_profile, ctx))
