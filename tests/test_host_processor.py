"""The host library is not tied to one processor: its sources name no other one's instructions where that processor is not
the target, and the copy pool's plain form copies like the one it stands for."""
import ctypes as C
import glob
import os
import subprocess

import numpy as np
import pytest

from anemone_b200 import build

BATCH_MOST = 64


class Copy(C.Structure):
    _fields_ = [("to", C.c_void_p), ("source", C.c_void_p), ("byte_count", C.c_size_t)]


class Batch(C.Structure):
    _fields_ = [("copies", Copy * BATCH_MOST), ("count", C.c_uint32), ("next", C.c_uint32), ("allowed", C.c_uint32),
                ("done", C.c_uint32 * BATCH_MOST), ("to_device", C.c_bool), ("shared", C.c_bool)]


def on_x86():
    return os.uname().machine == "x86_64"


@pytest.mark.parametrize("source", sorted(os.path.basename(path) for path in
                                          glob.glob(os.path.join(build.CSRC, "host", "*.c"))))
def test_sources_preprocess_for_another_processor(tmp_path, source):
    """As a compiler whose target is none of x86's sees them. (The C library's headers ask for a list of its stubs by word
    size, which this machine has for its own alone.)"""
    (tmp_path / "gnu").mkdir()
    (tmp_path / "gnu" / "stubs-32.h").write_text("")
    (tmp_path / "kernel_images.h").write_text("")
    gone = ["-U" + name for name in ("__x86_64__", "__x86_64", "__amd64__", "__i386__", "__SSE__", "__SSE2__")]
    command = [build.GCC] + build.GCC_FLAGS + gone + ["-E", "-I" + str(tmp_path),
                                                      os.path.join(build.CSRC, "host", source)]
    made = subprocess.run(command, capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    for name in ("emmintrin", "_mm_", "__builtin_ia32"):
        assert name not in made.stdout, name


@pytest.mark.parametrize("flags", [[], ["-mno-sse2"] if on_x86() else ["-DPLAIN"]])
def test_a_batch_copies_its_bytes(tmp_path, flags):
    """The pool's copies, past the caches and through them, with the processor's stores and without: odd addresses and
    sizes from nothing to several pieces, nothing written around them."""
    path = str(tmp_path / "libpool.so")
    made = subprocess.run([build.GCC] + build.GCC_FLAGS + flags + ["-shared", "-o", path,
                          os.path.join(build.CSRC, "host", "copy_pool.c"), "-lpthread"], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    pool = C.CDLL(path)
    pool.ab_copy_batch_help.restype = C.c_bool
    rng = np.random.default_rng(7)
    sizes = [1, 15, 16, 63, 64, 65, 79, 80, 127, 128, 4099, 1 << 20, (1 << 20) + 37, 300001]
    for to_device in (False, True):
        pool.ab_copy_pool_enter()
        sources = [rng.integers(0, 256, size=size + 64, dtype=np.uint8) for size in sizes]
        targets = [np.full(size + 64, 0xA5, dtype=np.uint8) for size in sizes]
        batch = Batch()
        for index, size in enumerate(sizes):
            batch.copies[index] = Copy(targets[index].ctypes.data + 16 + index % 7, sources[index].ctypes.data + index % 5,
                                       size)
        batch.count = batch.allowed = len(sizes)
        batch.to_device = to_device
        pool.ab_copy_batch_begin(C.byref(batch))
        while pool.ab_copy_batch_help(C.byref(batch)):
            pass
        pool.ab_copy_batch_end(C.byref(batch))
        pool.ab_copy_pool_leave()
        for index, size in enumerate(sizes):
            at = 16 + index % 7
            assert np.array_equal(targets[index][at:at + size], sources[index][index % 5:index % 5 + size])
            assert (targets[index][:at] == 0xA5).all() and (targets[index][at + size:] == 0xA5).all()
