"""The host library is not tied to one processor: its sources name no other one's instructions where that processor is not
the target, and the copy pool's plain form copies like the one it stands for."""
import ctypes as C
import glob
import os
import re
import subprocess
import time

import numpy as np
import pytest

from anemone_b200 import build

BATCH_MOST = 64


class Copy(C.Structure):
    _fields_ = [("to", C.c_void_p), ("source", C.c_void_p), ("byte_count", C.c_size_t)]


class Batch(C.Structure):
    _fields_ = [("copies", Copy * BATCH_MOST), ("count", C.c_uint32), ("next", C.c_uint32), ("allowed", C.c_uint32),
                ("done", C.c_uint32 * BATCH_MOST), ("to_device", C.c_bool), ("shared", C.c_bool), ("soon", C.c_bool)]


def test_the_batch_here_is_the_librarys(tmp_path):
    """Every field, in order, and every one's place: the library writes them all."""
    header = open(os.path.join(build.CSRC, "host", "copy_pool.h")).read()
    body = re.sub(r"/\*.*?\*/", "", re.search(r"struct ab_copy_batch \{(.*?)\};", header, flags=re.S).group(1), flags=re.S)
    names = re.findall(r"(\w+)(?:\[\w+\])?\s*[,;]", body)
    assert names == [field[0] for field in Batch._fields_]
    source = "#include <stdio.h>\n#include \"copy_pool.h\"\nint main(void){" + "".join(
        'printf("%%zu ", offsetof(struct ab_copy_batch, %s));' % name for name in names) + \
        'printf("%zu", sizeof(struct ab_copy_batch)); return 0; }'
    program = str(tmp_path / "places")
    made = subprocess.run([build.GCC, "-I" + os.path.join(build.CSRC, "host"), "-x", "c", "-", "-o", program], input=source,
                          capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    places = subprocess.run([program], capture_output=True, text=True, check=True).stdout.split()
    assert [int(place) for place in places] == [getattr(Batch, name).offset for name in names] + [C.sizeof(Batch)]


@pytest.fixture
def pool(tmp_path):
    """The pool as the library has it, with one user."""
    path = str(tmp_path / "libpool.so")
    made = subprocess.run([build.GCC] + build.GCC_FLAGS + ["-shared", "-o", path,
                          os.path.join(build.CSRC, "host", "copy_pool.c"), "-lpthread"], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    library = C.CDLL(path)
    library.ab_copy_batch_help.restype = library.ab_copy_batch_is_done.restype = C.c_bool
    library.ab_copy_pool_enter()
    yield library
    library.ab_copy_pool_leave()


def batch_of(count, size=5000):
    sources = np.random.default_rng(count).integers(0, 256, size=(count, size), dtype=np.uint8)
    targets = np.full((count, size), 0xA5, dtype=np.uint8)
    batch = Batch()
    for index in range(count):
        batch.copies[index] = Copy(targets[index].ctypes.data, sources[index].ctypes.data, size)
    batch.count = count
    return batch, sources, targets


@pytest.mark.parametrize("soon_at", [None, 0, 3])
def test_pieces_allowed_one_by_one(pool, soon_at):
    """A result's pieces as they arrive: none is made before it is allowed, each is then made by a thread of the pool (the
    caller only where there is none), the batch ends, and the pool takes the next."""
    for count in (9, 2, BATCH_MOST):
        batch, sources, targets = batch_of(count)
        pool.ab_copy_batch_begin(C.byref(batch))
        for piece in range(count):
            time.sleep(0.0005)
            assert (targets[piece:] == 0xA5).all()
            pool.ab_copy_batch_allow(C.byref(batch), piece + 1)
            if piece == soon_at:
                pool.ab_copy_batch_soon(C.byref(batch))
                assert batch.soon == batch.shared
            until = time.monotonic() + 20
            while not pool.ab_copy_batch_is_done(C.byref(batch), piece):
                if not batch.shared:
                    pool.ab_copy_batch_help(C.byref(batch))
                assert time.monotonic() < until
        pool.ab_copy_batch_end(C.byref(batch))
        assert np.array_equal(targets, sources) and not pool.ab_copy_batch_help(C.byref(batch))


@pytest.mark.parametrize("soon", [False, True])
@pytest.mark.parametrize("allowed", [0, 1, 7])
def test_a_cut_batch_makes_what_was_allowed(pool, soon, allowed):
    """After a failure in the middle of a result: what was allowed is made, the rest never, with the pool's threads looking
    out for it or not; they are free for the next batch and for the pool's end."""
    batch, sources, targets = batch_of(12)
    pool.ab_copy_batch_begin(C.byref(batch))
    pool.ab_copy_batch_allow(C.byref(batch), allowed)
    if soon:
        pool.ab_copy_batch_soon(C.byref(batch))
        time.sleep(0.002)
    pool.ab_copy_batch_cut(C.byref(batch))
    pool.ab_copy_batch_end(C.byref(batch))
    time.sleep(0.002)
    assert np.array_equal(targets[:allowed], sources[:allowed]) and (targets[allowed:] == 0xA5).all()
    following, others, copied = batch_of(BATCH_MOST)
    following.allowed = BATCH_MOST
    pool.ab_copy_batch_begin(C.byref(following))
    assert following.shared == batch.shared and not following.soon
    pool.ab_copy_batch_end(C.byref(following))
    assert np.array_equal(copied, others)


def test_two_batches_at_once(pool):
    """One batch at a time has the pool's threads; a second is made by its caller alone, with the same calls."""
    first, sources, targets = batch_of(10)
    pool.ab_copy_batch_begin(C.byref(first))
    pool.ab_copy_batch_allow(C.byref(first), 1)
    pool.ab_copy_batch_soon(C.byref(first))
    second, others, copied = batch_of(11)
    pool.ab_copy_batch_begin(C.byref(second))
    assert not (first.shared and second.shared)
    pool.ab_copy_batch_allow(C.byref(second), 4)
    pool.ab_copy_batch_soon(C.byref(second))
    assert not second.soon or second.shared
    pool.ab_copy_batch_end(C.byref(second))
    pool.ab_copy_batch_end(C.byref(first))
    assert np.array_equal(copied, others) and np.array_equal(targets, sources)


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
