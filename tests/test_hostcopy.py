"""Staged host copies (hostcopy.cu) over a CUDA runtime of host threads
(hostcopy_fake.cpp): every shape of copy, callers at once, and who holds the
page-locked buffers while a stream is busy."""
import ctypes
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "deconwolf_b200", "csrc")
MIB = 1 << 20
WAIT = 60.0


def _cuda_include():
    for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda"):
        if d and os.path.isfile(os.path.join(d, "include", "cuda_runtime.h")):
            return os.path.join(d, "include")
    return None


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = _cuda_include()
    if not shutil.which("g++") or not inc:
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("hostcopy") / "hostcopy.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", f"-I{inc}", f"-I{CSRC}", "-x", "c++",
                    os.path.join(CSRC, "hostcopy.cu"), os.path.join(HERE, "hostcopy_fake.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    vp, sz = ctypes.c_void_p, ctypes.c_size_t
    for f in ("fake_stream", "fake_gate"):
        getattr(L, f).restype = vp
    for f in ("fake_staged", "fake_driver"):
        getattr(L, f).restype = ctypes.c_longlong
    for f in ("fake_stream_end", "fake_gate", "fake_open", "fake_sync"):
        getattr(L, f).argtypes = [vp]
    L.to_device.argtypes = [vp, sz, vp, sz, sz, vp]
    L.to_host.argtypes = [vp, vp, sz, vp]
    return L


@pytest.fixture
def streams(lib):
    made = [lib.fake_stream() for _ in range(2)]
    yield made
    for s in made:
        lib.fake_stream_end(s)
    lib.release()


def _bytes(n, seed):
    return np.random.default_rng(seed).integers(0, 255, n, dtype=np.uint8)


# row bytes, rows, device pitch, whether the copy is staged: ragged rows, whole
# pieces and a remainder, exactly the least size, below it, rows longer than a buffer
@pytest.mark.parametrize("row,rows,pitch,staged", [
    (4 * 301, 260 * 31, 4 * 304, True), (4 * 701, 601 * 3, 4 * 704, True), (4096, 1024, 4096, True),
    (4 * MIB + 4 * 777, 1, 4 * MIB + 4 * 777, True), (4 * MIB, 1, 4 * MIB, True), (4 * MIB - 4, 1, 4 * MIB - 4, False),
    (4 * 301, 300, 4 * 304, False), (2 * MIB + 4, 4, 2 * MIB + 16, False)])
def test_copies_of_every_shape(lib, streams, row, rows, pitch, staged):
    a = _bytes(row * rows, 1)
    dev = np.zeros(pitch * rows, dtype=np.uint8)
    s0 = lib.fake_staged()
    assert lib.to_device(dev.ctypes.data, pitch, a.ctypes.data, row, rows, streams[0]) == 0
    lib.fake_sync(streams[0])
    np.testing.assert_array_equal(dev.reshape(rows, pitch)[:, :row], a.reshape(rows, row))
    assert not dev.reshape(rows, pitch)[:, row:].any()
    assert (lib.fake_staged() > s0) == staged
    s0 = lib.fake_staged()
    back = np.zeros_like(dev)
    assert lib.to_host(back.ctypes.data, dev.ctypes.data, dev.nbytes, streams[0]) == 0
    lib.fake_sync(streams[0])
    np.testing.assert_array_equal(back, dev)
    assert (lib.fake_staged() > s0) == (dev.nbytes // 4096 * 4096 >= 4 * MIB)


def test_two_callers_at_once(lib, streams):
    src = [_bytes(24 * MIB + 12, 7 + i) for i in range(2)]
    dev = [np.zeros_like(a) for a in src]
    out = [np.zeros_like(a) for a in src]

    def work(i):
        for _ in range(4):
            lib.to_device(dev[i].ctypes.data, src[i].nbytes, src[i].ctypes.data, src[i].nbytes, 1, streams[i])
            lib.to_host(out[i].ctypes.data, dev[i].ctypes.data, src[i].nbytes, streams[i])
            lib.fake_sync(streams[i])

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in th]
    [t.join(WAIT) for t in th]
    assert not any(t.is_alive() for t in th)
    for i in range(2):
        np.testing.assert_array_equal(out[i], src[i])


@pytest.mark.parametrize("upload", [False, True])
def test_a_busy_stream_does_not_hold_the_buffers(lib, streams, upload):
    """A copy behind a long queue on its stream leaves the page-locked buffers
    to others until the queue has run."""
    a, dev, back = _bytes(16 * MIB, 3), _bytes(16 * MIB, 4), np.zeros(16 * MIB, dtype=np.uint8)
    gate = lib.fake_gate(streams[0])
    if upload:
        t = threading.Thread(target=lib.to_device, args=(back.ctypes.data, a.nbytes, a.ctypes.data, a.nbytes, 1, streams[0]))
    else:
        t = threading.Thread(target=lib.to_host, args=(back.ctypes.data, a.ctypes.data, a.nbytes, streams[0]))
    t.start()
    t.join(0.5)
    assert t.is_alive()  # waits for its stream
    free = threading.Thread(target=lib.release)
    free.start()
    free.join(5.0)
    held = free.is_alive()
    d0, s0 = lib.fake_driver(), lib.fake_staged()
    other = np.zeros_like(dev)
    lib.to_device(other.ctypes.data, dev.nbytes, dev.ctypes.data, dev.nbytes, 1, streams[1])
    lib.fake_sync(streams[1])
    through = lib.fake_staged() > s0 and lib.fake_driver() == d0
    lib.fake_open(gate)
    t.join(WAIT)
    free.join(WAIT)
    lib.fake_sync(streams[0])
    assert not held and through
    np.testing.assert_array_equal(other, dev)
    np.testing.assert_array_equal(back, a)
