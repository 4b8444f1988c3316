"""Host paths that one GPU cannot show, against a stand-in for libcudart with two
devices (cpp/fake_cudart.cpp; no GPU): the library in a process of its own, whose loader finds
the stand-in first.
"""
import os
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent
PKG = TESTS.parent / "bd-cudatag_gb300"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))

PRELUDE = """
import ctypes, sys, threading, time
sys.path.insert(0, %r)
import numpy as np
import bdcudatag
L = bdcudatag.lib()

def device_frame(w, h):
    p = ctypes.c_void_p()
    assert L.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(w * h)) == 0
    return p.value

def frame(w, h, first=0, pad=0):
    f = np.zeros((h, w + pad), np.uint8)
    f[0, 0] = first
    return f
""" % str(PKG)


@pytest.fixture(scope="module")
def stand_in(tmp_path_factory):
    folder = tmp_path_factory.mktemp("cudart")
    versions = folder / "versions"
    versions.write_text("libcudart.so.13 { global: *; };\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{CUDA / 'include'}",
                    str(TESTS / "cpp" / "fake_cudart.cpp"), f"-Wl,--version-script={versions}",
                    "-Wl,-soname,libcudart.so.13", "-o", str(folder / "libcudart.so.13"), "-lpthread"], check=True)
    return folder


def run(stand_in, script):
    env = dict(os.environ, LD_LIBRARY_PATH=str(stand_in))
    env.pop("LD_PRELOAD", None)
    done = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(script)], env=env, capture_output=True,
                          text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr


@pytest.mark.parametrize("graph", [0, 1])
def test_other_current_device(stand_in, graph):
    """A plan of device 0 called from a thread whose current device is 1: its graphs
    run (no launches beside them), and the thread's device stays as it was."""
    run(stand_in, f"""
        batch = bdcudatag.Batch([(640, 480, 3), (320, 240, 1)], bdcudatag.default_config(use_cuda_graph={graph}))
        server = bdcudatag.Server([(640, 480, 3)])
        assert L.cudaSetDevice(1) == 0
        for _ in range(3):
            batch.detect([device_frame(640, 480), device_frame(320, 240)], [640, 320], device=True)
            batch.detect([frame(640, 480), frame(320, 240)])
            assert server.wait(server.submit(0, frame(640, 480)))[0] == 1
        assert (L.fake_launches() == 0) == ({graph} == 1)
        now = ctypes.c_int(-1)
        assert L.cudaGetDevice(ctypes.byref(now)) == 0 and now.value == 1
    """)


def test_submits_do_not_wait_for_each_other(stand_in):
    """While one thread's copy takes 400 ms, another camera's and another frame of the same
    camera are submitted, and a copy that fails is reported by its own submit."""
    run(stand_in, """
        server = bdcudatag.Server([(1920, 1080, 1), (640, 480, 1)], queue_depth=4)
        L.fake_slow(400)
        slow, failing = frame(1920, 1080, first=200), frame(640, 480, first=100)
        tickets = []
        thread = threading.Thread(target=lambda: tickets.append(server.submit(0, slow)))
        thread.start()
        time.sleep(0.1)
        for camera, f in ((1, frame(640, 480)), (0, frame(1920, 1080))):
            before = time.perf_counter()
            ticket = server.submit(camera, f)
            assert time.perf_counter() - before < 0.2
            assert ticket >= 0 and server.wait(ticket)[0] == 1
        assert server.submit(1, failing) == bdcudatag.ERROR_CUDA
        thread.join()
        assert server.wait(tickets[0])[0] == 1
        assert server.wait(server.submit(1, frame(640, 480)))[0] == 1
        server.close()
        assert L.fake_streams() == 0
    """)


def test_strided_submits_to_a_server(stand_in):
    """Rows with a gap: small frames through page-locked memory, as a batch takes them, large
    ones by the copy engine."""
    run(stand_in, """
        server = bdcudatag.Server([(640, 480, 1), (1920, 1080, 1)])
        L.fake_slow(300)
        before = time.perf_counter()
        assert server.wait(server.submit(0, frame(640, 480, first=200, pad=7), 647))[0] == 1
        assert time.perf_counter() - before < 0.2  # the copy engine would have taken 300 ms
        before = time.perf_counter()
        assert server.wait(server.submit(1, frame(1920, 1080, first=200, pad=7), 1927))[0] == 1
        assert time.perf_counter() - before >= 0.3
    """)


def test_refused_copies_are_staged(stand_in):
    """Pageable frames whose direct copy the runtime refuses go through page-locked memory, in
    a batch beside a page-locked one and in a server; no error is left behind."""
    run(stand_in, """
        batch = bdcudatag.Batch([(640, 480, 3), (320, 240, 1), (640, 480, 1)])
        server = bdcudatag.Server([(640, 480, 3)])
        p = ctypes.c_void_p()
        assert L.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(640 * 480), 0) == 0
        L.fake_refuse(1)
        before = L.fake_copies_from_page_locked()
        batch.detect([frame(640, 480), frame(320, 240), p.value], [640, 320, 640])
        assert L.fake_copies_from_page_locked() == before + 3
        for _ in range(20):  # streams are given back
            assert server.wait(server.submit(0, frame(640, 480)))[0] == 1
        assert L.fake_copies_from_page_locked() == before + 23
        assert L.cudaGetLastError() == 0
    """)


def test_errors_of_earlier_calls(stand_in):
    """An error that the caller's thread left behind does not fail a submit of pageable
    frames."""
    run(stand_in, """
        batch = bdcudatag.Batch([(640, 480, 3), (320, 240, 1)])
        for frames in ([frame(640, 480), frame(320, 240)], [frame(640, 480, pad=7), frame(320, 240, pad=7)]):
            assert L.cudaSetDevice(99) != 0
            batch.detect(frames)
    """)


def test_pageable_frames_of_a_batch(stand_in):
    """Several pageable frames: small ones are staged, larger ones are all queued before
    one wait; a frame alone is copied direct at any size."""
    run(stand_in, """
        for size, count, direct in ((64, 1, 1), (320, 16, 0), (1024, 5, 5)):
            batch = bdcudatag.Batch([(size, size * 3 // 4, 1)] * count)
            copies, waits = L.fake_direct_copies(), L.fake_waits()
            batch.detect([frame(size, size * 3 // 4) for _ in range(count)])
            assert L.fake_direct_copies() - copies == direct
            assert L.fake_waits() - waits == min(direct, 1)
        mixed = bdcudatag.Batch([(160, 120, 1), (1024, 768, 1)])
        copies = L.fake_direct_copies()
        mixed.detect([frame(160, 120), frame(1024, 768)])
        assert L.fake_direct_copies() - copies == 1
    """)
