"""Copies by several threads and scratch memory that calls share: large blocks whose size is no
multiple of a part, and calls of different sizes from several threads at once."""
import ctypes
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _child(*what):
    """In a process of its own: what is allocated in these threads and freed by this one would
    otherwise serve the tests after it."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), *what], cwd=root, capture_output=True, text=True,
                       timeout=300, env={**os.environ, "PYTHONPATH": root})
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("kind", ["u8", "f32"])
@pytest.mark.parametrize("size", ["2048x512", "2050x1023", "4097x1025", "8191x1024"])
def test_pageable_blocks_arrive_as_pinned_ones(size, kind):
    _child(size, kind)


def test_calls_share_scratch_between_threads():
    _child("threads")


def _blocks(ndump, nchans, kind):
    import transientx_gb300 as tx
    rt = ctypes.CDLL("libcudart.so")
    rng = np.random.default_rng(ndump)
    blocks = [rng.integers(90, 160, (ndump, nchans)).astype(np.uint8) for _ in range(4)]
    if kind == "f32":
        blocks = [b.astype(np.float32) * 0.37 for b in blocks]
    row = tx.SinglePulse(td=1, fd=1, dms=0.0, ddm=0.5, ndm=24, maxw=0.005, thre=6.0)
    f = 1500.0 - 300.0 / nchans * np.arange(nchans)
    out = []
    for pinned in (False, True):
        with tx.Search([row], nchans, 256e-6, f, ndump, flags=tx.FLAG_KEEP_SERIES, zapthre=0.0) as s:
            got = []
            for b in blocks:
                p = ctypes.c_void_p()
                if pinned:
                    assert rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(b.nbytes), 0) == 0
                    q = np.frombuffer((ctypes.c_char * b.nbytes).from_address(p.value), b.dtype).reshape(b.shape)
                    q[:] = b
                    b = q
                (s.push_block if kind == "u8" else s.push_block_f32)(b)
                s.sync()
                if pinned:
                    assert rt.cudaFreeHost(p) == 0
                if s.row_info(0).gated:
                    got.append(s.timdata(0).copy())
        out.append(got)
    assert len(out[0]) == len(out[1]) >= 1
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def _calls_from_threads():
    import transientx_gb300 as tx
    rng = np.random.default_rng(5)
    widths = tx.width_ladder(1e-4, 0.05, 0.1, 1e-4)
    sizes = [(3, 70), (40, 9001), (256, 8192), (90, 62496), (1500, 1024)]
    xs = [rng.normal(0, 20, s).astype(np.float32) for s in sizes]

    def call(x, dense):
        return tx.boxcar(x, widths, thre=3.5 if dense else 4.0, dense=dense, cand_capacity=1 << 18)

    want = [[call(x, d) for d in (False, True)] for x in xs]
    bad = []

    def work(seed):
        try:
            order = np.random.default_rng(seed).permutation(2 * len(xs))
            for k in order:
                got = call(xs[k // 2], bool(k % 2))
                for a, b in zip(got, want[k // 2][k % 2]):
                    if a is not None:
                        np.testing.assert_array_equal(a, b)
        except BaseException as e:  # noqa: BLE001 - reported by the test's thread
            bad.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[0]


if __name__ == "__main__":
    if sys.argv[1] == "threads":
        _calls_from_threads()
    else:
        _blocks(*map(int, sys.argv[1].split("x")), sys.argv[2])
