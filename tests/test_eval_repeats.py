"""Seven cards of which some repeat: the evaluator's header on the host, and
the kernels of few and of many hands, against the reference's score.  A rank
held five times or more without a flush is left out: it scores as four."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

_SRC = r"""
#include "mtt_device.cuh"
extern "C" void score(const uint8_t* c, uint32_t* s7, uint32_t* planes, long n) {
    for (long i = 0; i < n; ++i) {
        s7[i] = mtt::score7(c + 7 * i);
        mtt::Planes p;
        mtt::planes_clear(p);
        for (int k = 0; k < 7; ++k) mtt::planes_add(p, c[7 * i + k]);
        planes[i] = mtt::score_planes(p);
    }
}
"""


def _hands(n, seed):
    """Repeats of every kind: free draws, one suit, few cards, one card seven times."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 52, (n, 7))
    one = rng.integers(0, 13, (n, 7)) * 4 + rng.integers(0, 4, (n, 1))
    few = rng.integers(0, 52, (n, 3))[np.arange(n)[:, None], rng.integers(0, 3, (n, 7))]
    same = np.repeat(np.arange(52), 7).reshape(52, 7)
    h = np.concatenate([a, one, few, same]).astype(np.uint8)
    five = lambda v: (np.sort(v, axis=1)[:, 4:] == np.sort(v, axis=1)[:, :3]).any(axis=1)
    return h[five(h & 3) | ~five(h >> 2)]


def test_host_scores_of_repeated_cards(orc, tmp_path):
    src, lib = tmp_path / "s.cpp", tmp_path / "s.so"
    src.write_text(_SRC)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-x", "c++", str(src), "-o", str(lib),
                    "-I" + os.path.join(ROOT, "mtt-gpu-solver_b200", "csrc"), "-I" + os.path.join(CUDA, "include")],
                   check=True, capture_output=True)
    h = _hands(20000, 1)
    want = orc.eval7(h)
    out = [np.zeros(len(h), np.uint32) for _ in range(2)]
    ctypes.CDLL(str(lib)).score(h.ctypes.data_as(ctypes.c_void_p), *[o.ctypes.data_as(ctypes.c_void_p) for o in out],
                                ctypes.c_long(len(h)))
    assert all(np.array_equal(o, want) for o in out)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 20001])
def test_gpu_scores_of_repeated_cards(mtt, orc, cuda, n):
    import torch
    h = np.ascontiguousarray(_hands(20000, 2)[-n:])
    got = mtt.eval7(torch.from_numpy(h).to(cuda)).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, orc.eval7(h))
