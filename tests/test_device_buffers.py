"""DevBuf, the device buffers that packet lists are kept in: how often it
allocates when sizes change from step to step, and how much it may hold."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("devbuf") / "devbuf.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "devbuf_host.cu")], check=True)
    f = C.CDLL(so).devbuf_run
    f.argtypes = [C.c_void_p, C.c_int, C.c_longlong, C.c_void_p]

    def call(sizes, limit=0):
        s = np.array(sizes, np.int64)
        out = np.zeros(4, np.int64)
        assert f(s.ctypes.data, s.size, limit, out.ctypes.data) == 0
        return dict(zip(("allocs", "held", "most", "refused"), out.tolist()))

    return call


@pytest.mark.parametrize("swing", [0.001, 0.016, 0.05, 0.15])
def test_sizes_that_swing_settle(run, swing):
    """Packet counts that rise and fall by some percent, from the smaller size
    on: after the first growth the buffer stays."""
    n = 1_000_000
    assert run([int(n * (1 - swing)), n] * 20)["allocs"] <= 2
    rng = np.random.default_rng(1)
    assert run(rng.integers(int(n * (1 - swing)), n, 200).tolist())["allocs"] <= 4


def test_a_falling_count_gives_memory_back(run):
    """Packets escape step by step: few allocations, and what is held stays
    within 4/3 of what is used."""
    n, sizes = 1_000_000, []
    while n > 1000:
        sizes.append(n)
        n = int(n * 0.97)
    for k in range(1, len(sizes), 7):
        assert run(sizes[:k])["held"] <= 8 * sizes[k - 1] * 4 / 3 + 64
    assert run(sizes)["allocs"] <= 30


def test_large_buffers_are_exact(run):
    """From 1 GiB on a buffer has the size asked for."""
    g = (1 << 30) // 8
    r = run([g + 1, g + 100, g + 50, g + 2])
    assert r["allocs"] == 4 and r["held"] == 8 * (g + 2) and r["most"] == 8 * (g + 100)


def test_the_exact_size_is_taken_where_no_more_fits(run):
    assert run([1000, 2000], 8 * 2000)["refused"] == 0
    assert run([1000, 2001, 1000], 8 * 2000) == {"allocs": 2, "held": 8000, "most": 8000, "refused": 1}
    assert run([0, 10, 0])["held"] == 0
