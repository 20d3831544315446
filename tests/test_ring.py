"""The buffer and phase that the kernels' failure paths and last waits look at, with barriers that count their phases."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infllm_b200", "csrc")


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text('#include "ring.cuh"\nextern "C" int last(int c, int n, int b) { return infllm::ring_last(c, n, b); }\n'
                                'extern "C" unsigned parity(int i, int n) { return infllm::ring_parity(i, n); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "ring.cpp"), "-o", str(d / "ring.so")])
    return ctypes.CDLL(str(d / "ring.so"))


def _passes(completed, parity):
    """mbarrier.try_wait.parity: the phase before the current one has that parity (a fresh barrier passes parity 1)."""
    return (completed - 1) & 1 == parity


@pytest.mark.parametrize("n", [2, 3, 4])
def test_waiting_for_the_last_item_of_every_buffer_is_waiting_for_all(ring, n):
    for count in range(0, 5 * n):
        # an item is asked for when the one before it in its buffer has been used: at most the last of each buffer is on its way
        for landed in range(max(0, count - n), count + 1):
            through = True
            for b in range(n):
                item = ring.last(count, n, b)
                assert item == max((i for i in range(count) if i % n == b), default=-1)
                if item >= 0:
                    through = through and _passes(sum(1 for i in range(landed) if i % n == b), ring.parity(item, n))
            assert through == (landed == count)
