"""The search for a tile's segment, compiled for the CPU from the header that the kernels use."""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
THREADS, ROWS = 256, 64

_HARNESS = """
#include "seg_search.cuh"
using namespace vafa::tiles;
// order: the order in which the threads of a CTA come to look.  Returns the segment, rounds through `rounds`.
extern "C" int find(const int32_t* cu, int n_seg, int stack, long long slot, int threads, const int* order, int* rounds) {
  SegSearch s(n_seg, threads);
  for (*rounds = 0; !s.done(); ++*rounds) {
    int count = 0;
    for (int t = 0; t < threads; ++t) count += s.starts_by(cu, stack, slot, order[t]);
    s.narrow(count, threads);
  }
  return (int)s.lo;
}
"""


@pytest.fixture(scope="module")
def find(tmp_path_factory):
    d = tmp_path_factory.mktemp("seg")
    (d / "h.cpp").write_text(_HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "varlenabsorbflashattn_b200", "csrc"), str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    fn = C.CDLL(str(d / "h.so")).find
    fn.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_longlong, C.c_int, C.c_void_p, C.c_void_p]

    def call(cu, stack, slot, order=range(THREADS)):
        arr, o, n = (C.c_int32 * len(cu))(*cu), (C.c_int * THREADS)(*order), C.c_int()
        return fn(arr, len(cu) - 1, stack, slot, THREADS, o, C.byref(n)), n.value
    return call


def _first(cu, i, stack):
    v = cu[i] * stack  # (the kernel divides towards zero)
    return (v // ROWS if v >= 0 else -(-v // ROWS)) + i


@pytest.mark.parametrize("n", [1, 2, 63, 255, 256, 257, 511, 512, 513, 1000, 65536, 65537])
@pytest.mark.parametrize("stack", [1, 8])
def test_every_tile_has_its_segment(find, n, stack):
    rng = random.Random(n)
    cu = [0]
    for _ in range(n):
        cu.append(cu[-1] + rng.choice((0, 0, 1, rng.randrange(200), 64, 63, 65)))
    rows = [b - a for a, b in zip(cu, cu[1:])]
    for seg in sorted({0, n - 1, *(rng.randrange(n) for _ in range(40))}):
        for t in range(-(-rows[seg] * stack // ROWS)):
            got, rounds = find(cu, stack, _first(cu, seg, stack) + t)
            assert got == seg
            assert rounds <= (0 if n == 1 else 1 if n <= THREADS else 2 if n <= THREADS ** 2 else 3)


def test_sums_that_are_no_prefix_sums_have_one_answer(find):
    """Whatever the array holds, the answer is a segment of the batch and does not depend on the order of the threads."""
    rng = random.Random(1)
    two = 0
    for trial in range(300):
        n = rng.choice((3, 70, 130, 300, 700))
        lens = [rng.randrange(1, 400) for _ in range(n)]
        at = rng.randrange(1, n)
        cu = [0]
        for i, x in enumerate(lens):
            cu.append(x if i == at else cu[-1] + x)
        if trial % 3 == 0:
            cu[rng.randrange(n)] = rng.choice((-5, 2 ** 31 - 1, -2 ** 31))
        for _ in range(4):
            slot = rng.randrange(0, 2 * n + sum(lens) // ROWS)
            two += sum(_first(cu, i, 1) <= slot < _first(cu, i + 1, 1) for i in range(n)) > 1
            order = list(range(THREADS))
            answers = set()
            for _ in range(3):
                rng.shuffle(order)
                answers.add(find(cu, 1, slot, order)[0])
            assert len(answers) == 1 and 0 <= answers.pop() < n
    assert two > 100  # slots that two segments claim: taking whichever was written last, the CTAs of a cluster could differ
