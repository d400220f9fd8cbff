"""leaf_in_range (rt_internal.cuh), the guard of a leaf's triangle range in the walks, run
on the host: a range is accepted exactly when it lies within the tree's triangles,
also where position plus count passes 2^32 or a field of an imported node is
negative."""
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include "rt_internal.cuh"
int main() {
    long long pos, cnt, n;
    while (std::scanf("%lld %lld %lld", &pos, &cnt, &n) == 3)
        std::printf("%d\n", leaf_in_range((uint32_t)(int32_t)pos, (uint32_t)(int32_t)cnt, (uint32_t)n) ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from rtgpu import build
    d = tmp_path_factory.mktemp("leaf_range")
    (d / "p.cu").write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", str(build.INCLUDE), "-I", str(build.CSRC),
                    str(d / "p.cu"), "-o", str(d / "p"), "-lcudart"], check=True, capture_output=True)
    return d / "p"


def test_leaf_in_range(program):
    edge = [-2**31, -40, -1, 0, 1, 2, 31, 32, 39, 40, 41, 4999, 5000, 5001, 2**25 - 1, 2**25, 2**28 - 1, 2**31 - 1]
    cases = [(p, c, n) for p in edge for c in edge for n in (1, 40, 5000, 2**29)]
    out = subprocess.run([str(program)], input="".join("%d %d %d\n" % c for c in cases), check=True, capture_output=True,
                         text=True).stdout.split()
    assert len(out) == len(cases)
    for (p, c, n), got in zip(cases, out):
        assert int(got) == int(p >= 0 and c >= 0 and p + c <= n), (p, c, n)
