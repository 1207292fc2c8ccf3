"""Row chunks of the backward kernels with sixteen columns per lane: the function of the source, compiled by
itself for 148 SMs."""
import ctypes
import os
import re
import shutil
import subprocess
import time

import pytest

import slapo_b200

SOURCE = os.path.join(os.path.dirname(slapo_b200.__file__), "csrc", "elementwise.cu")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if shutil.which(cxx) is None:
        pytest.skip("no host compiler")
    with open(SOURCE) as f:
        text = f.read()
    body = "".join(re.search(r"^(?:static )?int %s\(.*?^}\n" % name, text, re.S | re.M).group(0)
                   for name in ("colsum_chunks", "wave_chunks", "slab_chunks"))
    at = tmp_path_factory.mktemp("slab")
    with open(at / "slab.cpp", "w") as f:
        f.write("#include <cstdint>\nstatic int sm_count() { return 148; }\n" + body +
                'extern "C" int chunks(int r, int c, int per) { return slab_chunks(r, c, per); }\n'
                'extern "C" int most(int r, int c) { return colsum_chunks(r, c); }\n'
                'extern "C" long many(int n, int r, int c) {\n'
                "  long s = 0;\n  for (int i = 0; i < n; ++i) s += slab_chunks(r + 8 * (i & 63), c, 2);\n"
                "  return s;\n}\n")
    out = str(at / "slab.so")
    subprocess.run([cxx, "-O2", "-shared", "-fPIC", "-o", out, str(at / "slab.cpp")], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("per_sm", [2, 4])
def test_whole_waves(host, per_sm):
    resident = 148 * per_sm
    for cols in (16, 256, 1024, 1536, 2048, 4096, 8192, 10240, 30528, 50304, 131072, 400000):
        slabs = -(-cols // 256)
        for rows in (64, 300, 1024, 2048, 8192, 16384, 100000):
            c = host.chunks(rows, cols, per_sm)
            assert 1 <= c <= host.most(rows, cols)
            waves = -(-c * slabs // resident)
            # no more of a last wave than rounding the chunks down leaves empty, but where rows or slabs are
            # the limit
            assert c == host.most(rows, cols) or slabs > resident or (c + 1) * slabs > waves * resident \
                or c == 148 * 8 // slabs


@pytest.mark.parametrize("rows,cols,waves", [
    (8192, 1024, 1), (1024, 8192, 1), (819, 10240, 1), (65536, 256, 1), (274, 30528, 1), (1099, 30528, 3),
    (1334, 50304, 2)])
def test_one_wave_unless_much_of_it_is_empty(host, rows, cols, waves):
    assert -(-host.chunks(rows, cols, 2) * -(-cols // 256) // 296) == waves


def test_costs_the_host_next_to_nothing(host):
    """A search through all numbers of chunks took 3.4 us a call for 256 columns; a hundredth of that here."""
    best = 1.0
    for _ in range(5):
        start = time.perf_counter()
        host.many(10000, 65536, 256)
        best = min(best, (time.perf_counter() - start) / 10000)
    assert best < 5e-7
