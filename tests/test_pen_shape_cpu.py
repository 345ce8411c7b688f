"""The penalty operator's launch shapes (host arithmetic): on devices of any
number of SMs the resident kernel's blocks are no more than the device holds of
the form they take, since a cooperative launch beyond that is refused; on 152
SMs the shapes are those the kernels were measured with."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mphimplicit_gb300", "csrc")
SRC = """
#include "mph_shapes.h"
extern "C" void shape(int N, int min_rows, int pair, int single, int fit, int* out)
{
    const mph::PenShape S = mph::pen_shape_for(N, min_rows, 512, pair, single, [fit](int r) { return r <= fit; });
    out[0] = S.rows; out[1] = S.w; out[2] = S.resident; out[3] = S.alone;
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "s.cpp"), "-o", str(d / "s.so")], check=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def get(*a):
        out = (ctypes.c_int * 4)()
        lib.shape(*a, out)
        return list(out)
    return get


SIZES = [1, 31, 5000, 28417, 29184, 29185, 56833, 58368, 58369, 76000, 77824, 77825, 155648, 155649, 1297696]


@pytest.mark.parametrize("sms", [1, 20, 76, 132, 147, 148, 151, 152, 160])
@pytest.mark.parametrize("min_rows", [192, 384])
def test_blocks_fit_the_device(shape, sms, min_rows):
    pair, single = min(2 * sms, 304), min(sms, 152)
    for n in SIZES:
        for fit in (512, 320, 128):
            for p, s in ((pair, single), (0, single), (pair, 0), (0, 0)):
                rows, w, resident, alone = shape(n, min_rows, p, s, fit)
                blocks = -(-n // rows)
                assert rows % 32 == 0 and 32 <= rows * w <= 512
                if resident:
                    assert rows <= fit and blocks <= (s if alone else p)
                else:
                    assert rows * w == 256


def test_shapes_of_152_sms(shape):
    for n, want in ((12148, [384, 1, 1, 1]), (22304, [192, 2, 1, 1]), (33576, [224, 2, 1, 1]), (77824, [512, 1, 1, 1]),
                    (77825, [288, 1, 1, 0]), (155103, [512, 1, 1, 0]), (155649, [256, 1, 0, 0])):
        assert shape(n, 384 if n == 12148 else 192, 304, 152, 512) == want, n
    assert shape(22304, 192, 304, 152, 100) == [64, 4, 0, 0]   # lists too long for shared memory
