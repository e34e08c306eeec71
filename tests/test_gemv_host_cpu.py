"""Which kernel a projection of many columns goes to (bk_gemv.cu), against fakes of the CUDA runtime and of the kernels' launchers: no GPU."""
import os
import shutil
import subprocess

import pytest

from bunker_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))

# K, rows, columns: us in launches of 8 columns, us on the dense tile kernel with the launch that makes its image (one B200, lane order, a caller's Q8_1 blocks)
MEASURED = [
    (6144, 9216, 9, 30.5, 26.0), (2048, 24576, 9, 25.0, 26.8), (2048, 49152, 9, 39.4, 36.3), (17408, 1024, 9, 35.8, 19.0),
    (4096, 2048, 10, 13.4, 14.7), (2048, 9216, 10, 15.7, 16.4), (2048, 12288, 10, 20.3, 19.4), (1024, 49152, 10, 34.5, 26.0), (5120, 512, 10, 15.9, 13.0),
    (8192, 512, 16, 28.7, 14.7), (6144, 1024, 16, 18.9, 13.7), (4096, 1024, 16, 14.7, 12.6), (4096, 3072, 16, 17.2, 15.6), (1024, 24576, 16, 21.1, 22.4),
    (1024, 49152, 16, 35.2, 28.5), (2048, 12288, 16, 21.5, 20.1),
    (1024, 9472, 24, 17.1, 18.6), (1024, 12288, 24, 21.2, 21.9), (2048, 12288, 24, 30.8, 26.0), (2304, 98304, 24, 172.3, 97.9),
    (256, 12288, 32, 20.5, 18.8), (512, 12288, 33, 27.5, 25.3), (512, 24576, 33, 37.5, 41.1),
]


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    if not (os.path.exists(B._nvcc()) and shutil.which("g++")):
        pytest.skip("needs nvcc and g++")
    d = tmp_path_factory.mktemp("fakes")
    flags = [f for f in B.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    obj, exe = str(d / "gemv.o"), str(d / "gemv_fakes")
    subprocess.check_call([B._nvcc(), *flags, "-c", os.path.join(B.CSRC, "bk_gemv.cu"), "-o", obj])
    cuda = os.path.join(os.path.dirname(os.path.dirname(B._nvcc())), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", cuda, os.path.join(HERE, "gemv_fakes.cpp"), obj, "-o", exe])

    def run(shapes):
        text = "".join(f"{K} {rows} {cols}\n" for K, rows, cols in shapes)
        return subprocess.run([exe], input=text, capture_output=True, text=True, timeout=60, check=True).stdout.split()
    return run


def test_blocks_of_many_columns_take_the_path_that_was_the_faster(routes):
    got = routes([m[:3] for m in MEASURED])
    wrong = [(m, r) for m, r in zip(MEASURED, got) if (r == "dense") != (m[4] < m[3])]
    assert len(got) == len(MEASURED) and not wrong, wrong


def test_eight_columns_and_fewer_never_take_the_dense_kernel(routes):
    assert routes([(K, rows, cols) for K in (256, 6144) for rows in (512, 98304) for cols in (2, 8)]) == ["1"] * 8
