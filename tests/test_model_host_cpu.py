"""Host logic of the model (bk_model.cu) against fakes of the CUDA runtime and of the kernels' launchers: no GPU."""
import os
import shutil
import subprocess

import pytest

from bunker_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))
OK, ARG, UNSUPPORTED, OUT_OF_MEMORY = 0, 10001, 10004, 2   # BK_* codes, cudaErrorMemoryAllocation


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not (os.path.exists(B._nvcc()) and shutil.which("g++")):
        pytest.skip("needs nvcc and g++")
    d = tmp_path_factory.mktemp("fakes")
    flags = [f for f in B.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    obj, exe = str(d / "model.o"), str(d / "model_fakes")
    subprocess.check_call([B._nvcc(), *flags, "-c", os.path.join(B.CSRC, "bk_model.cu"), "-o", obj])
    cuda = os.path.join(os.path.dirname(os.path.dirname(B._nvcc())), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", cuda, os.path.join(HERE, "model_fakes.cpp"), obj, "-o", exe])

    def run(*args):
        out = subprocess.check_output([exe, *map(str, args)], text=True, timeout=60)
        return {k: int(v) if v.lstrip("-").isdigit() else v for k, v in (line.split(" ", 1) for line in out.splitlines())}
    return run


@pytest.mark.parametrize("mode", [0, 2])
def test_one_launch_step_where_the_plan_can_be_made(program, mode):
    r = program(mode, OK)
    assert r["finalize"] == OK and r["plans"] == 1 and r["plans_left"] == 0
    assert r["step"] == r["eager"] == OK and r["plan_launches"] == 2 and r["gemvs"] == 0


def test_automatic_mode_goes_on_with_the_launch_chain(program):
    """What the device cannot do (tensor maps of the state that are not encoded, a kernel that does not fit an SM) is no error of the
    library's own choice: the plan is given back and the step is one launch per op."""
    r = program(0, UNSUPPORTED)
    assert r["finalize"] == OK and r["plans"] == 0
    assert r["step"] == r["eager"] == OK and r["plan_launches"] == 0 and r["gemvs"] > 0 and r["graphs"] == 4 and r["graph_launches"] == 1


@pytest.mark.parametrize("mode,rc", [(2, UNSUPPORTED), (2, OUT_OF_MEMORY), (0, OUT_OF_MEMORY)])
def test_other_failures_of_the_plan_are_reported(program, mode, rc):
    r = program(mode, rc)
    assert r["finalize"] == rc and r["plans"] == 0


def test_long_contexts_leave_the_one_launch_step(program):
    """One pair of query heads on one KV head and splits of 64 rows: a round of attention items is 148 * 64 = 9,472 rows and costs 6.68 us, the
    chain's kernel 12.46 us and 0.4 us per MB (3.88 a round), the other launches of two small layers 11.97 us: eight rounds pay, the ninth does not."""
    r = program(0, OK, 80000, 76000)
    assert r["finalize"] == OK and r["graphs"] == 6 and r["plan_graphs"] == 2
    assert r["first_chain"] == 8 * 9472 and r["back"] == 0


@pytest.mark.parametrize("mode,max_len", [(0, 9000), (2, 80000)])
def test_one_launch_step_at_every_position(program, mode, max_len):
    """A cache that ends within the rule, and a caller who asked for the one-launch step: no graph of the chain is captured."""
    r = program(mode, OK, max_len, min(max_len, 79000))
    assert r["finalize"] == OK and r["graphs"] == r["plan_graphs"] == 2 and r["first_chain"] == -1
