"""The trainer's host code over a stand-in for the CUDA runtime
(fake_cudart.cpp: no kernel runs, device memory is host memory)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def trainer_host(nes_lib, tmp_path_factory):
    import nes_build
    exe = str(tmp_path_factory.mktemp("host") / "trainer_host")
    subprocess.run([nes_build.NVCC, "-std=c++17", "-cudart", "none", "-I", nes_build.CSRC, "-I", nes_build.INCLUDE,
                    os.path.join(HERE, "trainer_host.cu"), os.path.join(HERE, "fake_cudart.cpp"),
                    os.path.join(nes_build.BUILD, "train.cu.o"), "-o", exe], check=True)
    return lambda *args: subprocess.run([exe] + [str(a) for a in args], check=True, capture_output=True,
                                        text=True).stdout.split()


@pytest.mark.parametrize("exact,kernel,part", [(0, "eval_tc_kernel", 2), (0, "backward_tc_kernel", 1),
                                               (0, "dw_tc_kernel", 2), (1, "adjoint_kernel", 2)])
def test_a_failed_step_leaves_no_gradient_behind(trainer_host, nes_lib, exact, kernel, part):
    """A batch in several parts whose step fails in one of them: the next
    gradient is that of its own parts alone."""
    step, parts, table, weights = trainer_host("failure", exact, kernel, part)
    assert int(step) == nes_lib.NES_ETIMEDOUT
    assert int(parts) >= 2
    assert float(table) == float(weights) == int(parts)
