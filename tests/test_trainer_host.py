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


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("rays", [1, 31, 33, 63, 2048, 4001, 16384, 65536, 131072, 200000, 1 << 18, 1 << 20])
def test_device_memory_of_a_trainer(trainer_host, exact, rays):
    """At most 64 KiB per ray (64 B per ray and march step), the staging of 2^21
    records in FP32 (472 values), the rays' own 88 bytes and 160 KB of weight
    images: what a trainer took before its samples' encodings were kept."""
    assert int(trainer_host("memory", exact, rays)[0]) <= (65536 + 88) * rays + (472 * 4 << 21) + 160000
