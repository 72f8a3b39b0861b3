"""Launch settings that belong to a device (a kernel's opt-in to more than 48
KiB of shared memory, its L1 carveout) are made on each device that renders,
not once per process: renders on two devices of a stand-in for the CUDA runtime
(fake_cudart.cpp: no kernel runs), which refuses a launch above its opt-in as
the runtime does."""
import glob
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_each_device_gets_its_launch_settings(nes_lib, tmp_path):
    import nes_build
    exe = str(tmp_path / "devices_host")
    subprocess.run([nes_build.NVCC, "-std=c++17", "-cudart", "none", "-I", nes_build.CSRC, "-I", nes_build.INCLUDE,
                    os.path.join(HERE, "devices_host.cu"), os.path.join(HERE, "fake_cudart.cpp"),
                    *glob.glob(os.path.join(nes_build.BUILD, "*.o")), "-lpthread", "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")[:2]
    assert [line.split() for line in out] == [["0", "0", "0", "14"]] * 2
