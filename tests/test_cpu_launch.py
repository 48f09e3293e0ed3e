"""Launch set-up per device: the launch functions of the binning and the pair pass over a stand-in
for the CUDA runtime (tests/fakes/fake_cudart.cpp), which keeps the opt-in for more than 48 KB of
shared memory per device as the runtime does.  An engine on a second device of the process has its
kernels set up there, with that device's occupancy."""
import ctypes as C
import os
import subprocess

import pytest

import build as tfg_build

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "fakes", "_build", "libtfg_launch.so")


@pytest.fixture(scope="module")
def fake():
    cuda = os.path.dirname(os.path.dirname(tfg_build.NVCC))
    inc = ["-I" + os.path.join(tfg_build.HERE, "csrc"), "-I" + os.path.join(tfg_build.ROOT, "include")]
    objs = [os.path.join(tfg_build.BUILD, o) for o in ("tfg_kernels.cu.o", "tfg_pair_tile.cu.o")]
    driver, rt = (os.path.join(HERE, "fakes", s) for s in ("launch_driver.cu", "fake_cudart.cpp"))
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.check_call([tfg_build.NVCC, "-std=c++17", "-O1", *tfg_build.ARCH, "-Xcompiler", "-fPIC", *inc, "-c", driver,
                           "-o", OUT + ".o"])
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs",
                           "-I" + os.path.join(cuda, "include"), "-o", OUT, rt, OUT + ".o", *objs])
    return C.CDLL(OUT)


def test_kernels_are_set_up_on_every_device(fake):
    for device, per_sm in ((0, 3), (1, 2), (0, 3)):
        fake.fake_set_device(device)
        for n, cells, homes, dpd in ((500, 125, 8, 0), (50_000, 20_000, 16, 0), (5_000, 8_000, 8, 1), (2_000_000, 150_000, 32, 0)):
            before = fake.fake_launches()
            fake.drive_step(n, cells, homes, dpd, 0, 152)
            assert fake.fake_launches() > before
            assert fake.fake_refused() == 0, (device, n)
        assert fake.fake_last_grid() == 152 * per_sm


@pytest.mark.parametrize("dpd", [0, 1])
def test_warps_of_a_block(fake, dpd):
    """By the home particles of a work item, or as the caller fixes them."""
    for homes, warps, threads in ((8, 0, 128), (16, 0, 128), (32, 0, 256), (8, 8, 256), (32, 4, 128), (32, 8, 256)):
        fake.drive_step(100_000, 20_000, homes, dpd, warps, 152)
        assert fake.fake_last_block() == threads, (homes, warps)
