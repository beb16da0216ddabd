"""What a launch needs to know of a device (csrc/per_device.h) is found out once on each, not once per process."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_each_device_gets_its_own_value(tmp_path):
    exe = str(tmp_path / "per_device_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-pthread",
                           "-I", os.path.join(os.path.dirname(HERE), "mcw_cppamp_torch_b200", "csrc"),
                           os.path.join(HERE, "per_device_test.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_large_products_on_a_second_device():
    """The two-SM engine wants more shared memory than a kernel has by default, allowed per device."""
    import mcw_cppamp_torch_b200 as gt
    if gt.get_device_count() < 2:
        pytest.skip("needs two GPUs")
    a = np.random.default_rng(1).standard_normal((512, 512)).astype(np.float32)
    got = []
    try:
        for device in (1, 2):
            gt.set_device(device)
            got.append(gt.GPUTensor(512, 512).addmm(0.0, 1.0, gt.gpu(a), gt.gpu(a)).float())
    finally:
        gt.set_device(1)
    assert np.array_equal(got[0], got[1])
