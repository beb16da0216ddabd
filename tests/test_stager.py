"""The staged upload (csrc/thc_stager.h) on the host, over a stand-in for the CUDA runtime whose copies run as late as they may."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SHIM = os.path.join(HERE, "stager_shim")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("stager") / "stager_test")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", SHIM,
                           "-I", os.path.join(os.path.dirname(HERE), "mcw_cppamp_torch_b200", "csrc"),
                           os.path.join(SHIM, "stager_test.cpp"), "-o", exe])
    return exe


def run(driver, what):
    r = subprocess.run([driver, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (what, r.returncode, r.stdout, r.stderr)


def test_an_upload_to_another_device_waits_for_the_pieces_in_flight(driver):
    run(driver, "devices")


def test_a_device_whose_events_cannot_be_made_leaves_the_others_usable(driver):
    run(driver, "event")


def test_without_a_second_thread_uploads_take_the_drivers_way(driver):
    run(driver, "thread")
