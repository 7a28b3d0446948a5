"""Host-side rules of the batched path, compiled with g++ (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def run_check(tmp_path, name):
    exe = tmp_path / name
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "sovereign_b200", "csrc"), os.path.join(ROOT, "tests", name + ".cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "failures 0" in r.stdout, r.stdout + r.stderr


def test_streams_and_events_stay_on_their_device(tmp_path):
    run_check(tmp_path, "handle_pool_check")


def test_width_rule(tmp_path):
    run_check(tmp_path, "batch_width_check")
