"""What cost models ask of a device is kept per device (`device_table.h`)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "kestrel-llm_b200", "csrc", "kernels")


def test_answers_are_kept_by_device(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    exe = str(tmp_path / "device_table_test")
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-pthread", "-I", KERNELS, os.path.join(ROOT, "tests", "c", "device_table_test.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


def test_resident_clusters_are_asked_of_the_current_device():
    with open(os.path.join(KERNELS, "attention_decode.cu")) as f:
        body = re.search(r"int kestrel_attention_decode_clusters\(.*?\n}", f.read(), re.S).group(0)
    assert "DeviceTable<" in body and "cudaGetDevice" in body and not re.search(r"static int ", body)
