"""The shared-memory opt-in of the dense kernels is made on every device that
launches them (smem_allowed.h, compiled for the host against a fake runtime)."""

import json
import os
import re
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gprx_b200", "csrc")


def test_attribute_is_set_once_per_device():
    exe = os.path.join(tempfile.mkdtemp(), "smem_allowed_driver")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I" + CSRC, "-I/usr/local/cuda/include", "-o", exe,
                           os.path.join(ROOT, "tests", "cpp", "smem_allowed_driver.cpp")])
    r = json.loads(subprocess.check_output([exe], text=True))
    # devices beyond the record are asked every time
    assert r == {"ok": 1, "failed": 1, "set": [0, 1, 3, 70, 70]}


def test_no_launcher_remembers_the_opt_in_for_the_process():
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.search(r"static bool \w+ = false;", f.read()), name
