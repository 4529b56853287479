"""CPU: kernels that need more dynamic shared memory than 48 KB are allowed it
on every device that launches them (pwm_gb300/csrc/device_once.hpp): the
setting is kept per device, so one made for the first is none for the second."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pwm_gb300", "csrc")


def test_once_per_device(tmp_path):
    exe = str(tmp_path / "once")
    src = os.path.join(ROOT, "tests", "host_logic", "once.cpp")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_no_setting_is_made_once_a_process():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.search(r"static\s+(std::atomic<)?bool", f.read()), name
