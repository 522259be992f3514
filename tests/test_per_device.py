"""What launches keep per GPU (rds_per_device.h), compiled for the host with a stand-in for the
CUDA runtime; and that no launcher keeps a number of the device for the whole process."""

import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pdekit_b200", "csrc")


def test_per_device(tmp_path):
    exe = tmp_path / "per_device_test"
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, "-I" + include,
                    os.path.join(ROOT, "tests", "cpp", "per_device_test.cpp"), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_number_of_the_device_is_kept_for_the_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            found = re.findall(r"^\s+static (?:int|bool|unsigned|long long) \w+[^(;]*;", f.read(),
                               re.M)
        assert not found, (path, found)
