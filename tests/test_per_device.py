"""What launchers remember per device: the host class on its own, and that no launcher remembers for the whole process."""
import glob
import os
import re
import subprocess

import popxl_addons_b200

CSRC = os.path.join(os.path.dirname(popxl_addons_b200.__file__), "csrc")


def test_devices_are_kept_apart(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text('#include "per_device.h"\n'
                   "int main() {\n"
                   "  static XlPerDevice a, b;\n"
                   "  a.set(0, 5); a.set(3, 7); a.set(64, 9); a.set(-1, 9);\n"
                   "  return !(a.get(0) == 5 && a.get(1) == 0 && a.get(3) == 7 && a.get(63) == 0 && a.get(64) == 0 && a.get(-1) == 0 && b.get(0) == 0);\n"
                   "}\n")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True)


def test_no_launcher_sets_an_attribute_once_per_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            text = f.read()
        assert not re.search(r"static (bool|int) \w+ = ", text), path
        assert "cudaFuncSetAttribute" not in text, path
