"""The rule that picks the list step's form, compiled for the host (tests/cpp/list_form_test.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_list_form_rule(tmp_path):
    exe = str(tmp_path / "list_form_test")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I" + os.path.join(ROOT, "pe_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "list_form_test.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "ok"
