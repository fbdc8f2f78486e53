"""CPU check of the serving loop's admission under scratch needs that do not
rise with a launch's size (tests/serve_need_check.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_admission_under_any_need(tmp_path):
    exe = str(tmp_path / "serve_need_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined",
                    "-o", exe, os.path.join(HERE, "serve_need_check.cpp")],
                   check=True, capture_output=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout == "ok\n"
