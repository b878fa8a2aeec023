"""The item lists of the Hermite-matrix engine (csrc/cqf_hg_items.hpp) stay in
the region given to them: the host and device arithmetic, compiled for the
host, on random launches (tests/cpp/hg_items.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_items_of_both_lists_fit_the_region(tmp_path):
    exe = str(tmp_path / "hg_items")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-o", exe,
                           os.path.join(HERE, "cpp", "hg_items.cpp")])
    r = subprocess.run([exe, "3000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
