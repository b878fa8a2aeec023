"""What a basis builds on first use (csrc/cqf_once.hpp: the engine's pair list
and coefficient tables) is published only once it is written; compiled for the
host, with the failures made there."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_build_is_not_published(tmp_path):
    exe = str(tmp_path / "once")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-o", exe,
                           os.path.join(HERE, "cpp", "once.cpp")])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
