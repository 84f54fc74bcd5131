"""Waiting for a launch's words in page-locked memory, compiled for the CPU: words that a
finished stream has not written are an error, not a value."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_words_never_written_are_an_error(tmp_path):
    exe = str(tmp_path / "result_wait")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"), "-x", "c++",
                    os.path.join(HERE, "host", "result_wait.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
