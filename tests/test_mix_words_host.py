"""The aligned word loads of the ragged RLC mix stay inside the digits and make the right
columns: the kernel's own address arithmetic, compiled for the CPU under the address sanitizer."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_mix_words_stay_inside_the_digits(tmp_path):
    exe = str(tmp_path / "mix_words")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", os.path.join(HERE, "host", "mix_words.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
