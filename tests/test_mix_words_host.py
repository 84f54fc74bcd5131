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


def test_every_mix_buffer_has_the_pad():
    import re
    csrc = os.path.join(os.path.dirname(HERE), "nightstream_b200", "csrc")
    core, fold = (open(os.path.join(csrc, f)).read() for f in ("core.cu", "fold.cu"))
    assert len(re.findall(r"rlc_mix_device\(ctx, rho_coeffs, dZs\.p", core)) == 1
    assert re.search(r"dZs\.alloc\([^;]*, MIX_PAD\)", core)
    # the witnesses of the fold's two lanes
    assert set(re.findall(r"rlc_dec_lane\(sh, [^,]+, [^,]+, [^,]+, sh->(\w+)\.p", fold)) == {"Zall", "valwit"}
    for buf in ("Zall", "valwit"):
        allocs = re.findall(r"%s\.(?:alloc|ensure)\(([^;]*)\);" % buf, fold)
        assert len(allocs) == 1 and allocs[0].rstrip(")").endswith(", MIX_PAD")
