"""The autotuner's search over launch shapes (va_tune.h) on made-up times, without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pair_of_shapes(tmp_path):
    exe = str(tmp_path / "tune_check")
    subprocess.run(["g++", "-O1", "-std=c++17", os.path.join(ROOT, "tests", "cpp", "tune_check.cpp"), "-o", exe], check=True)
    out = {ln.split()[0]: ln.split()[1:] for ln in subprocess.run([exe], check=True, capture_output=True,
                                                                    text=True).stdout.splitlines()}
    fb, fbps, bb, bbps = map(int, out["coupled"][:4])  # by the sum of the two sweeps, not each by itself
    assert fb * fbps == 512 and (bb * bbps == 512 or bb == 0)
    assert out["default"][:4] == ["0"] * 4  # no more than 1% to gain: the default shape stays
    fb, fbps, bb, bbps = map(int, out["apart"][:4])
    assert fb * fbps == 256 and bb * bbps == 384
    fb, _, bb, bbps = map(int, out["half"][:4])
    assert fb == 0 and bb * bbps == 128
    assert all(v[4] == "1" and v[5] == "few" for k, v in out.items() if k != "fails")
    assert out["fails"][4] == "0"
