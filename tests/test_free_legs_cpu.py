"""The rule that frees a field march of its wall limit, no GPU: the functions
that the kernel calls (free_leg_room and wall_ahead, csrc/anacor_internal.h)
are compiled with the host set-up of the face rules and run over random legs,
volumes and label boxes (tests/host/free_legs_check.cpp)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "anacor_public_gb300", "csrc")


def check(tmp_path, source_dir):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    m = re.search(r"kFieldMargin = (\d+)u \+ (\d+)u;", open(os.path.join(CSRC, "trace_kernels.cu")).read())
    exe = os.path.join(tmp_path, "free_legs_check")
    cmd = [gxx, "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off", f"-DMARGIN={int(m[1]) + int(m[2])}ll",
           "-I", source_dir, "-I", CSRC, "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "host", "free_legs_check.cpp"), os.path.join(CSRC, "reflection_setup.cpp"),
           "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return subprocess.run([exe], capture_output=True, text=True, timeout=120)


def test_free_legs_stay_inside(tmp_path):
    r = check(tmp_path, CSRC)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.parametrize("was,wrong", [("(int)(qmax >> 32) + 2", "(int)(qmax >> 32)"), ("? axis : 3 + axis", "? 3 + axis : axis")])
def test_a_wrong_rule_is_found(tmp_path, was, wrong):
    text = open(os.path.join(CSRC, "anacor_internal.h")).read()
    assert was in text
    with open(os.path.join(tmp_path, "anacor_internal.h"), "w") as f:
        f.write(text.replace(was, wrong))
    r = check(tmp_path, str(tmp_path))
    assert r.returncode == 1 and r.stdout.startswith("a free leg leaves"), r.stdout + r.stderr
