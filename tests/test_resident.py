"""Small registers held on chip: the cut of passes into sub-passes, on the
CPU, against the passes themselves (tests/c/sub_passes.c)."""

import subprocess

from conftest import ROOT


def test_sub_passes_equal_passes(tmp_path):
    exe = tmp_path / "sub_passes"
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off",
                    f"-I{ROOT}/include", f"-I{ROOT}/phase2_b200/csrc",
                    str(ROOT / "tests/c/sub_passes.c"), "-o", str(exe),
                    "-lm"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
