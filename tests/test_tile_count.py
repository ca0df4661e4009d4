"""The count of a short flush's tile runs against the runs themselves, on the
CPU (tests/c/tile_count.c)."""

import subprocess

from conftest import ROOT


def test_count_equals_runs(tmp_path):
    exe = tmp_path / "tile_count"
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off",
                    f"-I{ROOT}/include", f"-I{ROOT}/phase2_b200/csrc",
                    str(ROOT / "tests/c/tile_count.c"), "-o", str(exe),
                    "-lm"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
