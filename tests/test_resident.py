"""Passes cut into sub-passes and tile runs, on the CPU, against the passes
and the rotations themselves (tests/c/sub_passes.c, tests/c/tile_runs.c)."""

import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("name", ["sub_passes", "tile_runs"])
def test_cut_equals_passes(name, tmp_path):
    exe = tmp_path / name
    subprocess.run(["gcc", "-O2", "-std=gnu11", "-ffp-contract=off",
                    f"-I{ROOT}/include", f"-I{ROOT}/phase2_b200/csrc",
                    str(ROOT / f"tests/c/{name}.c"), "-o", str(exe),
                    "-lm"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
