"""CPU checks of the host side of the steps on neighbour lists."""

from __future__ import annotations

import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("name", ("list_buffers", "list_policy"))
def test_list_host(tmp_path, name):
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++20", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I", str(ROOT / "titsolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "cpp" / f"{name}.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    assert res.stdout.strip() == "ok"
