"""The cases of the deep-tile tests get deep tiles, their two-volume forms shallow ones,
and the rings of tests/test_large_rings_gpu.py lie on both sides of the table limit."""
import shutil
import subprocess
from pathlib import Path

import pytest

from tests.test_deep_tiles_gpu import CASES
from tests.test_large_rings_gpu import RINGS

ROOT = Path(__file__).resolve().parent.parent
UTAB_MAX = 1984  # kUTabMax


@pytest.fixture(scope="module")
def plans(built_lib, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("CUDA toolkit not present")
    out = tmp_path_factory.mktemp("depth") / "depth_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(Path(nvcc).resolve().parent.parent / "include"), "-I",
                    str(ROOT / "include"), "-I", str(ROOT / "rfba_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "depth_check.cpp"), "-o", str(out), "-L", str(built_lib.parent),
                    "-lrfba_srrf", f"-Wl,-rpath,{built_lib.parent}"], check=True, capture_output=True, text=True)

    def run(rows):
        text = "".join(" ".join(map(str, (*mag, axes, *shape))) + "\n" for mag, axes, shape in rows)
        r = subprocess.run([str(out)], input=text, capture_output=True, text=True, timeout=120, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


def test_series_of_the_deep_cases_get_deep_tiles(plans):
    rows = [(mag, axes, shape) for mag, shape, axes, _, _ in CASES] + [tuple(r) for r in RINGS]
    assert [r[0] for r in plans(rows)] == [8] * len(rows)
    assert {r[0] for r in plans([(m, a, (2,) + s[1:]) for m, a, s in rows])} == {4}


def test_rings_lie_on_both_sides_of_the_table_limit(plans):
    sizes = plans(RINGS)
    assert {s[1] <= UTAB_MAX for s in sizes} == {True, False}
    assert {s[2] <= UTAB_MAX for s in sizes} == {True, False}
