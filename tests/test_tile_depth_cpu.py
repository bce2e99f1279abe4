"""The cases of the deep-tile tests get deep tiles, their two-volume forms shallow ones,
those of tests/test_small_launches_gpu.py the depth they name, and the rings of
tests/test_large_rings_gpu.py lie on both sides of the table limit."""
import shutil
import subprocess
from pathlib import Path

import pytest

from tests.test_deep_tiles_gpu import CASES
from tests.test_large_rings_gpu import RINGS
from tests.test_small_launches_gpu import ADJOINT, FLAT, SERIES

ROOT = Path(__file__).resolve().parent.parent
UTAB_MAX = 1984  # kUTabMax


def _build(tmp_path_factory, built_lib, name):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("CUDA toolkit not present")
    out = tmp_path_factory.mktemp(name) / name
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(Path(nvcc).resolve().parent.parent / "include"), "-I",
                    str(ROOT / "include"), "-I", str(ROOT / "rfba_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / (name + ".cpp")), "-o", str(out), "-L", str(built_lib.parent),
                    "-lrfba_srrf", f"-Wl,-rpath,{built_lib.parent}"], check=True, capture_output=True, text=True)
    return out


@pytest.fixture(scope="module")
def plans(built_lib, tmp_path_factory):
    out = _build(tmp_path_factory, built_lib, "depth_check")

    def run(rows):
        text = "".join(" ".join(map(str, (*mag, axes, *shape))) + "\n" for mag, axes, shape in rows)
        r = subprocess.run([str(out)], input=text, capture_output=True, text=True, timeout=120, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


def test_series_of_the_deep_cases_get_deep_tiles(plans):
    rows = [(mag, axes, shape) for mag, shape, axes, _, _ in CASES] + [tuple(r) for r in RINGS]
    assert [r[0] for r in plans(rows)] == [8] * len(rows)
    assert {r[0] for r in plans([(m, a, (2,) + s[1:]) for m, a, s in rows])} <= {2, 4}


def test_small_launches_get_the_depth_they_name(plans):
    assert [r[0] for r in plans([(mag, axes, shape) for mag, axes, shape in FLAT])] == [2] * len(FLAT)
    assert [r[1] for r in plans([(mag, axes, shape) for mag, axes, shape, _ in ADJOINT])] == [c[3] for c in ADJOINT]
    full = [r[1] for r in plans([(mag, 5, (n, *volume)) for mag, volume, n in SERIES])]
    assert full == [8 if max(mag[1:]) <= 4 else 4 for mag, _, _ in SERIES]
    assert [2 * r[1] for r in plans([(mag, 5, (n // 8, *volume)) for mag, volume, n in SERIES])] == full


def test_rings_lie_on_both_sides_of_the_table_limit(plans):
    sizes = plans(RINGS)
    assert {s[2] <= UTAB_MAX for s in sizes} == {True, False}
    assert {s[3] <= UTAB_MAX for s in sizes} == {True, False}


def test_shared_memory_holds_what_the_kernels_index(built_lib, tmp_path_factory):
    prog = _build(tmp_path_factory, built_lib, "layout_check")
    out = subprocess.run([str(prog)], capture_output=True, text=True, timeout=300, check=True).stdout.splitlines()
    assert out[-1].startswith("0 of ") and int(out[-1].split()[-1]) > 20000, out
