"""Host-side checks in C++ of code that the Python interface cannot reach alone:
each program of tests/native is compiled with the engine's own sources and run
(no GPU)."""
import subprocess
from pathlib import Path


ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "soft-body-simulation-cuda_gb300" / "csrc"


def _run(tmp_path, name, *sources, link=()):
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-I", str(ROOT / "include"), "-I",
                    "/usr/local/cuda/include", str(ROOT / "tests" / "native" / f"{name}.cpp"),
                    *[str(CSRC / s) for s in sources], "-o", str(exe), "-pthread", *link], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)


def test_the_panel_update_stays_in_its_block(tmp_path):
    """Block sizes that leave one to seven columns for the last step of eight."""
    r = _run(tmp_path, "panel_indices")
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


def test_a_collision_list_is_never_longer_than_its_memory(tmp_path):
    """An allocation that fails while the list grows, then once more."""
    r = _run(tmp_path, "list_growth")
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_the_layout_survives_every_failed_allocation(tmp_path):
    """With threads already running, too."""
    r = _run(tmp_path, "layout_no_memory", "layout.cpp", link=("-L/usr/local/cuda/lib64", "-lcudart"))
    assert r.returncode == 0 and r.stdout == "ok 1\n", r.stdout + r.stderr
