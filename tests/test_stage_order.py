"""The consumers' wait for a stage of the apply engine, on the CPU: no order in
which staged copies can complete lets a group take an item that has not landed, and
none brings the ring to a halt (tests/stage_order_driver.cpp runs the wait of
csrc/cuda/stage_order.h through every interleaving of the first items)."""
import os
import subprocess

from rank_structured_cholesky_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(tmp_path, header_dir):
    exe = str(tmp_path / "driver")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", str(header_dir),
                    os.path.join(HERE, "stage_order_driver.cpp"), "-o", exe], check=True)
    return subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=120)


def test_no_item_is_taken_before_it_landed(tmp_path):
    p = _run(tmp_path, os.path.join(_build.CSRC, "cuda"))
    assert p.returncode == 0, p.stdout


def test_the_model_sees_a_wait_by_parity_alone(tmp_path):
    """The model can tell: with the wait for the item before left out, it finds the order."""
    src = open(os.path.join(_build.CSRC, "cuda", "stage_order.h")).read()
    planted = src.replace("if (use > 0 && !empty(s, (use - 1) & 1)) return false;", "")
    assert planted != src
    (tmp_path / "stage_order.h").write_text(planted.replace("Empty empty)", "Empty)"))
    p = _run(tmp_path, tmp_path)
    assert p.returncode == 1 and "before it has landed" in p.stdout
