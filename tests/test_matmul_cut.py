"""How the batched product deals its work, on the host (no GPU): the header the kernel is cut by, compiled with g++ and walked."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_every_tile_is_written_once_and_reserved_areas_hold_the_calls(tmp_path):
    exe = tmp_path / "matmul_cut_test"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'include'}", f"-I{ROOT / 'recipe_dev_b200' / 'csrc'}", str(ROOT / "tests/cpp/matmul_cut_test.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
