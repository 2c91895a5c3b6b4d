"""What a failed call leaves behind (csrc/context.cuh, Ctx::recover): a host
program built around the C entries' error handling, run without a device."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_failed_call_leaves_no_hash_error(tmp_path):
    exe = tmp_path / "recover"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-o", str(exe), str(ROOT / "tests" / "recover.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
