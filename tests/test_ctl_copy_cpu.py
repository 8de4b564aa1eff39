"""The host's copy of a pass's control block keeps a fault that the emit reports while the
copy is made (built and run on the CPU)."""
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


@pytest.mark.skipif(not shutil.which("nvcc"), reason="needs nvcc")
def test_fault_survives_the_copy(tmp_path):
    exe = tmp_path / "ctl_copy"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{PKG_DIR / 'csrc'}",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests" / "cpp" / "ctl_copy.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
