"""The block pool's book-keeping over several contexts of a device (built and run on the CPU,
with the runtime's calls replaced)."""
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


@pytest.mark.skipif(not shutil.which("nvcc"), reason="needs nvcc")
def test_contexts_keep_their_blocks(tmp_path):
    exe = tmp_path / "pool_contexts"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "shared",
                    f"-I{PKG_DIR / 'csrc'}", f"-I{ROOT / 'include'}", str(PKG_DIR / "csrc" / "pool.cu"),
                    str(ROOT / "tests" / "cpp" / "pool_contexts.cu"), str(ROOT / "tests" / "cpp" / "fake_runtime.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
