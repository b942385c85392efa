"""Small rules of the kernels' headers, compiled for the host and run with the undefined-
behaviour sanitizer (no GPU)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def _run(tmp_path, body):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src = tmp_path / "t.cpp"
    src.write_text('#include "kernels.h"\n#include <cstdio>\nint main() {\n' + body + "\n}\n")
    exe = str(tmp_path / "t")
    # only inline functions are used: nothing of the CUDA runtime is linked
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I", CSRC, "-I",
                    CUDA_INCLUDE, str(src), "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()


def test_seed_parts(tmp_path):
    """No queues (the initial state seeds none), fewer warps than queues, more warps."""
    out = _run(tmp_path, "for (int w : {1, 16}) for (int q : {0, 1, 2, 5, 16, 40}) "
                         'std::printf("%d ", fgpu::seedParts(w, q));')
    assert [int(x) for x in out] == [0, 1, 1, 1, 1, 1] + [0, 16, 8, 3, 1, 1]
