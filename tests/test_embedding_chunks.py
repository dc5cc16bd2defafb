"""Index arithmetic of the embedding backward at and below its limit of 2^31 - 257 tokens, on the
host (a batch of that size is not run)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
@pytest.mark.parametrize("n", [1, 64, 65, 65536, 65537, 2 ** 30 + 1, 2 ** 31 - 2 ** 21,
                               2 ** 31 - 2 ** 21 + 1, 2 ** 31 - 257])
def test_chunks_cover_the_tokens(n, tmp_path):
    exe = str(tmp_path / "embedding_chunks_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fwrapv", "-I",
                    os.path.join(ROOT, "dion_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "embedding_chunks_check.cpp"), "-o", exe],
                   check=True)
    run = subprocess.run([exe, str(n)], capture_output=True, text=True)
    assert run.stdout.strip() == "ok"
