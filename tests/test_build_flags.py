"""The engine's optional build flags compile (CPU only; unoptimised, nothing is run)."""
import os
import subprocess

import pytest

from amcafe_gb300 import build as b


@pytest.mark.parametrize("flag", ["-DCAFE_DETAIL_CYCLES"])
def test_engine_compiles_with(tmp_path, flag):
    flags = [f for f in b.NVCC_FLAGS if f not in ("-O3", "-shared", "-lineinfo")]
    subprocess.run([b._nvcc()] + flags + ["-O0", "-Xcicc", "-O0", flag, "-ptx", "-o", str(tmp_path / "engine.ptx"),
                                          os.path.join(b.CSRC, "cafe_host.cu")], check=True)
