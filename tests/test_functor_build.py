"""A caller's functor compiles with the command that include/hpmc_functor.cuh
and the integration notes give: no compiler flag beyond the architecture, the
language and the two include paths."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_functor_compiles_as_documented(hpmc, tmp_path):
    from hpmc_b200 import build as B

    with open(os.path.join(ROOT, "include", "hpmc_functor.cuh")) as f:
        text = f.read()
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17"]
    assert "nvcc " + " ".join(flags) in text
    r = subprocess.run([B.nvcc(), *flags, "-I" + os.path.join(ROOT, "include"), "-I" + B.CSRC, "-c",
                        os.path.join(B.APPS_DIR, "custom_functor.cu"), "-o", str(tmp_path / "functor.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:2000]
