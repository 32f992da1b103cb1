"""Layouts that the device code relies on, checked by compiling against its headers."""
import os
import shutil
import subprocess

import pytest

from pgxc import build as B


@pytest.mark.skipif(not (os.path.exists(B.nvcc()) or shutil.which(B.nvcc())), reason="no nvcc")
def test_basis_item_is_aligned_for_its_16_byte_loads(tmp_path):
    """Five 16-byte loads per record: every record, and a copy of one in local
    memory, has to begin on a 16-byte boundary."""
    src = tmp_path / "layout.cu"
    src.write_text('#include <cstdint>\n#include "basis.cuh"\n'
                   "static_assert(sizeof(pgxc::BasisItem) == 80, \"size\");\n"
                   "static_assert(alignof(pgxc::BasisItem) % 16 == 0, \"alignment\");\n")
    r = subprocess.run([B.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", B.CSRC, "-c",
                        str(src), "-o", str(tmp_path / "layout.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
