"""Dynamic shared memory that a kernel reads in wider pieces than its declared
element states that alignment: nothing else makes the compiler place it so."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "propack_gb300", "csrc")


# widest access through the array: float4 / double2 of the complex updates, 32-bit digit and BF16 pairs
@pytest.mark.parametrize("name,array,width", [("pgb_lanczos.cuh", "dyn", 16), ("pgb_gemm_tc.cu", "Bs", 4),
                                              ("pgb_mlp.cu", "wsm", 4), ("pgb_mlp.cu", "dws", 16)])
def test_declared_alignment(name, array, width):
    with open(os.path.join(CSRC, name)) as f:
        decl = re.findall(r"extern __shared__ (.*?)\b%s\[\];" % array, f.read())
    assert decl
    for d in decl:
        given = re.search(r"__align__\((\d+)\)", d)
        size = {"double": 8, "unsigned short": 2, "unsigned char": 1}[re.sub(r"__align__\(\d+\)", "", d).strip()]
        assert max(size, int(given.group(1)) if given else 0) >= width
