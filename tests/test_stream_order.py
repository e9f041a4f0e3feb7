"""Every clear and every upload goes to the stream whose kernels read it.  The
library's streams are non-blocking: they do not wait for a memset, or for the
device's part of a copy, that was queued on the default stream."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "propack_gb300", "csrc")


def test_no_clears_or_uploads_on_the_default_stream():
    found = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        found += [(name, m.group(0)) for m in re.finditer(r"\bcudaMemset(2D|3D)?\([^;]*;", text)]
        found += [(name, m.group(0)) for m in re.finditer(r"\bcudaMemcpy(2D)?\([^;]*HostToDevice[^;]*;", text)]
    assert found == []
