"""The library's streams do not wait for the default stream (they are created non-blocking), and
cudaMemcpy may return before a transfer from pageable memory, or a device-to-device copy, has
ended: no copy of the library goes to the default stream."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvm_gb300", "csrc")


def test_copies_name_their_stream():
    files = glob.glob(os.path.join(CSRC, "*.cu*"))
    assert files
    for f in files:
        src = re.sub(r"//[^\n]*", "", open(f).read())
        assert not re.search(r"\bcuda(Memcpy|Memset)(2D|3D|ToSymbol|FromSymbol)?\s*\(", src), os.path.basename(f)
