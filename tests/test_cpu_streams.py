"""Every copy and clear of the library names a stream. A copy from pageable memory on the default stream may
return before the data has arrived, and the contexts' streams, which do not wait for the default one, would
then run kernels on what was there before."""

import os
import re

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "kassiopeia_b200", "csrc")


def test_no_copy_on_the_default_stream():
    found = []
    for name in sorted(os.listdir(SRC)):
        with open(os.path.join(SRC, name)) as f:
            for k, line in enumerate(f, 1):
                if re.search(r"\bcuda(Memcpy|Memcpy2D|MemcpyToSymbol|MemcpyFromSymbol|Memset)\s*\(", line.split("//")[0]):
                    found.append(f"{name}:{k}: {line.strip()}")
    assert not found, found
