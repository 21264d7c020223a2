"""Tables that a plan copies from host memory are on the device when the call that makes them
returns: an apply on another, non-blocking stream is not ordered behind the legacy stream's
copy.  Every such copy goes through the two functions that wait for it (reads the source: a
race on memory is not shown by running it)."""

import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyfourier_b200", "csrc")


def test_host_copies_wait():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = open(path).read()
        plain = re.findall(r"\bcuda(?:Memcpy|Memset)\(", src)
        if os.path.basename(path) != "pfb_pool.cu":
            assert not plain, f"{path}: {len(plain)} copies outside upload_table / clear_table"
            continue
        assert len(plain) == 2
        for name in ("upload_table", "clear_table"):
            body = re.search(rf"int {name}\([^)]*\) {{(.*?)\n}}", src, re.S).group(1)
            assert re.search(r"cuda(Memcpy|Memset)\(.*cudaStreamSynchronize\(0\)", body, re.S)
