"""Tables that a plan copies from host memory are on the device when the call that makes them
returns: an apply on another, non-blocking stream is not ordered behind the legacy stream's
copy.  Every such copy goes through two functions, and every entry point that reaches them
waits before it returns (reads the source: a race on memory is not shown by running it)."""

import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyfourier_b200", "csrc")


def _read(name):
    return open(os.path.join(CSRC, name)).read()


def _body(src, name):
    return re.search(rf"int {name}\([^)]*\) {{\n(.*?)\n}}", src, re.S).group(1)


def test_host_copies_go_through_the_table_functions():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        plain = re.findall(r"\bcuda(?:Memcpy|Memset)\(", open(path).read())
        want = 2 if os.path.basename(path) == "pfb_pool.cu" else 0
        assert len(plain) == want, f"{path}: {len(plain)} copies"
    assert "cudaStreamSynchronize(0)" in _body(_read("pfb_pool.cu"), "wait_tables")


def test_entry_points_wait():
    makers = r"(upload_table|clear_table|rebuild_items|build_owner_items|fft_axes|fft_fused_ready)\("
    for file, name in (("pfb_plan.cu", "plan_create"), ("pfb_capi.cu", "pfb_plan_set_chunk"), ("pfb_capi.cu", "pfb_gram_create")):
        body = _body(_read(file), name)
        last = max(m.start() for m in re.finditer(makers, body))
        assert "wait_tables()" in body[last:], name
