"""Passes in which several lanes share a row and update its state in place: a lane's reads of
the row's stage state stand before a barrier of the whole warp, the other lanes' writes of it
behind.  Nothing else orders them, and a run whose lanes happen to keep in step shows nothing,
so the order is checked in the kernels' source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "mfree_iwf_gb300", "csrc")


def kernel_body(file, name):
    """The kernel's first definition in the file, without comments, from its opening brace on."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    start = text.index("{", re.search(r"__global__[^;{]*\b%s\(" % name, text).start())
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start + 1:i]
    raise AssertionError(name)


def whole_warp_barriers(body):
    """Positions of the warp barriers that stand in no branch or loop and behind no return."""
    depth = 0
    for m in re.finditer(r"[{}]|\breturn\b|__syncwarp\(\);", body):
        if m[0] in "{}":
            depth += 1 if m[0] == "{" else -1
        elif m[0] == "return":
            return
        elif depth == 0:
            yield m.start()


@pytest.mark.parametrize("file,kernel,read,write", [("mf_weak.cu", "k_p_pass64", r"\bs\.v[xy]\b", r"p_rk64\("),
                                                    ("mf_ul.cu", "k_pair64", r"\bsv\.S\w\w\[i\]", r"\bS\[i\] =")])
def test_barrier_between_reads_and_writes_of_a_row(file, kernel, read, write):
    body = kernel_body(file, kernel)
    last_read = [m.start() for m in re.finditer(read, body)][-1]
    first_write = re.search(write, body).start()
    assert last_read < first_write
    assert any(last_read < p < first_write for p in whole_warp_barriers(body))
