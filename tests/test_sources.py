"""Rules that the CUDA sources keep and that no run of theirs can show on one healthy device."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudapp_b200", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h"))):
        with open(path) as f:
            yield os.path.basename(path), f.read()


def test_no_cuda_status_is_kept_for_the_process():
    """a status in a static would make one failed call (another current device, a passing shortage) the answer of every later one"""
    kept = [(name, m.group(0)) for name, text in sources() for m in re.finditer(r"\bstatic\b[^;{}()]*=\s*cuda\w+\(", text)]
    assert not kept, kept


def test_row_entries_allocate_without_exceptions():
    """gemv and row-table entries: running out of host memory is a return code, as in the rest of the C interface, and no std::bad_alloc through it"""
    text = dict(sources())["fp8_gemv.cu"]
    assert not re.findall(r"std::(vector|string|make_unique|function)", text)
