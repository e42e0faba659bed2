"""What a launch through SCN_LAUNCH relies on, checked in the sources: every kernel's first statement waits for the kernel
before it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparseconvnet_b200", "csrc")


def _close(text, at):
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def test_every_kernel_waits_first():
    defined, waiting = set(), set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//.*", "", open(path).read())
        if "SCN_LAUNCH" not in text:  # a file that launches its kernels itself
            continue
        for m in re.finditer("__global__", text):
            name = re.compile(r"\b(k_\w+)\s*\(").search(text, m.end())
            body = text[_close(text, name.end() - 1):].lstrip()
            if body.startswith("{"):
                defined.add(name.group(1))
                if body[1:].lstrip().startswith("SCN_GRID_WAIT();"):
                    waiting.add(name.group(1))
    assert len(defined) > 60
    assert defined == waiting, sorted(defined - waiting)
