"""What the kernels rely on, checked in the sources: every kernel's first statement waits for the kernel before it; the kernels on
row tiles end well when a wait has run out."""
import ctypes
import glob
import os
import random
import re
import subprocess

import pytest

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


TILE_KERNELS = ["conv_tile.cu", "conv_six.cu"]


def _source(name):
    return re.sub(r"//.*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name,wait,said", [
    (name, r"land_copies\(C, P\.n_stages, kProdGroups\)", [r"\n    if \(brings_weights\) C\.ordered\.slabs\[group\] = filled;",
                                                           r"\n      C\.ordered\.slots = slot;"]) for name in TILE_KERNELS] +
    [("conv_dweight.cu", r"land_slots\(C\.s_full, C\.slots\)", [r"\n      C\.slots = n;"])])
def test_bulk_copies_land_on_every_way_out(name, wait, said):
    """Whatever made a role leave, and when: behind the block's last barrier the abort flag alone decides whether the bulk copies are
    waited for, and every role that orders them has said which, unconditionally."""
    text = _source(name)
    end = text[text.rindex("__syncthreads();", 0, text.index("tmem_dealloc(tmem")):text.index("tmem_dealloc(tmem")]
    assert re.search(r"if \(\*abort\) \{[^}]*%s;\s*\}" % wait, end)
    assert all(re.search(s, text) for s in said)
    assert text.count("bulk_copy_g2s(") == len(said)


def _role(text, name):
    return re.search(r"// =+ %s =+\n(.*?)(?=// =====|\n  __syncthreads)" % name, text, re.S).group(1)


def _decided_by_lanes(text):
    """Waits and looks at the abort flag in `text` whose outcome may differ between the lanes of a warp."""
    looks = re.sub(r"__(any|all)_sync\(0xffffffffu, [^;]*?\*abort != 0\)", "", re.sub(r"\*abort = 1", "", re.sub(r"//.*", "", text)))
    return re.findall(r"\bmbar_wait\(|\*abort", looks)


@pytest.mark.parametrize("name,role", [(name, role) for name, stores in zip(TILE_KERNELS, ("epilogue", "drain"))
                                       for role in ("producers", "MMA issue", stores)] +
                         [("conv_dweight.cu", role) for role in ("rows", "MMA issue")])
def test_warps_leave_as_a_whole(name, role):
    """Behind a wait that can run out, or the abort flag, all lanes of a warp go the same way: the collectives that follow
    (__syncwarp, shuffles, tcgen05.ld) would wait without limit for a lane that has left.  And all of them have seen the phase:
    one lane's wait and a shuffle order nothing for the others."""
    assert not _decided_by_lanes(_role(open(os.path.join(CSRC, name)).read(), role))


def test_last_slab(tmp_path):
    """The slab that a stage may still be waiting for, against a ring played step by step: two groups of warps, or one, order
    weights when a stage is free, steps are consumed in their turn, and everybody stops at some point."""
    text = _source("conv_tile.cuh")
    at = text.index("__host__ __device__ inline int last_slab")
    body = text[at:text.index("\n}\n", at) + 3].replace("__host__ __device__ inline", 'extern "C"')
    src, lib = tmp_path / "last_slab.cpp", tmp_path / "last_slab.so"
    src.write_text(body)
    subprocess.check_call([os.environ.get("CXX", "g++"), "-shared", "-fPIC", "-o", str(lib), str(src)])
    last_slab = ctypes.CDLL(str(lib)).last_slab
    rng = random.Random(5)
    for groups in (1, 2):
        for stages in range(2, 13):
            for _ in range(60):
                ordered, consumed, total = [0] * groups, 0, rng.randrange(0, 40)
                for _ in range(rng.randrange(0, 120)):
                    g = rng.randrange(groups + 1)
                    if g == groups:  # the next step has been consumed, if it is there
                        consumed += consumed // groups < ordered[consumed % groups]
                    elif (step := g + ordered[g] * groups) < total and step - stages < consumed:
                        ordered[g] += 1
                steps = {g + i * groups for g in range(groups) for i in range(ordered[g])}
                for st in range(stages):
                    mine = [n for n in steps if n % stages == st]
                    assert last_slab((ctypes.c_int * 2)(*ordered), groups, stages, st) == max(mine, default=-1)
                    assert all(n < consumed for n in mine if n != max(mine))  # the others need no waiting for
