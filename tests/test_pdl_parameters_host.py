"""Source rule for programmatically launched kernels (csrc/fused.cuh,
pdl_launch): a kernel that waits for its predecessor with griddepcontrol.wait
holds no __restrict__ pointer to anything that another kernel writes.

The qualifier tells the compiler that nothing else touches the memory, the
wait's memory clobber included, so it may move such a load above the wait.  Only
data that no kernel of a solve writes may carry it: level views, operator and
coarse inverse, the dense tail, volumes and the two-block system."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "twophaseamr.jl_b200" / "csrc"
STATIC = {"levels", "lv", "G", "M", "vol"}
WAITS = re.compile(r"\b(pdl_entry|pdl_wait|tile_down|tile_up)\b\s*[(<]")


def kernels():
    """(file, name, text from __global__ to the end of the body) of every kernel."""
    for path in sorted(CSRC.glob("*.cu*")):
        src = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", src):
            body = src.index("{", m.start())
            depth, end = 0, body
            while True:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
                if depth == 0:
                    break
            head = src[m.start():body]
            if ";" in head:  # a declaration
                continue
            head = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", head)
            name = re.search(r"(\w+)\s*\(", head).group(1)
            yield path.name, name, src[m.start():end]


def test_waiting_kernels_hold_no_restrict_pointer_to_what_kernels_write():
    bad, waiting = [], 0
    for file, name, text in kernels():
        if not WAITS.search(text):
            continue
        waiting += 1
        for p in re.finditer(r"__restrict__\s+(\w+)", text):
            if p.group(1) not in STATIC:
                bad.append((file, name, p.group(1)))
    assert waiting > 40  # the search finds them
    assert not bad, bad
