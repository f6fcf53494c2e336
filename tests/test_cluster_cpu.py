"""Thread-block clusters: a CTA may touch another's shared memory only once that CTA is known to run."""
import glob
import os
import re

from conftest import ROOT


def kernels(text):
    """(name, body) of every __global__ function of a source file."""
    for m in re.finditer(r"__global__", text):
        at = text.index("{", text.index(") {", m.end()))
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield re.findall(r"(\w+)\s*\(", text[m.end():at])[-1], text[at:end]


def test_remote_shared_memory_is_touched_after_every_cta_has_started():
    """A cluster barrier (arrive and wait) stands before the first remote store of every kernel that has one."""
    seen = []
    for path in sorted(glob.glob(os.path.join(ROOT, "transformer-surgeon_b200", "csrc", "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for name, body in kernels(text):
            remote = re.search(r"(st|atom|red)\.\w*\.?shared::cluster\.[a-z]\d+ |st\.shared::cluster", body)
            if not remote:
                continue
            seen.append(name)
            before = body[:remote.start()]
            assert "barrier.cluster.arrive" in before and "barrier.cluster.wait" in before, f"{os.path.basename(path)}: {name}"
    assert {"kv_fp8_scales_kernel", "argmax_rows_kernel", "linear_gv_kernel"} <= set(seen)
