"""Programmatic dependent launch: a kernel that triggers before its own wait lets its successor start while its predecessor still
writes, so no kernel may read what another one writes before griddepcontrol.wait.  Checked on the sources: in every kernel with a
wait, the text in front of it names none of the kernel's pointers to data, constants and address-only uses (prefetches) aside."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "glm-flash-rs_b200", "csrc")
CONSTANT = {"wr", "suh", "svh", "suh0", "suh1", "map"}               # weights and scales: no kernel writes them
# combine_kernel stands behind kernels that trigger after their own wait (its comment names them): the routing table is complete
BEHIND_ORDERED = {("combine_kernel", "picks"), ("combine_kernel", "route_w")}


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            body = text[text.index("{", i):]
            end = body.find("\n}\n")
            yield os.path.basename(path), m.group(1), params, body[:end]


def names_read(params, front):
    front = re.sub(r'asm volatile\("prefetch[^\n]*', "", front)
    front = re.sub(r'asm volatile\("" ::"r"\(reinterpret_cast<const int \*>\(&a\)\[tid\]\)\);', "", front)   # (the parameter itself)
    for p in re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:,|$)", params):
        if p not in CONSTANT and re.search(r"(?<![\w.])%s\b" % p, front):
            yield p
    # kernels with an argument struct `a`: members that are data
    for p in re.findall(r"\ba\.(\w+)\s*(?:\[|\+)", front):
        if p in ("picks", "x", "ids", "count", "members", "route_w", "ctrl", "sync", "plan", "chunks", "src_pair"):
            yield "a." + p
    for p in re.findall(r"(?:__ldcg|__ldg)\(a\.(\w+)", front):
        yield "a." + p


def test_every_chained_kernel_is_seen():
    seen = {k for _, k, _, body in kernels() if "pdl_wait()" in body}
    assert {"stream_kernel", "window_kernel", "combine_kernel", "stage_in_kernel", "grouping_kernel", "route_kernel", "topk_kernel", "fast_plan_kernel",
            "fast_rot_kernel", "fast_gemm_kernel", "ep_combine_kernel", "ep_combine_ll_kernel", "ep_exchange_rows_kernel"} <= seen


@pytest.mark.parametrize("file,kernel,params,body", [pytest.param(*k, id=k[1]) for k in kernels() if "pdl_wait()" in k[3]])
def test_nothing_is_read_before_the_wait(file, kernel, params, body):
    front = body[:body.index("pdl_wait()")]
    bad = [p for p in names_read(params, front) if (kernel, p) not in BEHIND_ORDERED]
    assert not bad, f"{file}: {kernel} names {bad} before its wait"


def test_kernels_in_front_of_the_chunk_combine_wait_before_they_trigger():
    for file, kernel, _, body in kernels():
        if kernel in ("grouping_kernel", "fast_plan_kernel", "fast_rot_kernel", "fast_gemm_kernel"):
            assert body.index("pdl_wait()") < body.index("pdl_launch_dependents()"), f"{file}: {kernel} triggers before its wait"
