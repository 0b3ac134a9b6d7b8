"""Rules of the step loop's kernels that no result can show on every run, checked in their source.

With programmatic launch a kernel of the step loop is resident while the kernels before it still
run.  So it touches no memory before griddepcontrol.wait, and what another kernel of the loop
writes (the weights of plastic edges) it does not read through the read-only path: ld.global.nc
asks for data that stay constant for the kernel's whole life, the wait included."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nest-gpu_b200", "csrc")


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(src, start):
    """The braced block that opens at or after `start`."""
    a = src.index("{", start)
    depth = 0
    for i in range(a, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[a + 1:i]
    raise ValueError("unbalanced braces")


def test_delivery_reads_weights_past_the_read_only_path():
    src = _read("ngpu_kernels.cu")
    body = _body(src, src.index("void deliver_batch("))
    assert "A.edge" in body
    assert not re.findall(r"__ldg\([^;]*edge[^;]*;", body)
    load = _body(src, src.index("load_edge("))
    assert "__ldcg" in load and "__ldg(" not in load


def test_kernels_of_the_step_loop_wait_first():
    n = 0
    for name in ("ngpu_kernels.cu", "ngpu_stdp.cu", "ngpu_aeif.cuh"):
        src = _read(name)
        for m in re.finditer(r"__global__ void[^{;]*?(\w+_kernel)\(", src):
            if not re.search(r"launch_k\(%s\b" % m.group(1), src):
                continue
            assert _body(src, m.end()).lstrip().startswith("pdl_enter();"), m.group(1)
            n += 1
    assert n >= 12
