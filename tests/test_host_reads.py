"""The host does not read the pinned copy of a step's scalars while the device is
still writing it: step_once queues kernels between the copy and the wait for it, and
neither it nor what it calls there may look at h_scalars.  Read from the source, as
the values agree in any run that happens to be fast enough."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def body(text, head):
    """The braces of the first definition that matches head."""
    m = re.search(head + r"[^;{]*\{", text)
    assert m, head
    depth, k = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        k += 1
    return text[m.end():k]


def test_no_host_read_while_the_scalars_are_copied():
    text = open(os.path.join(ROOT, "cuda-rp_b200", "csrc", "sim.cu")).read()
    text = re.sub(r"//[^\n]*", "", text)
    step = body(text, r"crp_status step_once\(\)")
    start = step.index("cudaMemcpyAsync(h_scalars")
    window = step[step.index("if (ahead) {", start):step.index("cudaEventSynchronize(ev)", start)]
    assert "picard_gate" in window
    called = set(re.findall(r"\b(build_order|launch_[a-z]+|[a-z]+_kernel)\b", window))
    assert {"build_order", "launch_rp"} <= called
    called.add("radius_kernel")
    for f in called:
        assert "h_scalars" not in body(text, r"\b(?:cudaError_t|auto|crp_status) " + f + r"\("), f
    assert "h_scalars" not in window
