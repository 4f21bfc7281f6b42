"""What a kernel launched to overlap its predecessor may do before its wait,
read from the source: such a kernel must not hold tensor memory while it waits
(the kernel ahead, when it is a caller's that lets dependents in early, could
still have to allocate its own, and neither would go on)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "physis_gb300",
                    "csrc")


def _bodies(text):
    """(name, body) of every __global__ function."""
    attributes = r"(?:\s*__(?:launch_bounds|maxnreg|cluster_dims)__\([^)]*\))*"
    head = r"__global__(?: void)?" + attributes + r"(?: void)?" + attributes
    for m in re.finditer(head + r"\s*(\w+)\s*\([^{;]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def test_tensor_memory_is_allocated_after_the_wait():
    text = open(os.path.join(CSRC, "nn.cu")).read()
    bodies = dict(_bodies(text))
    overlapped = set(re.findall(r"launch_kernel\(\s*(\w+)", text))
    assert "conv_pad_kernel" in overlapped
    seen = 0
    for name in overlapped:
        body = bodies[name]
        assert "wait_for_predecessors();" in body, name
        if "tcgen05.alloc" in body:
            seen += 1
            assert body.index("wait_for_predecessors();") < body.index("tcgen05.alloc"), name
    assert seen == 1
