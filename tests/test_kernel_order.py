"""What the kernels order before what, read from their source: a missing wait or warp
synchronisation shows in no result that a test could rely on."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def kernel(file, name):
    """The text of a kernel without its comments, from its name to the brace that closes it."""
    text = open(os.path.join(ROOT, "sinking-simulator_b200", "csrc", file)).read()
    text = re.sub(r"//[^\n]*", "", text)
    start = re.search(r"\b%s\(" % name, text[text.index("__global__"):]).start() + text.index("__global__")
    depth = 0
    for at in range(text.index("{", start), len(text)):
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        if depth == 0:
            return text[start:at + 1]
    raise AssertionError("unbalanced")


def test_shell_rotation_is_synchronised_before_its_readers():
    """Narrow form: one lane an element leaves the rotation in shared memory and all eight
    read it for the forces.  A warp that finishes at its first test passes no other
    synchronisation in between, so the next statement on shared memory after the store's
    own record has to be one."""
    body = kernel("shell_step.cu", "shell_forces")
    stores = [m.end() for m in re.finditer(r"\bgeo\[kGeoQ \+ k\] = q\[k\];", body)]
    assert len(stores) == 1
    after = body[stores[0]:]
    sync = after.index("__syncwarp();")
    assert sync < after.index("load_record<"), "the rotation is stored after the last synchronisation"
    assert sync < after.index("geo[kGeoQ + k]")


def test_shell_order_is_written_before_the_next_kernel_may_start():
    """The element pass reads the order of its groups before it waits for the pass ahead, so
    the block that renews it must not let the next kernel start first."""
    body = kernel("shell_step.cu", "shell_nodes")
    assert "pdl_next();" in body
    assert "pdl_next();" not in body[:body.index("shell_order(")]
