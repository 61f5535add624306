"""What the order of a few instructions in the kernels' sources has to be, read from the sources: on a GPU the wrong order shows only
by chance, and as a hang."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwenny_b200", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for body in re.split(r"(?=__global__ void)", src)[1:]:
            name = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^{;]*?\)\s*(?=\w+\s*\()|__cluster_dims__\([^)]*\)", "", body[len("__global__ void"):]))
            yield os.path.basename(path), name.group(1), body


def test_dependents_start_only_once_tensor_memory_is_held():
    """tcgen05.alloc waits without a limit. A kernel that lets its dependents start before its own blocks hold their tensor memory can find
    it taken by a dependent's block, which waits for the kernel's end. (A block that returns before it takes any may let them start.)"""
    seen = 0
    for where, name, body in kernels():
        at = body.find("tcgen05.alloc.")
        if at < 0:
            continue
        seen += 1
        for m in re.finditer(r"pdl_launch_dependents\(\);", body[:at]):
            assert re.match(r"\s*(pdl_wait\(\);)?\s*return;", body[m.end():]), f"{where}: {name} lets its dependents start before it holds tensor memory"
        assert "pdl_launch_dependents();" in body[at:], f"{where}: {name}"
    assert seen == 5


def test_the_first_kernels_of_a_step_wait_before_they_let_others_start():
    """What the model runner reads ahead of its kernels relies on it (launch.h)."""
    first = {name: body for _, name, body in kernels() if name in ("mark_seen_kernel", "embed_kernel")}
    assert len(first) == 2
    for name, body in first.items():
        assert 0 <= body.find("pdl_wait();") < body.find("pdl_launch_dependents();"), name


def test_decode_attention_follows_its_rings_order():
    """The order in which a block's quads share the ring's slots is dec_ring.h's, played through by test_dec_ring_cpu.py; here only that the
    kernel takes it from there: it looks for its stage's number before it waits, and writes the number behind the slot's barrier."""
    body = {name: body for _, name, body in kernels()}["attn_dec4_kernel"]
    wait = body.index("mbar_wait(&full[sl], par)")
    looks = body.rfind("while (issued[sl] != order.number(j)", 0, wait)
    assert looks > 0 and "if (Ring::looks(j))" in body[looks - 60:looks] and "par = order.parity(j)" in body[looks - 400:looks]
    asks = body.index("mbar_expect_tx(")
    assert re.match(r"mbar_expect_tx\([^;]*\);\s*issued\[Ring::slot\(j\)\] = order\.number\(j\);", body[asks:])
