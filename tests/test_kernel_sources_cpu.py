"""Orders inside kernels whose violation would stop a GPU: shown on the sources, never by running a kernel that breaks them."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mllm_b200" / "csrc"


def _kernels(path):
    """(name, body) of the ``__global__`` functions of a source, without comments."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        at = text.index("{", text.index(")", m.end()))
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), text[at:end]


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_tensor_memory_is_allocated_before_the_next_kernel_may_start(source):
    """tcgen05.alloc waits until its columns are free.  A kernel that has let the next one start before it has its own would wait for
    blocks that wait for its end."""
    for name, body in _kernels(CSRC / source):
        alloc, trigger = re.search(r"\btmem_alloc(_pair)?\(", body), re.search(r"\bpdl_launch_dependents\(", body)
        if alloc and trigger:
            assert alloc.start() < trigger.start(), name


def _roles(body):
    """The branches of a kernel's body in their order, statements between them included: (text, whether it is a branch)."""
    depth, at = 0, 1
    for i, c in enumerate(body[1:-1], 1):
        depth += {"{": 1, "}": -1}.get(c, 0)
        if c == "{" and depth == 1:
            yield body[at:i], False
            at = i
        elif c == "}" and depth == 0:
            yield body[at:i + 1], True
            at = i + 1
    yield body[at:-1], False


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_bounded_waits_begin_behind_the_stream_order_wait(source):
    """A kernel that is launched early stays resident for as long as the kernels in front run.  A role whose bounded wait began before
    the stream-order wait would count their time against its limit and give up in a healthy run."""
    for name, body in _kernels(CSRC / source):
        ordered = False
        for text, branch in _roles(body):
            first = re.search(r"\bmbar_wait\w*\(", text)
            wait = re.search(r"\bpdl_wait(_loads)?\(\)", text)
            if branch and first and not ordered:
                assert wait and wait.start() < first.start(), (name, text[:80])
            ordered = ordered or (wait is not None and not branch)


# what the kernels read through the read-only path: parameters, which no kernel writes
PARAMETERS = ("p.scales", "p.zeros")


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_read_only_loads_without_a_fence_are_of_parameters(source):
    """Loads through the read-only path are not ordered by the stream-order wait: where it stands without its fence they may return
    what was in a buffer before the kernel in front wrote it."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", (CSRC / source).read_text(), flags=re.S)
    for name, body in _kernels(CSRC / source):
        if "pdl_wait_loads()" in body and "pdl_wait()" not in body:
            for m in re.finditer(r"__ldg\(", body):
                assert any(p in body[m.end():m.end() + 70] for p in PARAMETERS), (name, body[m.start():m.end() + 70])
    if "pdl_wait_loads()" in text and "pdl_wait()" not in text:
        for m in re.finditer(r"__ldg\(", text):
            assert any(name in text[m.end():m.end() + 70] for name in PARAMETERS), text[m.start():m.end() + 70]


def test_prefill_attention_without_its_registers_is_left_to_the_other_kernel():
    """Fewer registers than the roles share out are a compiler's choice and no error of the call: 1 takes the single-role kernel."""
    text = (CSRC / "attention.cu").read_text()
    launch = text[text.index("int launch_prefill_ws("):]
    assert re.search(r"if \(regs \*[^;]*\) return (-?\d+);", launch[:launch.index("\n}\n")]).group(1) == "1"
