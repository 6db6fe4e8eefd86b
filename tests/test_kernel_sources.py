"""What the kernels' sources have to keep to, read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm_mojo_b200", "csrc")


def block(text, at):
    """The brace block that opens at ``at``, without its braces."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced braces")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        plain = set(re.findall(r"(\w+)\s*(?:<[^<>;]*>)?\s*<<<", text))
        for m in re.finditer(r"__global__[^;{}]*?\b(\w+_kernel)\s*\(", text):
            yield f"{os.path.basename(path)}:{m.group(1)}", block(text, text.index("{", m.end())), m.group(1) in plain


def exits_without_wait(body):
    """Blocks before the kernel's own pdl_wait() that return without one of their own (a lambda's return is not an exit)."""
    waits, bad, i = False, [], 0
    while i < len(body):
        if body.startswith("pdl_wait();", i):
            return True, bad
        if body.startswith("return", i) and not body[i - 1:i].isalnum():
            bad.append(body[max(0, i - 60):i + 10])
        if body[i] == "{":
            inner = block(body, i)
            is_lambda = re.search(r"\[[&=]?\]\s*(?:\([^()]*\))?\s*$", body[:i])
            if not is_lambda and re.search(r"\breturn\b", inner) and not re.search(r"pdl_wait\(\);.*\breturn\b", inner, re.S):
                bad.append(inner[:80])
            i += len(inner) + 1
        i += 1
    return waits, bad


@pytest.mark.parametrize("name,body", [(n, b) for n, b, plain in kernels() if not plain], ids=lambda v: v if ":" in v and len(v) < 60 else "")
def test_dependent_launches_wait_on_every_path(name, body):
    """A kernel launched with the programmatic attribute that exits without waiting completes while the kernel before it may still run,
    and the wait of the kernel after it covers this one only."""
    waits, bad = exits_without_wait(body)
    assert waits and not bad, (name, bad)


def unused_loads(text):
    """Inline loads none of whose results is read in the rest of the block they stand in."""
    bad = []
    for m in re.finditer(r'asm(?:\s+volatile)?\s*\("ld[^;]*?;"\s*:([^:;]*):[^;]*;', text):
        rest, depth = "", 0
        for ch in text[m.end():]:
            depth += {"{": 1, "}": -1}.get(ch, 0)
            if depth < 0:
                break
            rest += ch
        rest = re.sub(r'"=\w"\(\w+\)', "", rest)
        if not any(re.search(rf"\b{v}\b", rest) for v in re.findall(r'"=\w"\((\w+)', m.group(1))):
            bad.append(m.group(0))
    return bad


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_the_result_of_an_inline_load_is_read(path):
    """The assembler drops a plain load whose result nothing reads, volatile or not: it is no prefetch."""
    assert not unused_loads(re.sub(r"//[^\n]*", "", open(path).read()))


def test_the_check_sees_a_load_without_a_reader():
    load = 'asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));'
    assert len(unused_loads("{ uint32_t v; if (a) { " + load + load + " } }")) == 2
    assert not unused_loads("{ uint32_t v; " + load + " return v; }")


def test_the_check_sees_an_exit_without_a_wait():
    assert exits_without_wait("int a; if (a) { b(); return; } pdl_wait(); c();") == (True, [" b(); return; "])
    assert exits_without_wait("if (a) { pdl_wait(); return; } auto f = [&](int x) { return x; }; pdl_wait();") == (True, [])
    assert exits_without_wait("if (a) { pdl_wait(); } c();") == (False, [])
