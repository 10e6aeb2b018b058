"""Order between threads and between launches, read off the kernel sources; nothing is launched.

A barrier that is crossed once per turn of a loop is met by all of its threads only if none of them leaves the loop, or skips to its
next turn ahead of the barrier, on its own account (a bounded wait that ran out in one warp and was met in the next)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "emmy_b200" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])
BARRIER = re.compile(r"__syncthreads(?:_and|_or|_count)?\s*\(|cluster_sync\s*\(|bar\.sync\b|barrier\.sync\b|barrier\.cta\b")
LEAVE = re.compile(r"\b(?:break|return|goto|continue)\b")


def _code(text):
    """Comments blanked; string literals stay, inline assembly is in them."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)


def _kind(lead):
    """What the text in front of a brace opens."""
    if re.match(r"(?:#pragma unroll[^\n]*\s+)?(?:for|while|do)\b", lead):
        return "loop"
    if lead.startswith("switch"):
        return "switch"
    return "lambda" if re.search(r"\[[&=\w, ]*\]\s*(?:\([^{}]*\))?$", lead) else "other"


def _blocks(code):
    """(start, end, kind) of every brace pair."""
    stack, out, head = [], [], 0
    for i, c in enumerate(code):
        if c == "{":
            stack.append((i, _kind(code[head:i].strip())))
            head = i + 1
        elif c == "}":
            start, kind = stack.pop()
            out.append((start, i, kind))
            head = i + 1
        elif c == ";" and code[head:i].count("(") == code[head:i].count(")"):  # not the semicolons of a loop's head
            head = i + 1
    return out


def deserters(text):
    """(line, word) of every statement by which a thread can miss a barrier that its loop crosses each turn."""
    code = _code(text)
    plain = re.sub(r'"(?:[^"\\\n]|\\.)*"', lambda m: " " * len(m.group()), code)  # the braces of inline assembly are not the program's
    blocks = _blocks(plain)

    def owner(at, kinds):
        return max(((s, e) for s, e, k in blocks if s < at < e and k in kinds), default=(-1, -1))

    found = []
    for start, end, kind in blocks:
        crossed = [m.start() for m in BARRIER.finditer(code, start, end) if owner(m.start(), {"loop", "lambda"}) == (start, end)]
        if kind != "loop" or not crossed:
            continue
        for m in LEAVE.finditer(plain, start, end):
            word = m.group()
            of = {"break": {"loop", "lambda", "switch"}, "continue": {"loop", "lambda"}}.get(word, {"lambda"})
            if owner(m.start(), of)[0] > start:  # it leaves a loop, switch or lambda inside this one
                continue
            if word == "continue" and m.start() > max(crossed):
                continue
            found.append((code.count("\n", 0, m.start()) + 1, word))
    return found


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_thread_leaves_a_loop_that_crosses_a_barrier(path):
    assert deserters(path.read_text()) == []


def test_the_reading_finds_what_it_looks_for():
    loop = """void f() {
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        if (x) { FIRST }
        asm volatile("{ bar.sync 1, 256; }" ::: "memory");
        if (!wait(t)) { flag(); LAST }
    }
}
"""
    read = lambda first, last: deserters(loop.replace("FIRST", first).replace("LAST", last))
    assert read("a();", "break;") == [(6, "break")]
    assert read("a();", "return;") == [(6, "return")]
    assert read("continue;", "") == [(4, "continue")]
    assert read("a();", "broken = true; continue;") == []
    assert read("for (int i = 0; i < 4; ++i) { if (i) break; }", "auto g = [&](int i) { return i; };") == []


@pytest.mark.parametrize(
    "source,kernel",
    [
        ("fp8_linear.cu", "quant_fp8_rows_vec_kernel"),
        ("fp8_block.cu", "quant_fp8_groups_kernel"),
        ("fp8_block.cu", "quant_fp8_groups_vec_kernel"),
        ("nvfp4_linear.cu", "quant_nvfp4_act_kernel"),
        ("nvfp4_linear.cu", "quant_nvfp4_act_atoms_kernel"),
    ],
)
def test_a_quantizer_on_its_own_releases_nothing(source, kernel):
    """A quantizer that is also an entry of its own (no status word) may be writing a weight, and a linear fetches its weights ahead of
    its wait: only inside a linear does it let the kernel behind it start."""
    code = _code((CSRC / source).read_text())
    body = code[code.index(kernel + "(") :]
    body = body[: body.index("\n}\n")]
    release = [line.strip() for line in body.splitlines() if "griddepcontrol.launch_dependents" in line]
    assert release and all(line.startswith("if (status) asm volatile") for line in release)
    assert "griddepcontrol.wait" in body
