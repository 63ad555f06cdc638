"""Kernels launched as dependent passes start before their predecessors end and
wait in begin_pass (csrc/dev_common.cuh).  A load through a `const
__restrict__` parameter, or `__ldg`, counts as invariant to the compiler and
may be moved above that wait where it always runs, so what stands unguarded
after begin_pass must not hold one.  Read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "hetegeneous_parallel_programming_gb300" / "csrc"


def closing(text, at):
    """Index past the bracket that closes the one at `at`."""
    pairs, depth = {"(": ")", "{": "}", "[": "]"}, 0
    opened, closed = text[at], pairs[text[at]]
    for i in range(at, len(text)):
        depth += (text[i] == opened) - (text[i] == closed)
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def statement(text, at):
    """Index past the statement or block that starts at `at`."""
    while text[at].isspace():
        at += 1
    if text[at] == "{":
        return closing(text, at)
    head = re.match(r"(if|for|while)\s*(?=\()", text[at:])
    if head:
        end = statement(text, closing(text, at + head.end()))
        other = re.match(r"\s*else\b", text[end:])
        return statement(text, end + other.end()) if other else end
    while text[at] != ";":
        at = closing(text, at) if text[at] in "({[" else at + 1
    return at + 1


def always_runs(text):
    """The parts of a block that run whatever the data, up to its first guarded return."""
    out, at = "", 0
    while at < len(text):
        head = re.match(r"\s*(if|for|while)\s*(?=\()", text[at:])
        if not head:
            end = at + 1 if text[at].isspace() else statement(text, at)
            out += text[at:end]
            at = end
            continue
        cond0 = at + head.end()
        cond1 = closing(text, cond0)
        cond = text[cond0 + 1:cond1 - 1]
        end = statement(text, at)
        body = text[cond1:end]
        if head.group(1) == "for":
            cond = ";".join(cond.split(";")[:2])
            if re.search(r"<\s*[A-Z][A-Z_0-9]+(\s*/\s*\d+)?\s*$", cond):  # a constant number of rounds
                out += always_runs(body.strip()[1:-1] if body.strip().startswith("{") else body)
        out += cond + ";"
        if head.group(1) == "if" and re.match(r"\s*\{?\s*return\b", body):
            return out
        at = end
    return out


def dependent_kernels():
    found = {}
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/|^\s*#[^\n]*", "", path.read_text(), flags=re.S | re.M)
        for k in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^)]*\)\s*)?(\w+)\s*(?=\()", text):
            params_end = closing(text, k.end())
            body_at = re.match(r"\s*\{", text[params_end:])
            if not body_at:
                continue
            at = params_end + body_at.end() - 1
            body = text[at + 1:closing(text, at) - 1]
            if "begin_pass();" in body:
                found[k.group(1)] = (text[k.end() + 1:params_end - 1], body.split("begin_pass();", 1)[1])
    return found


KERNELS = dependent_kernels()


def unguarded_reads(params, body):
    straight = always_runs(body)
    names = re.findall(r"const\s+[\w:]+(?:\s+\w+)*\s*\*\s*__restrict__\s+(\w+)", params)
    bad = [n for n in names
           if re.search(rf"\b{n}\s*\[|(?<![\w)\]]\s)(?<![\w)\]])\*\s*{n}\b|[(,]\s*{n}\s*(?=[,)])", straight)]
    return bad + re.findall(r"__ldg\s*\(", straight)


def test_the_check_sees_what_it_is_for():
    assert len(KERNELS) > 20 and "direct_place_kernel" in KERNELS
    for params, body, bad in (("const int *__restrict__ a", "int x = a[0];", ["a"]),
                              ("const int *__restrict__ a", "if (off(a, 3)) return;", ["a"]),
                              ("const int *__restrict__ a", "const int n = *a;", ["a"]),
                              ("const int *__restrict__ a", "for (int k = 0; k < PER; ++k) s += a[k];", ["a"]),
                              ("const int *a", "int x = a[0];", []),
                              ("const int *__restrict__ a", "for (int i = 0; i < n; ++i) s += a[i];", []),
                              ("const int *__restrict__ a", "if (n == 0) return;\nint x = a[0];", []),
                              ("const int *__restrict__ a", "const int4 *p = f<int4 *>(a + 4);", [])):
        assert unguarded_reads(params, body) == bad, body


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_unguarded_invariant_load(name):
    assert unguarded_reads(*KERNELS[name]) == []


def test_the_off_check_is_ordered_by_the_wait():
    """direct_off is the first read of every later direct pass: an instruction of its own, so no pass takes it early."""
    text = (CSRC / "direct.cu").read_text()
    body = text[text.index("bool direct_off("):]
    assert re.search(r"asm volatile\(\"ld\.global[^;]*;\"[^;]*\"memory\"\)", body[:closing(body, body.index("{"))])
