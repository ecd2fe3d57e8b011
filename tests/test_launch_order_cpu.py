"""Kernels that are scheduled when the one before them ends (launch_kernel, launch_clusters) wait for its writes before their first access to global memory, and
have nothing that lets a load go ahead of that wait: no `__restrict__` pointer and no read-only load, which count as constant for the whole kernel."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "maidenx_b200" / "csrc"
WAIT = "after_previous_kernel();"


def _closing(text, at, pair):
    """The place behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced source")


def _without_comments(text):
    return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S)


def _kernels(text):
    """(name, parameters, body) of every kernel that `text` defines."""
    for m in re.finditer(r"__global__", text):
        i = m.end()
        bounds = re.compile(r"\s*void\s*__launch_bounds__\s*\(|\s*__launch_bounds__\s*\(").match(text, i)
        if bounds:
            i = _closing(text, bounds.end() - 1, "()")
        head = re.compile(r"\s*(?:void\s+)?(\w+)\s*\(").match(text, i)
        assert head, text[m.start():m.start() + 120]
        end = _closing(text, head.end() - 1, "()")
        body = re.compile(r"\s*\{").match(text, end)
        if body:  # else a declaration
            yield head.group(1), text[head.end():end], text[body.end():_closing(text, body.end() - 1, "{}")]


def violations(sources):
    text = {name: _without_comments(s) for name, s in sources.items()}
    everything = "\n".join(text.values())
    ordinary = set(re.findall(r"(\w+)\s*(?:<[^;{}]*?>)?\s*<<<", everything))
    bad = []
    for file, s in text.items():
        for name, params, body in _kernels(s):
            waits = WAIT in body
            if not waits and name not in ordinary:
                bad.append(f"{file}: {name} is started by launch_kernel and does not wait")
            if waits and "__restrict__" in params + body:
                bad.append(f"{file}: {name} waits and has a __restrict__ pointer")
            if waits and re.search(r"__ldg|ld\.global\.nc|ldg", body):
                bad.append(f"{file}: {name} waits and reads as constant")
        for m in re.finditer(r"__device__ __forceinline__[^;{]*\{", s):  # parts of kernels
            if "__restrict__" in m.group(0):
                bad.append(f"{file}: {m.group(0)[:80]}")
    return bad


def _sources():
    return {p.name: p.read_text() for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}


def test_kernels_that_wait_read_nothing_as_constant():
    assert not violations(_sources())


def test_the_rule_finds_what_breaks_it():
    s = _sources()
    assert len([k for t in s.values() for k in _kernels(_without_comments(t))]) > 50
    broken = dict(s, **{"extras.cu": s["extras.cu"].replace("softmax_rows_kernel(const T* in,", "softmax_rows_kernel(const T* __restrict__ in,")})
    assert any("softmax_rows_kernel waits" in v for v in violations(broken))
    silent = dict(s, **{"conv_s1.cuh": s["conv_s1.cuh"].replace(WAIT, "")})
    assert any("im2col_s1_kernel is started" in v for v in violations(silent))


def gate_without_launch(source):
    """What is wrong with how tc_launch_f32_pairs hands out its gate: a gate that is set where nothing was launched stays shut, and the product behind it is never computed."""
    s = _without_comments(source)
    head = re.search(r"bool tc_launch_f32_pairs\([^)]*\)\s*\{", s)
    body = s[head.end():_closing(s, head.end() - 1, "{}")]
    at = [m.start() for m in re.finditer(r"\brun\.gate(\.\w+)?\s*=[^=]", body)]
    return [] if at and "return false" not in body[at[0]:] and body.index("split_pairs_kernel") > at[0] else ["the caller's gate is set before the last way out without a launch"]


def test_a_product_in_pairs_that_is_not_launched_leaves_no_gate():
    s = _sources()["matmul_tc_pairs.cu"]
    assert not gate_without_launch(s)
    assert gate_without_launch(s.replace("Gate mine;", "Gate mine; run.gate = mine;"))
