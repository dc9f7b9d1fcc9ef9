"""Kernels launched with programmatic serialisation (launch.cuh) become resident
while the kernel before them still runs, so what a step writes must be read behind
their dep_wait() / pair_begin() by coherent loads: not through the read-only path,
whose data nobody may write during the kernel's lifetime, not through a pointer
declared unaliased (the compiler may turn such a load into the read-only one, or
move it above the wait), and not by an intrinsic that the compiler may move.
Read from the sources: such a load goes wrong only now and then."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "konglong_b200", "csrc")
# what no kernel of a step writes: model volumes, tile and factor tables, line matrices
CONSTANT = {"vel", "eps", "del", "pjx", "pjy", "rho", "tiles", "Bg", "tl", "tu", "tr"}


def _sources():
    return {f: re.sub(r"//[^\n]*", "", open(f).read())
            for f in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))}


def _functions(text):
    """{name: (parameters, body, is a kernel)} of the device functions."""
    out = {}
    for m in re.finditer(r"__(global|device)__", text):
        head = re.compile(r"\b(\w+)\s*\(").search
        at = m.end()
        while True:  # the name before the parameter list, past __launch_bounds__(...)
            h = head(text, at)
            if h is None or h.group(1) not in ("__launch_bounds__", "__align__"):
                break
            at = _close(text, h.end() - 1)
        if h is None:
            continue
        end = _close(text, h.end() - 1)
        brace = re.compile(r"\s*(const\s*)?\{").match(text, end)
        if brace is None:
            continue
        body_end = _close(text, brace.end() - 1)
        name, params, body = h.group(1), text[h.end():end - 1], text[brace.end():body_end - 1]
        old = out.get(name, ("", "", False))
        out[name] = (old[0] + "," + params, old[1] + body, old[2] or m.group(1) == "global")
    return out


def _close(text, at):
    """The place behind the bracket that closes the one at `at`."""
    pair = {"(": ")", "{": "}"}
    o, c, depth = text[at], pair[text[at]], 0
    for k in range(at, len(text)):
        depth += (text[k] == o) - (text[k] == c)
        if depth == 0:
            return k + 1
    raise ValueError("unbalanced source")


def _reached(name, funcs):
    seen, todo = set(), [name]
    while todo:
        f = todo.pop()
        if f in seen or f not in funcs:
            continue
        seen.add(f)
        todo += re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", funcs[f][1])
    return seen


def _dependent():
    """(file, kernel, device functions it can see) of every dependent kernel."""
    src = _sources()
    shared = {}
    for f, text in src.items():
        if f.endswith(".cuh"):
            shared.update(_functions(text))
    for f, text in src.items():
        if f.endswith(".cu"):
            funcs = dict(shared, **_functions(text))
            for name, (_, body, kernel) in funcs.items():
                if kernel and re.search(r"\b(dep_wait|pair_begin)\s*\(", body):
                    yield os.path.basename(f), name, funcs


DEPENDENT = sorted(_dependent(), key=lambda d: d[:2])


def test_every_dependent_launch_is_of_a_waiting_kernel():
    waiting = {name for _, name, _ in DEPENDENT}
    assert len(waiting) >= 14
    for f, text in _sources().items():
        for k in re.findall(r"\blaunch_dep\(\s*(\w+)", text):
            if k == "k":  # chosen just before
                named = re.findall(r"auto \*k = [^;]*;", text)
                assert named and all(set(re.findall(r"\b(\w+_k)\b", n)) <= waiting for n in named)
            elif k != "void":
                assert k in waiting, (f, k)


@pytest.mark.parametrize("file, kernel", [d[:2] for d in DEPENDENT])
def test_step_data_is_read_by_coherent_loads(file, kernel):
    funcs = next(d[2] for d in DEPENDENT if d[:2] == (file, kernel))
    wrong = []
    for f in sorted(_reached(kernel, funcs)):
        params, body, _ = funcs[f]
        for decl in re.findall(r"[^,;(){}]*__restrict__\s*\w+", params + ";" + body):
            if decl.split()[-1] not in CONSTANT:
                wrong.append("%s: %s" % (f, " ".join(decl.split())))
        for m in re.finditer(r"\b(__ldg|ldg|__ldcg|__ldca|__ldcs|__ldlu)\s*(?:<[^>]*>)?\s*\(", body):
            arg = body[m.end():_close(body, m.end() - 1) - 1]
            if m.group(1) not in ("__ldg", "ldg") or not set(re.findall(r"\w+", arg)) & CONSTANT:
                wrong.append("%s: %s(%s)" % (f, m.group(1), arg))
    assert not wrong, wrong
