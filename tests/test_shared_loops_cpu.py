"""A loop over chunks of work whose body holds block barriers must not step
by a shared variable: the step is read behind the body's last barrier, where a
warp that is ahead may already have written the next chunk's value (a warp
that then reads it takes other chunks than the rest of its block, or leaves
the loop at another barrier).  A parity run need not catch that; this check
reads the sources."""
import re

from test_launch_dep_lint_cpu import _kernel_bodies, _sources


def _strip_comments(text):
    return re.sub(r"/\*.*?\*/|//[^\n]*", " ", text, flags=re.S)


def _shared_names(body):
    names = set()
    for mo in re.finditer(r"__shared__\s+(?:__align__\(\d+\)\s*)?(?:unsigned\s+|const\s+)*\w+\s+([^;]*);", body):
        for part in mo.group(1).split(","):
            names.add(re.match(r"\s*(\w+)", part).group(1))
    return names


def _for_loops(body):
    """(step expression, loop body) of every for loop"""
    for mo in re.finditer(r"\bfor \(", body):
        depth, i = 1, mo.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        head = body[mo.end():i - 1].split(";")
        j = i + len(body[i:]) - len(body[i:].lstrip())
        if len(head) != 3:
            continue
        if body[j] != "{":
            yield head[2], body[j:body.index(";", j)]
            continue
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(body[k], 0)
            k += 1
        yield head[2], body[j:k]


def test_loops_with_barriers_do_not_step_by_shared_variables():
    looked, bad = 0, []
    for f, text in _sources().items():
        for name, body in _kernel_bodies(_strip_comments(text)):
            shared = _shared_names(body)
            for step, inner in _for_loops(body):
                if "__syncthreads" not in inner and ".sync()" not in inner:
                    continue
                looked += 1
                used = shared & set(re.findall(r"\w+", step))
                if used:
                    bad.append((f, name, step.strip(), sorted(used)))
    assert looked >= 1, "no loop with a barrier found"
    assert not bad, bad
