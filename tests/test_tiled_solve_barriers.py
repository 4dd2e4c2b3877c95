"""The tiled solve's dot sums against its barriers, read off the source: no GPU.

Between two barriers of all CTAs the CTAs of a solve run in any order, so what
one of them writes there no other may read or write there. The sums of the
tree-order dots are the arrays that every CTA reads whole. This test takes the
statements of tw_solve (sdr_b200/csrc/pressure_tiles.cuh) from the first sweep
to the end of the third iteration in both forms (the cluster form folds the
direction into the next matvec and has a barrier fewer), in the default dot
order, and looks for an array that is written and used between two barriers."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sdr_b200", "csrc",
                   "pressure_tiles.cuh")


def _source():
    text = open(SRC).read()
    return re.sub(r"//[^\n]*", "", text)


def _block(text, at):
    """Text between the brace at `at` and the one that closes it, and the place behind."""
    assert text[at] == "{"
    depth = 0
    for q in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[q], 0)
        if depth == 0:
            return text[at + 1:q], q + 1
    raise AssertionError("unbalanced braces")


def _function(text, name):
    m = re.search(r"\b%s\([^;{]*\{" % name, text)
    return _block(text, m.end() - 1)[0]


def _paren(text, at):
    depth = 0
    for q in range(at, len(text)):
        depth += {"(": 1, ")": -1}.get(text[q], 0)
        if depth == 0:
            return text[at + 1:q], q + 1
    raise AssertionError("unbalanced parentheses")


def _taken(text, known):
    """The text with every `if (cond) {..} else {..}` of a known condition replaced by the branch it takes."""
    out, at = "", 0
    for m in iter(lambda: re.compile(r"\bif \(").search(text, at), None):
        cond, end = _paren(text, m.end() - 1)
        cond = " ".join(cond.split())
        out += text[at:m.start()]
        at = end
        if cond not in known:
            out += "if_(" + cond + ")"
            continue
        brace = text.index("{", at)
        assert not text[at:brace].strip(), cond
        yes, at = _block(text, brace)
        no = ""
        if re.match(r"\s*else \{", text[at:]):
            no, at = _block(text, text.index("{", at))
        out += _taken(yes if known[cond] else no, known)
    return out + text[at:]


def _last(name):
    return re.split(r"\.|->", name)[-1]


def _events(cluster, iterations=3):
    src = _source()
    solve = _function(src, "tw_solve")
    matvec_writes = _last(re.search(r"if \(lane == 0\) (\S+)\[tb \+ w\] = acc", _function(src, "tw_matvec_by")).group(1))
    zr_writes = _last(re.search(r"if \(lane == 0\) (\S+)\[tl\] = acc", _function(src, "tw_dot_zr")).group(1))
    total_reads = set(re.findall(r"__ldcg\((\S+) \+", _function(src, "tw_tile_total")))
    assert len(total_reads) == 1
    total_reads = total_reads.pop()
    loop = re.search(r"for \(int it = 0; it < a\.max_iters; \+\+it\) \{", solve)
    body, _ = _block(solve, loop.end() - 1)
    before = solve[solve.index("tw_sweep_all<TW_FORWARD"):loop.start()]
    texts = [_taken(before, {"a.exact_dots": False})]
    for it in range(iterations):
        texts.append(_taken(body, {"a.exact_dots": False, "CL && it > 0": cluster and it > 0, "!CL": not cluster}))
    events = []
    call = re.compile(r"\b(tw_grid_sync|tw_grid_max|tw_matvec|tw_dot_zr|tw_tile_total)\b(?:<\w+>)?\(([^,)]*)")
    for text in texts:
        for m in call.finditer(text):
            what, arg = m.group(1), m.group(2)
            if what in ("tw_grid_sync", "tw_grid_max"):
                events.append(("barrier", what))
            elif what == "tw_matvec":
                events.append(("write", matvec_writes))
            elif what == "tw_dot_zr":
                events.append(("write", zr_writes))
            else:
                events.append(("read", _last(arg) if total_reads == "sums" else _last(total_reads)))
    return events


@pytest.mark.parametrize("cluster", [False, True])
def test_dot_sums_are_parted_by_barriers(cluster):
    events = _events(cluster)
    # the dots of the solve: z*r before the loop and s*As and z*r in each iteration
    assert sum(e[0] == "write" for e in events) == 7 and sum(e[0] == "read" for e in events) == 7
    between = [[]]
    for kind, name in events:
        if kind == "barrier":
            between.append([])
        else:
            between[-1].append((kind, name))
    for step in between:
        for q, (kind, name) in enumerate(step):
            rest = step[:q] + step[q + 1:]
            assert kind != "write" or all(other != name for _, other in rest), step
    # and every sum that is read was written before
    written = set()
    for kind, name in events:
        if kind == "write":
            written.add(name)
        assert kind != "read" or name in written
