"""The hand-over between the warps of the column scans, as a model that walks every interleaving.

What each role waits for and signals is read from the kernels' sources; the model then checks, for any
order in which the warps and the copies can run, that no wait misses its phase (a parity wait that comes
two phases late blocks for good) and that nobody reads a tile or slot of another chunk.
"""

import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "delta_feedback_experiment_b200", "csrc")
STAGES, SLOTS = 3, 2
OPS = re.compile(r"\b(?:tc::)?(mbar_wait2|mbar_wait|warp_arrive|mbar_arrive|mbar_expect_tx)\(")
LOOP = re.compile(r"for \(int [ij] = 0; [ij] < sq\.nchunks; \+\+[ij]\) \{")
SHARED = "const bool out = kOut && role == 1;"   # one loop for the output warps (out) and the store warps


def _closing(text, at, pair):
    """Index behind the bracket that closes the one opened just before ``at``."""
    depth = 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        at += 1
    return at


def _as_role(text, out):
    """The loop body as one role runs it: the branches on ``out`` resolved."""
    while m := re.search(r"if \((!?)out\) \{", text):
        end = _closing(text, m.end(), "{}")
        body, rest = text[m.end():end - 1], text[end:]
        other = ""
        if e := re.match(r" else \{", rest):
            stop = _closing(rest, e.end(), "{}")
            other, rest = rest[e.end():stop - 1], rest[stop:]
        taken = body if out != bool(m.group(1)) else other
        text = text[:m.start()] + taken + ("" if "continue;" in taken else rest)
    return text


def _ops(text):
    ops = []
    for m in OPS.finditer(text):
        bars = re.findall(r"\bbar_(full|empty|ready|free)\b", text[m.end():_closing(text, m.end(), "()")])
        if m.group(1) == "mbar_expect_tx":
            bars = ["full"]
        ops += [("wait" if "wait" in m.group(1) else "signal", b) for b in bars]
    return ops


def roles_of(source):
    """``{role: [("wait" | "signal", barrier), ...]}`` of one chunk, in the order of the source."""
    text = open(os.path.join(CSRC, source)).read()
    marks = [(m.group(1), m.end()) for m in re.finditer(r"// -{8,} the (copies|chain|stores)\b", text)]
    if SHARED in text:
        marks.append(("shared", text.index(SHARED)))
    ends = [at for _, at in marks[1:]] + [text.index("template <int NW", marks[-1][1])]
    roles = {}
    for (name, at), end in zip(marks, ends):
        loop = LOOP.search(text, at)
        block = text[loop.end():min(end, _closing(text, loop.end(), "{}"))]
        if name == "shared":
            roles.update(output=_ops(_as_role(block, True)), stores=_ops(_as_role(block, False)))
        else:
            roles[name] = _ops(block)
    return roles


def walk(roles, groups, chunks):
    """Visits every reachable state; returns the first fault found, or None."""
    users = sum(1 for r in ("chain", "output") if ("signal", "empty") in roles.get(r, ()))
    readers = sum(1 for r in ("output", "stores") if ("signal", "free") in roles.get(r, ()))
    need = {"empty": groups * users, "ready": 1, "free": readers}
    workers = [(name, g) for name in roles if name != "copies" for g in range(groups)]
    bars = ([("full", s) for s in range(STAGES)] + [("empty", s) for s in range(STAGES)] +
            [(b, g, s) for b in ("ready", "free") for g in range(groups) for s in range(SLOTS)])
    index = {b: i for i, b in enumerate(bars)}

    def bar(name, g, i):
        return index[(name, i % STAGES) if name in ("full", "empty") else (name, g, i % SLOTS)]

    def turn(name, i):   # the phase of the barrier that belongs to chunk i
        return i // (STAGES if name in ("full", "empty") else SLOTS)

    # state: phases completed and arrivals of the running one per barrier, position per worker, chunks asked
    # for by the copy warp, chunks landed
    start = (tuple((0, 0) for _ in bars), tuple((0, 0) for _ in workers), 0, 0)
    seen, todo = {start}, [start]
    while todo:
        phases, pos, asked, landed = todo.pop()
        nxt = []

        def signal(ph, at, count):
            done, got = ph[at]
            ph = list(ph)
            ph[at] = (done + 1, 0) if got + 1 == count else (done, got + 1)
            return tuple(ph)

        if asked < chunks:   # the copy warp: bar_empty of the chunk that held the stage before
            e = index[("empty", asked % STAGES)]
            if asked < STAGES or (phases[e][0] - 1) % 2 == (asked // STAGES - 1) % 2:
                nxt.append((phases, pos, asked + 1, landed))
        if landed < asked:   # a copy arrives (the copies of a stage are one transaction count)
            nxt.append((signal(phases, index[("full", landed % STAGES)], 1), pos, asked, landed + 1))
        for w, (name, g) in enumerate(workers):
            i, k = pos[w]
            if i == chunks:
                continue
            kind, b = roles[name][k]
            at = bar(b, g, i)
            if kind == "wait":
                # bar_free is waited for before the slot is written: the phase before the chunk's own
                want = turn(b, i) - (1 if b == "free" else 0)
                if (phases[at][0] - 1) % 2 != want % 2:
                    continue
                if phases[at][0] - 1 != want:
                    return f"{name} {g} passes {b} of chunk {i} in phase {phases[at][0] - 1} instead of {want}"
                ph = phases
            else:
                if b == "empty" and asked > i + STAGES:
                    return f"{name} {g} read the stage of chunk {i} after it was asked for again"
                if b == "free" and phases[index[("ready", g, i % SLOTS)]][0] != turn(b, i) + 1:
                    return f"{name} {g} read the slot of chunk {i} after it was written again"
                ph = signal(phases, at, need[b])
            p = list(pos)
            p[w] = (i, k + 1) if k + 1 < len(roles[name]) else (i + 1, 0)
            nxt.append((ph, tuple(p), asked, landed))
        if not nxt and (landed < chunks or any(i < chunks for i, _ in pos)):
            return "stuck: " + ", ".join(f"{n} {g} at chunk {i}" for (n, g), (i, _) in zip(workers, pos))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("source,outputs", [("pkda_scan_fwd.cu", True), ("pkda_scan_fwd.cu", False),
                                            ("pkda_scan_bwd.cu", False)])
@pytest.mark.parametrize("groups,chunks", [(1, 9), (2, 5)])
def test_no_wait_misses_its_phase(source, outputs, groups, chunks):
    roles = roles_of(source)
    assert {"copies", "chain", "stores"} <= set(roles), "a role of the scan was not found in the source"
    assert roles["copies"] == [("wait", "empty"), ("signal", "full")]
    assert ("wait", "ready") in roles["stores"] and ("signal", "free") in roles["stores"]
    if not outputs:
        roles.pop("output", None)
    assert walk(roles, groups, chunks) is None


@pytest.mark.parametrize("outputs", [True, False])
def test_a_wait_for_a_stage_that_goes_on_alone_is_found(outputs):
    """The store warp holds no stage: were it to wait for the stage's barrier too, it could come two phases late."""
    roles = roles_of("pkda_scan_fwd.cu")
    if not outputs:
        roles.pop("output")
    roles["stores"] = [("wait", "full"), *roles["stores"]]
    assert "stuck" in walk(roles, 1, 9)
