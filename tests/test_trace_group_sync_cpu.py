"""k_trace_group shares one stack in shared memory among eight lanes: lane 0
pushes, all pop, often in the same step.  Votes and shuffles order no memory,
so a __syncwarp() that every lane reaches has to stand between the push and
the pop, and another between the pop and the next step's push.  Hardware that
happens to run the lanes together gives right answers without them, so this
reads the kernel's source."""
from __future__ import annotations

import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "firefly_b200" / "csrc" / "ff_trace.cu"


def _kernel():
    text = SRC.read_text()
    start = text.index("k_trace_group(FFBvhView")
    body = text[text.index("{", start):]
    depth = 0
    for i, c in enumerate(body):
        depth += {"{": 1, "}": -1}.get(c, 0)
        if depth == 0:
            return body[:i + 1]
    raise AssertionError("unbalanced braces")


def _loop_syncs(body):
    """Offsets of the __syncwarp() calls directly in the persistent loop, i.e.
    in no branch (a lane could miss those)."""
    depth, out = 0, []
    for m in re.finditer(r"[{}]|__syncwarp\(\)", body):
        if m.group() == "{":
            depth += 1
        elif m.group() == "}":
            depth -= 1
        elif depth == 2:     # the function's body, the loop's
            out.append(m.start())
    return out


def test_a_barrier_stands_between_push_and_pop():
    body = _kernel()
    push = [m.start() for m in re.finditer(r"stack\[sp\]\s*=", body)]
    pop = [m.start() for m in re.finditer(r"=\s*stack\[--sp\]", body)]
    assert len(push) == 1 and len(pop) == 1 and push[0] < pop[0]
    syncs = _loop_syncs(body)
    assert any(push[0] < s < pop[0] for s in syncs), "push and pop in one step without a barrier"
    assert any(s > pop[0] or s < push[0] for s in syncs), "pop and the next step's push without a barrier"
