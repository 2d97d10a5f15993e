"""Control flow of kernels that cannot be provoked on a device: what a wait that runs out does in
the middle of a launch is checked on the source."""

import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "snoo.py_b200", "csrc")


def _kernel(name):
    """Body of a kernel (comments removed)."""
    with open(os.path.join(CSRC, "elem_krylov.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    at = src.index("{", re.search(rf"\b{name}\(const DofPassArgs", src).start())
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        end += 1
        if depth == 0:
            return src[at:end]


def test_staged_dof_pass_leaves_together():
    """``done`` may change while blocks of this launch are starting (a block whose bounded wait ran out
    sets it).  Its consumer warps meet at a barrier that counts all of them, so none may leave by a value
    of its own: what a thread read goes into the barrier's vote, and the producer's read leads to bounded
    waits only."""
    body = _kernel("k_epass2_bj")
    split = re.search(r"}\s*else\s*{?[^{]*pass_begins\(\)", body).start()
    producer, consumer = body[body.index("if (producer)"):split], body[split:]
    reads = re.findall(r"[^;{}]*st->done(?!\s*=[^=])[^;{}]*", consumer)
    assert [r.strip() for r in reads] == ["const bool finished = st->done != 0"]
    uses = re.findall(r"[^;{}]*\bfinished\b[^;{}]*", consumer)
    assert [u.strip() for u in uses[1:]] == ["if (consumer_sync_any(!here || finished))", "if (finished) s_done = 1"]
    # nothing between the threads' own reads and the vote leaves the block or the loop
    between = consumer[consumer.index("finished ="):consumer.index("consumer_sync_any")]
    assert not re.search(r"\b(return|break|continue|goto)\b", between)
    waits = re.findall(r"\bmbar_\w*wait\w*|__syncthreads|consumer_sync\w*|mbar_try", producer)
    assert waits and set(waits) == {"mbar_wait_bounded"}


def test_staged_dof_pass_waits_for_its_copies():
    """The consumer warps may leave by a ``done`` that the producer thread did not see.  The thread that
    issued the copies waits for the last of every stage on each way out."""
    body = _kernel("k_epass2_bj")
    producer = body[body.index("if (producer)"):re.search(r"}\s*else\s*{?[^{]*pass_begins\(\)", body).start()]
    tail = producer[producer.rindex("for ("):]
    assert re.match(r"for \(int q = it > kDofStages \? it - kDofStages : 0; q < it; \+\+q\)\s*"
                    r"mbar_wait_bounded\(full \+ q % kDofStages, \(uint32_t\)\(\(q / kDofStages\) & 1\)\);\s*}\s*"
                    r"__syncwarp\(\);\s*$", tail)
    # the loop stands behind every branch and loop of the thread's own block, and nothing returns before it
    before = producer[producer.index("int it = 0;"):producer.rindex("for (")]
    assert before.count("{") == before.count("}") and "return" not in before and "goto" not in before
    # each copy counts once: the stage and phase waited for are those of the issue
    assert len(re.findall(r"\bissue\(tile, it, it == 0\)", before)) == 1
    assert re.search(r"const int s = it % kDofStages;.*issue\(tile, s, false\);", before, re.S)
