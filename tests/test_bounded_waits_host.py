"""Every wait inside a kernel is bounded, and one that runs out leaves a flag.
No test makes a kernel's wait run out on the GPU; these read the sources for
what has to hold when one does."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "rust-nmf_b200" / "csrc"

# What puts kernels with bounded waits on a stream, and how their flag is read.
QUEUES = re.compile(r"\b(enqueue_iteration|enqueue_objective|enqueue_objective_partials|h_step|"
                    r"w_step|run_graphed|launch_trees|L\.iteration|L\.objective)\b")
READS = re.compile(r"\bfinish_checked\(|\btimeout\b|\bgave_up\b")


def _top_level(text):
    """The file's top-level definitions (each begins and ends in column 0)."""
    block = []
    for line in text.splitlines():
        block.append(line)
        if line in ("}", "};"):
            yield "\n".join(block)
            block = []


def _waiting_functions():
    for path in sorted(CSRC.glob("*.cu")):
        for body in _top_level(path.read_text()):
            if QUEUES.search(body) and "cudaStreamSynchronize(" in body:
                yield path.name, body
            elif QUEUES.search(body) and "finish_checked(" in body:
                yield path.name, body


def test_a_result_is_read_with_its_time_out_flag():
    """A function that queues such kernels and waits for their results reads
    the flag: a sum that lacks a block's part is not returned as a result."""
    seen = []
    for name, body in _waiting_functions():
        head = re.search(r"(\w+)\([^;{]*\{", body)
        seen.append(head.group(1) if head else "?")
        assert READS.search(body), f"{name}: {seen[-1]}"
    assert {"run_loop", "single_step", "objective_host", "run_snmf"} <= set(seen), seen


def _kernel(path, name):
    """The body of a kernel, without its comments."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    start = text.index("{", text.index(")", text.index(name + "(")))
    return text[start:text.index("\n}\n", start)]


def _braced(text, start):
    """text[start:] from its first brace to the one that closes it."""
    at = text.index("{", start)
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1], i + 1
    raise AssertionError("unbalanced braces")


def test_tree_leaves_by_one_barrier():
    """A thread of a tree's cluster whose wait ran out leaves the steps at any
    of them.  Every thread passes the same hardware barriers all the same:
    those before the steps and the one after them, none in between and no way
    round.  Its block then stays while what was sent to it may be on its way."""
    body = _kernel(CSRC / "linkage.cu", "nn_chain_average")
    barrier = re.compile(r"\bcl\.sync\(|\b__syncthreads\(|\bbarrier\.cluster|\bbar\.sync")
    before = body[:body.index("while (k < p - 1)")]
    steps, end = _braced(body, body.index("while (k < p - 1)"))
    after = body[end:]
    assert not barrier.search(steps)
    assert not re.search(r"\breturn\b", steps)
    # what the steps call holds none either
    for name in re.findall(r"const auto (\w+) = \[&\]", before):
        helper, _ = _braced(before, before.index(f"const auto {name} ="))
        assert not barrier.search(helper), name
    assert len(barrier.findall(after)) == 1
    assert not re.search(r"\breturn\b", after[:after.index("cl.sync(")])
    # each wait of the steps that runs out is noted, and awaited once more
    for m in re.finditer(r"if \(!(bar_wait|meet)\(", steps):
        given_up, _ = _braced(steps, m.start())
        assert "late = true;" in given_up and "break;" in given_up
    assert "bar_wait(" in after[after.index("cl.sync("):]
    assert "atomicExch(gave_up" in after


def test_tree_warp_gives_up_as_one():
    """The lanes of a warp leave a wait with one answer: one that went on alone
    would reduce over lanes that have left the steps."""
    body = _kernel(CSRC / "linkage.cu", "bool bar_wait")
    assert re.findall(r"(if \([^\n]*\) )?return (\w+);", body) == [
        ("if (__all_sync(0xffffffffu, ok)) ", "true"), ("", "false")]
