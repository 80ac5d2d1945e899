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
