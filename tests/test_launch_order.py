"""The host engine's two streams and its chained launches.

A kernel launched with the programmatic dependency waits for the kernel before
it in its own stream. Where the stream has waited for another stream's event,
the next kernel reads that stream's results too, so it has to be launched
plainly: read from the sources, on any machine.

Handles of several threads, each evaluated, run, restarted and run again,
give what each gives alone, bit for bit, in every form of the transforms."""
import os
import re
import threading

import numpy as np
import pytest

from texo_gb300 import abi, problem as P
from texo_gb300.placer import Placer, default_params

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "texo_gb300", "csrc")


def text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def block_end(s, i):
    """Past the block that opens at s[i]."""
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(s[i], 0)
        i += 1
        if depth == 0:
            return i


def next_launch(s, i):
    """The launcher called after s[i] on the same path (an else branch is another path)."""
    while True:
        m = re.compile(r"launch_\w+(?=\()|\}\s*else\s*(?=\{)").search(s, i)
        if not m.group().startswith("}"):
            return m.group()
        i = block_end(s, m.end())


def test_a_kernel_behind_another_streams_event_is_launched_plainly():
    kernels = text("kernels.cu")
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".cpp")):
            continue
        s = text(name)
        for m in re.finditer(r"cudaStreamWaitEvent\(", s):
            launcher = next_launch(s, m.end())
            body = re.search(r"void %s\([^)]*\) \{" % launcher, kernels)
            found.append((name, launcher, kernels[body.end():block_end(kernels, body.end() - 1)]))
    assert len(found) == 2   # the second stream's kernel, and the first one after it is joined
    for name, launcher, body in found:
        assert "<<<" in body and "follow(" not in body, (name, launcher)


def test_a_kernel_behind_a_stream_ordered_allocation_is_launched_plainly():
    """The memory may have been freed by another stream, which the allocation then makes this one wait for."""
    kernels, engine = text("kernels.cu"), text("engine.cu")
    uses = [m.end() for m in re.finditer(r"buf\.get\(", engine)]
    assert len(uses) == 3   # coordinates in, a point out, an evaluation out
    for i in uses:
        launcher = next_launch(engine, i)
        body = re.search(r"void %s\([^)]*\) \{" % launcher, kernels)
        body = kernels[body.end():block_end(kernels, body.end() - 1)]
        assert "<<<" in body and "follow(" not in body, launcher


FORMS = [dict(bins_x=128, bins_y=128), dict(bins_x=96, bins_y=80), dict(bins_x=128, bins_y=128, dct_mode=abi.DCT_TENSOR)]


@pytest.mark.gpu
def test_handles_of_many_threads_restarted_give_what_each_gives_alone():
    problems = [P.synthetic(96, 4000 + 500 * k, 60, 5000, 6.0, k) for k in range(6)]

    def work(k):
        prm = default_params(engine=abi.ENGINE_HOST, best_effort=1, max_iterations=40, **FORMS[k % len(FORMS)])
        out = []
        with Placer(problems[k], prm) as g:
            c, _, _ = g.initial()
            for _ in range(3):
                e = g.evaluate(c, 5.0)
                out += [e["wirelength"], e["potential"], e["wa_gradient"], e["field_gradient"]]
                t, x, _ = g.run(4, allow_nonconverged=True)
                out += [t, x]
                g.reset()
        return out

    alone = [work(k) for k in range(6)]
    got = [None] * 6

    def run(k):
        got[k] = [work(k) for _ in range(3)]

    threads = [threading.Thread(target=run, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(6):
        assert all(np.array_equal(a, b) for a, b in zip(alone[k], alone[k][6:]))   # a restart changes nothing
        for r in got[k]:
            assert all(np.array_equal(a, b) for a, b in zip(alone[k], r))


def test_tables_sent_from_pageable_memory_have_arrived_before_another_stream_reads_them():
    """Each function of the engine that fills a table with cudaMemcpy waits for the legacy stream before it publishes it."""
    s = text("engine.cu")
    for m in re.finditer(r"cudaError_t shared_\w+\([^)]*\) \{", s):
        body = s[m.end():block_end(s, m.end() - 1)]
        if "cudaMemcpy(" in body:
            assert "sent(" in body and body.index("sent(") < body.index("cache.emplace"), m.group()
    assert re.search(r"cudaError_t sent\(.*cudaStreamSynchronize\(cudaStreamLegacy\)", s)
