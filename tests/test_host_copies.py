"""Copies to and from host memory are asynchronous: no call may return, with whatever status, while one is queued that reads
or writes the caller's memory or its own locals. Read from the sources: such copies are queued by the helpers alone, and
every function that calls one holds a CopiesDone, or what it copies is its callers', who then hold one."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rust-compress_gb300", "csrc")

HELPERS = {"copy_to_device", "read_back", "copy_to_host", "symbol_to_device"}
# Functions whose host memory outlives them, and where it lives.
CALLERS = {
    "search_prepare": "SearchRun",
    "score_batch": "the context's work_list",
    "exact_candidate": "static",
    "settle_ties": "the caller's SearchState",
    "pullback_inputs": "the caller's images",
    "batch_scores_out": "the caller's scores",
}


def _functions():
    """name -> body of every function defined at the start of a line (bodies end at a brace in the first column)."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"^(?:static |inline )?[\w:*& ]+?[ *](\w+)\(([^;{}]*)\)(?: const)? \{\n(.*?)^\}", text,
                             re.M | re.S):
            out[m.group(1)] = m.group(3)
    return out


def _calls(body, names):
    return {n for n in names if re.search(r"\b%s\(" % n, body)}


def test_copies_are_queued_by_the_helpers_alone():
    at = {n: b for n, b in _functions().items() if re.search(r"cudaMemcpy\w*Async\([^;]*(HostToDevice|DeviceToHost)", b)}
    assert set(at) == {"copy_to_device", "read_back"}
    texts = [open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*"))]
    queued = sum(len(re.findall(r"cudaMemcpy\w*Async\([^;]*(?:HostToDevice|DeviceToHost)", t)) for t in texts)
    assert queued == 3  # those two and symbol_to_device


def test_who_copies_waits():
    functions = _functions()
    assert {"rcg_search_metric", "rcg_search_batch_lockstep", "score_batch", "plan_scans", "jpeg_decode",
            "rcg_ssimulacra2_grad", "sweep_group"} <= set(functions)
    bad = []
    for name, body in functions.items():
        if name in HELPERS or not _calls(body, HELPERS | set(CALLERS)):
            continue
        if "CopiesDone done(ctx" not in body and name not in CALLERS:
            bad.append(name)
    assert not bad, bad
    assert "CopiesDone done(ctx, &ctx->lock_subs)" in functions["rcg_search_batch_lockstep"]
