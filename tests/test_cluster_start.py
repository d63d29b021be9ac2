"""Distributed shared memory may only be touched once every CTA of the cluster
has started, which a cluster barrier guarantees.  Each kernel's text is walked
in program order, device functions entered where they are called: a barrier
comes before the first access to a peer's shared memory."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "atsc3_b200", "csrc")
BARRIER = {"cluster_sync_all", "cluster_wait"}
REMOTE = re.compile(r"dsmem_(ld|st|red)\w*$")


def functions(text):
    """name -> (is a kernel, body) of the CUDA functions of a source."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", " ", text, flags=re.S)
    out = {}
    for m in re.finditer(r"__(global|device)__\b", text):
        head = re.compile(r"[;{]").search(text, m.end())
        if head is None or head.group() == ";":
            continue
        name = [c.group(1) for c in re.finditer(r"(\w+)\s*\(", text[m.end():head.start()])
                if c.group(1) not in ("__launch_bounds__", "demap_ctas", "__align__")]
        if not name:
            continue
        depth, i = 1, head.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[name[0]] = (m.group(1) == "global", text[head.end():i])
    return out


def events(fns, body, seen=()):
    for m in re.finditer(r"(\w+)\s*(?:<[^;(){}]*>)?\s*\(", body):
        name = m.group(1)
        if name in BARRIER:
            yield "barrier"
        elif REMOTE.match(name):
            yield "remote"
        elif name in fns and name not in seen:
            yield from events(fns, fns[name][1], seen + (name,))


@pytest.mark.parametrize("source", ["bch.cu", "cpe.cu", "ldpc_flood.cu",
                                    "ldpc_qc.cu", "ldpc_qce.cu"])
def test_barrier_before_peer_access(source):
    with open(os.path.join(CSRC, source)) as f:
        fns = functions(f.read())
    kernels = [k for k, (is_kernel, _) in fns.items() if is_kernel]
    touching = 0
    for k in kernels:
        ev = list(events(fns, fns[k][1], (k,)))
        if "remote" in ev:
            touching += 1
            assert ev[0] == "barrier", k
    assert touching
