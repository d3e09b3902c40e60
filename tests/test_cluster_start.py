"""Every kernel whose CTAs reach into a peer's shared memory synchronises its
cluster first: until the barrier, a peer need not have started.  Read from the
sources, with the device functions that a kernel calls taken in."""
import glob
import os
import re

import pytest

from conftest import PKG

REMOTE = ("map_shared_rank", "mbar_arrive_cluster")


def _functions(text):
    """{name: body} of the functions of a source, and the names of kernels."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__(launch_bounds|cluster_dims)__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
    bodies, kernels = {}, set()
    for m in re.finditer(r"(__global__|__device__)([^;{}]*?)\b(\w+)\s*\(([^;{}]*?)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        bodies[m.group(3)] = text[m.end():i]
        if m.group(1) == "__global__":
            kernels.add(m.group(3))
    return bodies, kernels


def _first(name, bodies, seen=()):
    """The first cluster event in textual order: 'sync', 'remote' or None."""
    for m in re.finditer(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\s*\(", bodies[name]):
        word = m.group(1)
        if word == "sync" and bodies[name][: m.start()].endswith("cl."):
            return "sync"
        if word in REMOTE:
            return "remote"
        if word in bodies and word not in seen:
            event = _first(word, bodies, seen + (name,))
            if event:
                return event
    return None


SOURCES = [p for p in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu"))) if "map_shared_rank" in open(p).read()]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_clusters_synchronise_before_they_reach_a_peer(path):
    bodies, kernels = _functions(open(path).read())
    events = {k: _first(k, bodies) for k in kernels}
    assert "remote" not in events.values(), events
    assert "sync" in events.values()  # the kernel that uses the peers was found
