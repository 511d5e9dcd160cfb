"""A CTA's shared memory may be addressed by the other CTAs of its cluster only once that CTA is known to run, so
every kernel that stores or loads through shared::cluster addresses has to pass a cluster barrier first. A run on
the GPU rarely shows a missing one; the order is read off the sources instead."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REMOTE = re.compile(r"\bmapa[.a-z:0-9]*|\b(?:st|ld|red|atom)[.a-z0-9]*\.shared::cluster")


def kernels():
    """(file, name, body) of every __global__ function, comments taken out."""
    for path in sorted(glob.glob(os.path.join(ROOT, "colibri_b200", "csrc", "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            name = re.search(r"\b(k_\w+)\s*\(", text[a:b])
            yield os.path.basename(path), name.group(1) if name else "?", text[a:b]


def test_cluster_barrier_before_remote_shared_memory():
    seen = []
    for path, name, body in kernels():
        first = REMOTE.search(body)
        if not first:
            continue
        seen.append(name)
        before = body[:first.start()]
        arrive, wait = before.find("barrier.cluster.arrive"), before.find("barrier.cluster.wait")
        assert 0 <= arrive < wait, f"{path} {name}: no cluster barrier before {first.group(0)}"
        # ... and one behind the last access, before a CTA whose memory was addressed may leave
        last = [m.end() for m in REMOTE.finditer(body)][-1]
        assert "barrier.cluster.wait" in body[last:], f"{path} {name}: no cluster barrier behind the last access"
    assert "k_argmax_rows" in seen
