"""Rules of the programming model that no result shows when they are broken,
read off the kernels' source."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gsap_b200",
                    "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
BARRIER = r"(?:\bcl|this_cluster\(\))\.sync\(\)"


def code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def before(text, pos):
    """The part of the device function around `pos` that comes before it."""
    starts = [m.start() for m in re.finditer(r"\b__device__\b", text[:pos])]
    return text[starts[-1]:pos]


@pytest.mark.parametrize("path", [f for f in FILES if "map_shared_rank" in open(f).read()],
                         ids=os.path.basename)
def test_cluster_barrier_before_remote_shared_memory(path):
    # another CTA's shared memory may be accessed only once all CTAs of the
    # cluster are known to have started
    text = code(path)
    for m in re.finditer("map_shared_rank", text):
        head = before(text, m.start())
        if re.search(BARRIER, head):
            continue
        name = re.search(r"(\w+)\s*\(", head).group(1)
        calls = [c.start() for c in re.finditer(rf"\b{name}(?:<[^;()]*>)?\(", text)
                 if c.start() not in range(m.start() - len(head), m.start())]
        assert calls and all(re.search(BARRIER, before(text, c)) for c in calls), name
