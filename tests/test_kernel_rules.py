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


# what no kernel of the partition loop writes: the graph, the launch records
CONSTANT = {"a.oidx", "a.iidx", "a.ow", "a.iw", "a.osrc", "d.gsrc", "d.gidx", "d.gptr", "d.gw",
            "oidx", "iidx", "ow", "iw", "sp.cta0", "src"}
# by file: the x log2 x table, general mode's loops over a direction, the edges
# a graph is built from (and the row pointers of a kernel launched in stream order)
LOCAL = {"common.cuh": {"tab"}, "nodal.cu": {"idx", "wt"},
         "ingest.cu": {"a.other", "a.src", "a.dst", "a.w", "ptr"}}


def arguments(text):
    for m in re.finditer(r"__ldg\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        yield text[m.end():end - 1]


@pytest.mark.parametrize("path", [f for f in FILES if "launch_kernel" in open(f).read()
                                  or "multi.cuh" in open(f).read() or f.endswith(".cuh")],
                         ids=os.path.basename)
def test_read_only_loads_of_constant_data(path):
    # a kernel launched by programmatic dependent launch is resident while its
    # predecessors write, so __ldg, which is for data that stays the same over
    # the kernel's lifetime, may not load what the loop's kernels write; nor
    # may a pointer to it be declared __restrict__ (loads then become such)
    text = code(path)
    names = CONSTANT | LOCAL.get(os.path.basename(path), set())
    for arg in arguments(text):
        base = re.match(r"\(\w+(?:\[j\])? \? ([\w.]+)(?: \+ \w+)? : ([\w.]+)(?: \+ \w+)?\)", arg)
        base = base.groups() if base else (re.match(r"[\w.]+", arg).group(0),)
        assert set(base) <= names, arg
    for m in re.finditer(r"(\w+)\s*\*\s*__restrict__\s+(\w+)", text):
        assert m.group(2) in names, m.group(0)
