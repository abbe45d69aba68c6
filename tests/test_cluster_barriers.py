"""Distributed shared memory: a block may touch another block's shared memory only
once every block of the cluster has started, and end only after the others are
done with its own.  So each function that maps another block's shared memory has
a cluster barrier before the first use and after the last one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcls_b200", "csrc")


def functions(text):
    """(name, body) of the functions at namespace level."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"^[^\n#]*?(\w+)\(([^;{}]*?)\)\s*\{$", text, re.M):
        depth, k = 1, m.end()
        while depth and k < len(text):
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), text[m.end():k]


def remote_users():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        seen = set()
        for name, body in functions(open(path).read()):
            if "map_shared_rank(" in body and name not in seen:
                seen.add(name)
                yield pytest.param(body, id=f"{os.path.basename(path)}:{name}")


@pytest.mark.parametrize("body", list(remote_users()))
def test_remote_shared_memory_is_between_barriers(body):
    barrier = re.compile(r"\.sync\(\)|barrier_wait\(\)")
    first, last = body.index("map_shared_rank("), body.rindex("map_shared_rank(")
    assert barrier.search(body, 0, first), "no cluster barrier before the first remote access"
    assert barrier.search(body, last), "no cluster barrier after the last remote access"


def test_the_kernels_are_found():
    assert len(list(remote_users())) >= 2
