"""Rules on the kernels' sources that no run shows: checked on the text."""
import glob
import os
import re

from conftest import PKG


def _sources():
    for path in sorted(glob.glob(os.path.join(PKG, "csrc", "*"))):
        with open(path) as f:
            yield os.path.basename(path), f.read()


def test_no_multicast_loads():
    """The library also runs as one of several replicas on a node (one process per GPU):
    none of its copies is a multicast.  (tcgen05.commit's multicast arrival on the barriers
    of a CTA pair is no copy.)"""
    found = []
    for name, text in _sources():
        # adjacent string literals of an asm statement joined
        joined = re.sub(r'"\s*\n\s*"', "", text)
        found += [(name, m) for m in re.findall(r"cp\.[\w.:]*multicast[\w.:]*", joined)]
    assert found == []
