"""CPU: rules of the kernel sources that a run on this chip would not show to be broken."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flint_b200", "csrc")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_waits_for_stores_of_a_neighbour_cta_acquire_at_cluster_scope(path):
    """A barrier that asynchronous stores of other CTAs complete (`xbar` in the kernels that send such stores) orders the waiter behind their data
    only if the wait acquires at cluster scope: the form with template argument true, whose default is the scope of the CTA."""
    code = _code(path)
    waits = re.findall(r"mbar_(?:wait|try)\w*(<\w+>)?\(\s*xbar\b", code)
    assert all(w == "<true>" for w in waits)
    assert bool(waits) == ("xbar" in code)
    if "mbar_try(uint64_t*" in code:
        assert re.search(r"if \(REMOTE\)\s*asm volatile\(\s*\"[^\"]*mbarrier\.try_wait\.parity\.acquire\.cluster\.", code)
