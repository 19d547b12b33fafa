"""Rules of the device code that a run cannot show, read from the sources.

Passes of a plan may start while the pass before them still runs (tma.cuh):
what a pass writes is read with ordinary loads, after pdl_wait.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imresh_b200", "csrc")
HEADERS = sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh"))


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


# twiddle and chirp-z tables, written before any pass is launched, and the
# modulus (and its tiles), complete before the graph of the passes starts
READ_ONLY = {"tw", "gtw", "chirp", "p.chirp", "spec", "mt", "mt_base", "J.M"}


@pytest.mark.parametrize("name", HEADERS)
def test_non_coherent_loads_only_of_what_no_pass_writes(name):
    args = re.findall(r"__ldg\(\s*([^)]*)", _code(name))
    assert [a for a in args if re.split(r"[\s+]", a)[0] not in READ_ONLY] == []
