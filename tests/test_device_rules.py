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


def _bodies(name):
    """(head, body) of each function: the text before its braces, and what they hold."""
    s = _code(name)
    for m in re.finditer(r"\)\s*\{", s):
        start = s.rfind("\n\n", 0, m.start()) + 1
        depth, i = 1, m.end()
        while depth and i < len(s):
            depth += {"{": 1, "}": -1}.get(s[i], 0)
            i += 1
        yield s[start:m.start()], s[m.end():i - 1]


@pytest.mark.parametrize("name", HEADERS)
def test_tap_tables_are_read_within_their_cycles(name):
    """The tables hold n_cycles + 1 cycles; a job that ended by its count stands at
    cycle n_cycles + 1.  A pass reads them after its stop test (or walks live jobs
    only), or at a cycle held to the last one."""
    found = 0
    for head, body in _bodies(name):
        if "__device__" not in head and "__global__" not in head:
            continue
        at = body.find("J.ntaps[")
        if at < 0:
            continue
        found += 1
        assert re.search(r"if \((st->)?stop\)|next_live|c = min\(st->cycle, J\.n_cycles\)", body[:at]), head
    assert found or name not in ("kernels.cuh", "kernels_mx.cuh")


@pytest.mark.parametrize("name", HEADERS)
def test_no_block_leaves_with_copies_in_flight(name):
    """After a kernel has requested asynchronous copies into shared memory, a
    return or a skipped item comes after a wait for them."""
    request = re.compile(r"cp_async[48]\(|col_bs16_load<|mx_col_request<")
    for head, body in _bodies(name):
        if "__global__" not in head:
            continue
        m = request.search(body)
        if not m:
            continue
        rest = body[m.end():]
        leave = re.search(r"\b(return|continue)\b", rest)
        if leave:
            assert "cp_async_wait()" in rest[:leave.start()], head


def test_pipelined_passes_trigger_by_their_length():
    """The pipelined passes let the next pass start early only at lengths that gain."""
    triggers = {}
    for head, body in _bodies("kernels.cuh"):
        name = re.search(r"\b(k_row_hio_p|k_row_finish_p|k_col_p|k_col_p16)\(const JobDev", head)
        if name and "__global__" in head and name.group(1) not in triggers:
            triggers[name.group(1)] = re.findall(r"if \(([^;]*)\) pdl_trigger\(\)", body)
    assert set(triggers) == {"k_row_hio_p", "k_row_finish_p", "k_col_p", "k_col_p16"}
    for name, conds in triggers.items():
        assert conds and all(c.startswith("pdl_length(N) && ") for c in conds), name


def test_pipelined_passes_of_a_batch_request_their_first_tile_first():
    """Where an item has to be read to know the job (a batch's lists), the tables come
    after the first live tile has been found."""
    seen = {}
    for head, body in _bodies("kernels.cuh"):
        name = re.search(r"\b(k_row_hio_p|k_row_finish_p|k_col_p|k_col_p16)\(const JobDev", head)
        if name and "__global__" in head and name.group(1) not in seen:
            seen[name.group(1)] = re.search(r"const bool early = (pdl_length\(N\) && )?!walk\.items;", body)
    assert len(seen) == 4 and all(seen.values()), seen
