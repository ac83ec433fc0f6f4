"""The device waits' limits, by their source: a wait that runs out cannot be provoked without hanging a kernel."""

import re

from conftest import ROOT

CSRC = ROOT / "costal_gb300" / "csrc"


def _sources():
    return {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def test_every_wait_counts_its_own_polls():
    """A poll counter is set to zero directly before the loop that it bounds. One that lived through a CTA's
    whole walk added up the polls of thousands of waits, and a long healthy walk could reach the limit."""
    calls = 0
    for name, text in _sources().items():
        for call in re.finditer(r"wait_budget\(\w+, (\w+)\)", text):
            start = text.rfind(f"long long {call[1]} = 0;", 0, call.start())
            assert start >= 0, name
            between = text[start:call.start()]
            assert len(re.findall(r"\bwhile \(", between)) == 1 and "for (" not in between, (name, between)
            calls += 1
    assert calls >= 2


def test_a_role_that_gives_up_waits_for_its_own_work():
    """Every kernel that starts bulk copies or MMAs waits for those in flight before a role that has given up
    lets the CTA end: they read and write its shared memory."""
    kernels = 0
    for name, text in _sources().items():
        for body in text.split("__global__")[1:]:
            body = body[:body.find("\n}\n")]
            if "tma_load_2d(" in body:
                kernels += 1
                assert "drain_ring(" in body, name
            if "mma_commit(" in body:
                assert "mbar_drain(&bars->drain" in body, name
    assert kernels == 3
