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

