"""The host's tables of what the native sources export and report, against the sources."""
import re

from batchspec_b200.csrc.build import CSRC
from batchspec_b200.kernels import ops

SOURCES = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu"))}


def test_every_report_and_trace_of_the_sources_is_asked_for():
    found = {kind: sorted(n for text in SOURCES.values() for n in re.findall(kind + r"\((\w+)\)", text))
             for kind in ("BSPEC_DEFINE_BOUNDS_REPORT", "BSPEC_DEFINE_TRACE_SETTER")}
    assert found["BSPEC_DEFINE_BOUNDS_REPORT"] == sorted(ops._BOUNDS_REPORTS)
    assert found["BSPEC_DEFINE_TRACE_SETTER"] == sorted(ops._TRACE_SETTERS)


def test_every_code_of_the_sources_has_a_meaning():
    waits = {(name, int(code)) for name, text in SOURCES.items() for code in re.findall(r"status, (\d+)\)", text)}
    assert len(waits) > 20
    assert [w for w in sorted(waits) if ops.wait_meaning(w[1]) == "unknown"] == []
    bounds = {int(code) for text in SOURCES.values() for code in re.findall(r"in_range\(.*?, (\d+)\)", text)}
    assert bounds and bounds <= set(ops.BOUNDS_CODES)
