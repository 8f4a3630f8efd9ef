"""CPU: the device code leaves division, reciprocals, roots and elementary functions to the compiler's own
(correctly rounded or documented) operations: no approximate PTX instruction to build them from."""
import re
from pathlib import Path

SOURCES = Path(__file__).resolve().parents[1] / "hsolve_b200" / "csrc"


def test_no_approximate_instructions():
    approx = re.compile(r"\b(rcp|div|sqrt|rsqrt|ex2|lg2|sin|cos|tanh)\.(approx|full)|__frcp|__fdividef|__expf|rcp64h")
    files = sorted(p for p in SOURCES.iterdir() if p.suffix in (".cu", ".cuh"))
    assert files
    found = [f"{p.name}:{n}: {line.strip()}" for p in files for n, line in enumerate(p.read_text().splitlines(), 1)
             if approx.search(line)]
    assert not found, found
