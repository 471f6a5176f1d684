"""tcgen05.ld returns before its registers are valid.  A bare tcgen05.wait::ld orders memory, not registers, so the compiler may
schedule what uses a loaded value above it; the wait has to name the registers.  Read from the sources."""
import re

from test_dependency_wait import SOURCES, code_of


def test_every_wait_names_the_loaded_registers():
    calls = [(p.name, args.strip()) for p in SOURCES if p.suffix == ".cu"
             for args in re.findall(r"\btc_wait_ld\(([^)]*)\)", code_of(p))]
    assert len(calls) >= 3
    assert all(args for _, args in calls), calls
    common = code_of(next(p for p in SOURCES if p.name == "common.cuh"))
    assert not re.search(r"\btc_wait_ld\(\s*\)", common)
