"""Asynchronous copies into shared memory are ordered against plain accesses.

An inline-assembly statement without a "memory" clobber is no barrier to the
compiler: a load of the bytes an asynchronous copy replaces could move below the
copy, one of the bytes it brings above the wait.  Whether that happens is up to one
compiler's scheduling, so the statements themselves are looked at.
"""
import re

from conftest import ROOT

ASM = re.compile(r"\basm\s+volatile\s*\((.*?)\)\s*;", re.S)


def test_cp_async_statements_are_compiler_barriers():
    found = 0
    for path in sorted((ROOT / "modisp_b200" / "csrc").glob("*.cu*")):
        text = path.read_text()
        statements = [m.group(1) for m in ASM.finditer(text) if '"cp.async' in m.group(1)]
        assert text.count('"cp.async') == len(statements), path.name
        for s in statements:
            assert s.rstrip().endswith('"memory"'), f"{path.name}: {s}"
        found += len(statements)
    assert found
