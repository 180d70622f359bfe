"""The packed passes (csrc/pair_*.cu*) start while the pass ahead of them may still be writing, so they
may read through the read-only path only what no pass writes: their plan's tables.  The source is
checked (no GPU): a stale read would depend on timing and on the compiler."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spim_registration_gb300", "csrc")
TABLES = {"copy_table", "table_root"}


def _code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _functions(code):
    """(name, parameters, body) of every function definition."""
    for m in re.finditer(r"\b(\w+)\(([^;{}]*)\)\s*(?:const\s*)?(?::[^{;]*)?\{", code):
        depth, i = 1, m.end()
        while depth and i < len(code):
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
        yield m.group(1), m.group(2), code[m.end():i]


def test_passes_that_start_early_read_only_tables_through_the_read_only_path():
    files = sorted(glob.glob(os.path.join(CSRC, "pair_*.cu*")))
    assert len(files) >= 5
    seen = set()
    for path in files:
        code = _code(path)
        reads = len(re.findall(r"__ldg\(|\.nc\.", code))
        inside = 0
        for name, params, body in _functions(code):
            if name in TABLES:
                inside += len(re.findall(r"__ldg\(|\.nc\.", body))
                seen.add(name)
            else:  # a const __restrict__ pointer lets the compiler choose that path by itself
                consts = re.findall(r"const\s+(\w+)\s*\*\s*(?:const\s+)?__restrict__", params)
                assert set(consts) <= {"TileDesc"}, (path, name, consts)
        assert reads == inside, path
    assert seen == TABLES
