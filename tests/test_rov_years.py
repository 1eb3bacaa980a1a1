"""The order of the backward pass's launches (csrc/to_rov_years.h), compiled as
plain C++ on the CPU: every year is prepared and selected before its fit,
within the scratch's slots, and a fit starts ahead of its predecessor's end
except where that is the selection whose lists it copies."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CASES = [(Y, slots, sel) for Y in (3, 4, 5, 11, 50) for slots in (1, 2, 3, 48) for sel in (1, 2, 3, 48)
         if sel <= slots]


def test_fit_after_a_selection_is_not_started_ahead(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include "to_rov_years.h"\nint main() {\n' + "".join(
        f'{{ to_rov_years y({Y}, {a}, {b}); while (y.next()) std::printf("%d,%d,%d,%d,%d,%d ", y.t, '
        'y.low, y.prepare, y.sel, y.select, (int)y.fit_ahead()); std::printf("\\n"); }\n'
        for (Y, a, b) in CASES) + "return 0;\n}\n")
    exe = tmp_path / "t"
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I",
                    str(ROOT / "transportoptimiser_gb300" / "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) == len(CASES)
    for (Y, slots, sel_slots), line in zip(CASES, lines):
        prepared, selected, before = set(), set(), None
        years = [tuple(map(int, w.split(","))) for w in line.split()]
        assert [y[0] for y in years] == list(range(Y - 2, 0, -1))
        for t, low, prepare, sel, select, ahead in years:
            launches = []
            if prepare:                    # the slots are written anew
                assert prepare <= slots
                prepared, selected = set(range(low, low + prepare)), set()
                launches.append("prepare")
            if select:
                assert select <= sel_slots
                selected = set(range(sel, sel + select))
                launches.append("select")
            assert selected <= prepared and t in selected, (Y, slots, sel_slots, t)
            before = launches[-1] if launches else "decide"
            assert bool(ahead) == (before == "decide"), (Y, slots, sel_slots, t)
