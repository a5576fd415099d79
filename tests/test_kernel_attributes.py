"""A kernel's shared-memory limit belongs to the device that is current when it
is set, and the library serves every device of a process: no limit may be set
behind a flag that holds for the whole process."""
import re

from conftest import ROOT


def test_limits_are_not_set_once_per_process():
    bad = []
    for p in sorted((ROOT / "manifoldann_gb300" / "csrc").glob("*.cu*")):
        txt = re.sub(r"//[^\n]*", "", p.read_text())
        for m in re.finditer(r"call_once\s*\(", txt):
            depth, e = 1, m.end()
            while depth:  # to the end of the call
                depth += {"(": 1, ")": -1}.get(txt[e], 0)
                e += 1
            if "cudaFuncSetAttribute" in txt[m.start():e]:
                bad.append(f"{p.name}: {txt.count(chr(10), 0, m.start()) + 1}")
    assert not bad, bad
