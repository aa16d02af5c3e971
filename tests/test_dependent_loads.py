"""Kernels that start as programmatic dependents read nothing through ld.global.nc,
which asks for data that are read-only for the kernel's lifetime: that begins while
the predecessor still writes them, and no wait orders such a load."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lattibol_0.3.31f_gb300", "csrc")
NC = r"__ldg\s*\(|ld\.global\.nc"
WAIT = r"after_predecessor\s*\(\s*\)|griddepcontrol\.wait"


def functions(csrc):
    """(name, text) of every device function and kernel of the sources"""
    for path in sorted(glob.glob(os.path.join(csrc, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__(?:global|device)__[^;{]*?(\w+)\s*\((?:[^(){};]|\([^()]*\))*\)"
                             r"\s*(?:const\s*)?\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield m.group(1), text[m.start():i]


def offenders(csrc):
    fns = list(functions(csrc))
    # functions that read through ld.global.nc whatever their caller is
    nc = {n for n, t in fns if re.search(NC, t) and not re.search(r"\bDEP\s*\?", t)}
    dependents = [(n, t) for n, t in fns if "__global__" in t and re.search(WAIT, t)]
    assert len(dependents) >= 12, [n for n, _ in dependents]
    bad = []
    for name, text in dependents:
        used = [f for f in nc - {name} if re.search(r"\b%s\s*(<[^;(]*>)?\s*\(" % f, text)]
        if re.search(NC, text) or used or re.search(r"ld_stream<false|pull_native<S>\s*\(", text):
            bad.append(name)
    return bad


def test_no_read_only_loads():
    assert offenders(CSRC) == []
