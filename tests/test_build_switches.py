"""The field and curve headers have one form of each product: the kernels that inline products know no
other, so a build switch that selects one would change some of the sites and not the rest."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyzkp_gb300", "csrc")


def _conditionals(name):
    """Macros that a conditional of the file tests, apart from defaults (#ifndef X / #define X value)."""
    lines = open(os.path.join(CSRC, name)).read().splitlines()
    out = set()
    for i, line in enumerate(lines):
        m = re.match(r"\s*#\s*(ifdef|ifndef|if|elif)\b(.*)", line)
        if not m:
            continue
        names = re.findall(r"ZK_\w+", m.group(2))
        if m.group(1) == "ifndef" and re.match(r"\s*#\s*define\s+%s\s+\S" % names[0] if names else r"$^", lines[i + 1]):
            continue
        out.update(names)
    return out


def test_no_switch_selects_another_arithmetic():
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh")):
        assert _conditionals(name) == set(), name
