"""Every device-side wait reports a site of its own: an error word names one place in the sources."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zip_kernel_b200", "csrc")


def _sites():
    """(name, id) of every site constant: enums count on from the last given value."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in re.findall(r"enum\s*:\s*int\s*\{([^}]*)\}", text):
            value = -1
            for entry in filter(None, (e.strip() for e in body.split(","))):
                name, _, given = (x.strip() for x in entry.partition("="))
                value = int(given, 0) if given else value + 1
                if name.startswith("SITE_"):
                    out.append((name, value))
        out += [(n, int(v, 0)) for n, v in re.findall(r"constexpr int (SITE_\w+) = (\w+);", text)]
    return out


def test_error_sites_are_distinct():
    sites = _sites()
    assert len(sites) > 20
    by_id = {}
    for name, value in sites:
        by_id.setdefault(value, []).append(name)
    assert not {v: n for v, n in by_id.items() if len(n) > 1}
    assert all(0 < v < 0x80 for v in by_id)
