"""Kernel attributes (dynamic shared memory above 48 KB) and occupancies belong
to a device.  A flag kept per process would skip them on a second device, whose
launches then fail; no such flag may guard them: they go through the
per-context helpers."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kelvin_gb300",
                    "csrc")


def sources():
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.h"))):
        with open(f) as h:
            yield os.path.basename(f), h.read()


def test_attributes_are_set_by_the_context_helper_only():
    uses = {f: len(re.findall(r"\bcudaFuncSetAttribute\s*\(", s)) for f, s in sources()}
    assert {f: n for f, n in uses.items() if n} == {"kvft_ctx.cu": 1}


def test_no_process_wide_launch_state():
    found = [(f, m) for f, s in sources()
             for m in re.findall(r"^\s+static (?:bool|int|long long|size_t) \w+ = .*;", s, re.M)]
    assert found == []
