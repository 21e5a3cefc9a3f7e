"""The rule of csrc/tc05.cuh on kernels that may start before the launch before them has ended, checked in their sources: they wait
for it before they read anything, and read by loads that the wait orders."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "causal_trainer_dev_b200" / "ops" / "csrc"


def _without_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _kernels():
    """name -> (parameters, body) of every kernel."""
    found = {}
    for path in sorted(CSRC.glob("*.cu")):
        text = _without_comments(path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?(\w+)\s*\(([^{;]*?)\)\s*\{", text):
            end = text.index("\n}\n", m.end())
            found[path.name, m.group(1)] = (m.group(2), text[m.end():end])
    return found


def _launched_chained():
    """(file, kernel) of the kernels that a launch_chained call names, by itself or through a variable that it is given by."""
    names = set()
    for path in sorted(CSRC.glob("*.cu")):
        text = _without_comments(path.read_text())
        for m in re.finditer(r"launch_chained\(", text):
            call = text[m.start():text.index(";", m.start())]
            words = set(re.findall(r"\w+", call))
            for variable in words & {"kern", "reduce"}:
                value = list(re.finditer(r"auto %s = ([^;]*);" % variable, text[:m.start()]))[-1].group(1)
                words |= set(re.findall(r"\w+", value))
            here = {w for w in words if (path.name, w) in KERNELS}
            assert here, call
            names |= {(path.name, w) for w in here}
    return names


KERNELS = _kernels()
CHAINED = sorted(_launched_chained())


def test_the_sources_are_read_as_meant():
    assert len(KERNELS) > 40 and len(CHAINED) >= 20
    # whoever waits is launched so, and the other way round
    assert {k for k, (_, body) in KERNELS.items() if "wait_for_predecessor();" in body} == set(CHAINED)


@pytest.mark.parametrize("kernel", CHAINED, ids=lambda k: k[1])
def test_a_chained_kernel_reads_behind_its_wait(kernel):
    parameters, body = KERNELS[kernel]
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", parameters), "read-only loads of what a predecessor may write"
    # (attention reads routing lists of grouped and sparse calls through helpers; those calls are not chained)
    assert not re.search(r"__ld(g|cs|cg|ca|lu|cv)\s*\(", body)
    ahead = body[:body.index("wait_for_predecessor();")]
    if kernel[0] in ("elementwise.cu", "tp_collectives.cu"):
        assert "[" not in ahead and "*" not in ahead          # nothing at all comes first
