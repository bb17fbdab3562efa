"""Source rules of the staged launches, which may be resident before the
launch ahead of them has ended (programmatic dependent launch): what a
launch of the same step writes is read after the wait, by loads that the
wait orders."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "openswpc_b200" / "csrc"


def test_scales_are_not_read_by_read_only_loads():
    """The FP16 scales are written by the re-centring kernels between the
    launches of a step: no accessor of theirs is a read-only load."""
    src = (CSRC / "swpc_kernels.cuh").read_text()
    accessors = re.findall(r"float (sc_\w+)\(const float \*s[^{]*\{([^}]*)\}", src)
    assert {n for n, _ in accessors} == {"sc_sS_in", "sc_sR_in", "sc_sS", "sc_iS", "sc_sR", "sc_iR"}
    for name, body in accessors:
        assert "__ldg" not in body and "ld.global.nc" not in body, name
