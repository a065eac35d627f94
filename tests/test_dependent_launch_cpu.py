"""Programmatic dependent launch, by reading the kernels: a kernel lets the next one start only after its own
wait.  A kernel that reads something before its wait (the grouped GEMM reads the routing table) can then count on
everything ahead of its direct predecessor, whichever kernel that is."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flydsl_b200", "csrc")


def functions():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in re.split(r"(?=__global__|__device__)", text):
            yield os.path.basename(path), body


def test_every_trigger_comes_after_a_wait():
    seen = 0
    for name, body in functions():
        if re.match(r"__device__ __forceinline__ void pdl_(wait|trigger)\(", body):
            continue  # the statements themselves
        assert "griddepcontrol.launch_dependents" not in body, f"{name}: use pdl_trigger"
        first = body.find("pdl_trigger(")
        if first >= 0:
            seen += 1
            waits = [m.start() for m in re.finditer(r"pdl_wait(<>)?\(|griddepcontrol\.wait;", body)]
            assert waits and waits[0] < first, f"{name}: {body[:120]}"
    assert seen >= 14


def test_the_switch_is_read_in_one_place():
    text = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*")) if p.endswith((".cu", ".cuh", ".h", ".cpp")))
    assert text.count('getenv("FLYB200_PDL")') == 1
