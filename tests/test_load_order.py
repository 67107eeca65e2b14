"""The load-ordering rule of the kernels launched with programmatic stream
serialisation, checked on their sources: such a kernel may start while the
previous one still runs, so what kernels write may be read only behind
griddepcontrol.wait.  Loads that the compiler may move (load4_nc, load4_x,
ldg_any, __ldg, and the face loads built on them) therefore take pointers to
kernel-written buffers from after_wait(), never straight from the launch
arguments; volatile loads (gload4, load4_now) keep their place by themselves."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zhijian_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# launch-argument members that point to what a kernel writes
WRITTEN = "U|U0|dU|Uout|Tin|Tout|FV|FVout|GQ|R|dR|L|W|T|TQ|Db|Tb|DUb|X0|X1|X2|partials"
MOVABLE = r"(?:load4_nc|load4_x|ldg_any|__ldg)"


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", FILES)
def test_movable_loads_take_no_raw_pointer_to_written_data(name):
    text = code(name)
    raw = re.findall(MOVABLE + r"\s*\(\s*a\.(?:%s)\b[^;]*;" % WRITTEN, text)
    assert raw == [], raw
    # the face loads of a stage get the pointer behind the wait
    for arg in re.findall(r"load_(?:own|neighbour)_face<N1>\(a, ([^,]+),", text):
        assert arg == "Tin"
    for dst, src in re.findall(r"const \w+\* (\w+) = (a\.(?:%s));" % WRITTEN, text):
        raise AssertionError(f"{dst} = {src} without after_wait")


@pytest.mark.parametrize("name", FILES)
def test_after_wait_follows_the_wait(name):
    """Between a kernel's wait and any after_wait() of it no other kernel
    begins, and none precedes its wait."""
    text = code(name)
    for body in re.split(r"__global__", text)[1:]:
        at = body.find("after_wait(a.")
        if at >= 0:
            assert 0 <= body.find("pdl_wait();") < at
