"""The step kernels may be launched while the kernel before them still writes
(programmatic dependent launch), so their read-only loads (__ldg, pull) may only
name arrays that no step writes; the state and the corner forces are read with
ordinary loads.  Checked on the kernels' source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "v.1.1_gb300", "csrc")
# written by the set-up or the host before a block's first step, by no step kernel
STATIC = {"conn", "slot", "node_ptr", "node_bc", "minv", "minv2", "Lref32", "wJ", "G", "wJ32", "wJ32lo", "G32", "G32lo",
          "fxE", "fxS", "fxD", "fxw"}


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def arguments(text, name):
    """The argument texts of every call of `name` (not of its own definition)."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        arg = text[m.end():k - 1]
        if not arg.startswith("const T *"):
            yield arg


def body(text, head):
    """The source from `head` to the end of the function it begins."""
    at = text.index(head)
    return text[at:text.index("\n}", at)]


@pytest.mark.parametrize("load", ["__ldg", "pull"])
def test_read_only_loads_name_static_arrays(load):
    text = source("msx_device.cuh")
    wrapper = body(text, "__device__ __forceinline__ T ld_step(const T *x)")
    args = list(arguments(text.replace(wrapper, ""), load))
    assert len(args) >= 8
    for a in args:
        names = re.findall(r"\bp\.(\w+)", a)
        assert names and names[0] in STATIC, a


def test_step_data_take_the_read_only_path_only_without_dependent_launch():
    """ld_step<DEP> uses __ldg when DEP is false: the node kernels of blocks that are all resident (BATCH, the only ones
    launched dependently) and the element gathers of a dependent launch (Problem::dependent) have it true."""
    text = source("msx_device.cuh")
    assert "return DEP ? *x : __ldg(x);" in body(text, "__device__ __forceinline__ T ld_step(const T *x)")
    flags = re.findall(r"\bld_step<(\w+)>\(", text)
    assert flags.count("BATCH") + flags.count("DEP") == len(flags) >= 6
    assert "BATCH" not in re.findall(r"\bld_step<(\w+)>\(", body(text, "void gather_u4("))
    gather = body(text, "void gather_u(")
    assert "p.u4 && !p.dependent) {\n        gather_u4<false>" in gather and gather.count("gather_u4<false>") == 1
    assert text.count("gather_u4<false>") == 1
    launch = body(source("msx_fast.cu"), "static void launch_solve(")
    assert "P.dependent = c.numAttrs = n <= q.pdl ? 1 : 0;" in launch
    assert re.search(r"cudaLaunchKernelEx\(&c, f, P,", launch)
