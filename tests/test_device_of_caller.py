"""A call works on its encoder's device, whichever device the calling thread has current (csrc/runtime.cu): what looks at the current device,
or sets a kernel up on it, comes after the call has made the encoder's device current.  (One more GPU would be needed to see it run.)"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_native_b200", "csrc")
# planners that count the device's SMs or clusters, and what makes the encoder's device current
PLANNERS = r"\b(qmm_duo_cost|qmm_tc_pick_nt|qmm_duo_pick_nt|sm_count_of_device|duo_pairs)\("
SETS = r"\b(cudaSetDevice|op_begin|encoder_begin_work)\("


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def functions(src):
    """(name, body) of the functions that start at the left margin."""
    for m in re.finditer(r"^(?:extern \"C\" |static )?[\w:<> *]+?\b(\w+)\([^;{]*\) \{$", src, re.M):
        end = src.index("\n}", m.end())
        yield m.group(1), src[m.end():end]


def test_device_is_set_before_it_is_asked():
    seen = []
    for name, body in functions(read("runtime.cu")):
        planner = re.search(PLANNERS, body)
        if planner:
            seen.append(name)
            sets = re.search(SETS, body)
            assert sets and sets.start() < planner.start(), name
    assert {"dispatch_mm", "encoder_flush_pending", "mlxn_quantized_matmul_mm_tensor_perm021"} <= set(seen)


def test_what_is_asked_before_depends_on_the_call_alone():
    body = dict(functions(read("qmm_duo.cu")))["qmm_duo_takes"]
    assert not re.search(r"cuda|duo_plan|" + PLANNERS, body)
