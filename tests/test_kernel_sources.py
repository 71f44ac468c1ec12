"""Orders inside the kernels that no run can be asked to break."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "darknet_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_dependents_start_once_a_cta_has_its_tensor_memory(path):
    """A dependent kernel's CTA may take all of an SM's tensor memory and hold it until this kernel ends: a CTA that let it start before
    its own allocation would wait for it for ever.  The allocation is one warp's; a barrier of the CTA lies between it and the trigger."""
    with open(path) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    for kernel in text.split("__global__")[1:]:
        if "tcgen05.alloc" not in kernel or "pdl_trigger()" not in kernel:
            continue
        between = kernel[kernel.index("tcgen05.alloc"):kernel.index("pdl_trigger()")]
        assert kernel.index("tcgen05.alloc") < kernel.index("pdl_trigger()") and "__syncthreads();" in between


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_waits_for_tensor_memory_loads_hold_the_registers(path):
    """A load from tensor memory fills its registers some time after the instruction.  The wait takes them as operands: without, only the
    compiler's order of instructions keeps arithmetic on them behind it (a clobber of memory holds back accesses, not arithmetic)."""
    with open(path) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    for rest in text.split('"tcgen05.wait::ld')[1:]:
        assert re.match(r'[^"]*"\s*:\s*"\+r"', rest), rest[:120]
