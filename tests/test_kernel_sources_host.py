"""What a compiler may reorder in the kernels, read from their sources: no GPU needed."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlsys-contest-syfi-agent-assisted_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_waits_for_tensor_memory_loads_name_the_loaded_registers(path):
    """Arithmetic on the registers of a tcgen05.ld is no volatile statement: only a wait that has them as operands stays in
    front of it whatever the compiler does."""
    text = open(path).read()
    for statement in re.findall(r"asm volatile\((.*?)\);\n", text, flags=re.S):
        if "tcgen05.wait::ld" in statement:
            assert '"+r"' in statement, statement
    pending = set()
    for load, args in re.findall(r"\b(tmem_ld8|tmem_ld16|tmem_ld_wait\w*)\(([^;{]*)\);", text):
        if load.startswith("tmem_ld_wait"):
            named = {a.strip() for a in args.split(",")}
            assert not pending or pending == named, (pending, args)
            pending = set()
        else:
            pending.add(args.split(",")[-1].strip())
    assert not pending
