"""What the kernels' sources promise and no run can show: an order whose violation would hang a GPU is looked for in the text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "riemannengine_b200", "csrc")


def _kernels():
    """(file, kernel name, text from its head to the next kernel) of every __global__ function."""
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            yield name, re.search(r"\b(k_\w+)", text[a:b]).group(1), text[a:b]


@pytest.mark.parametrize("file,kernel,text", [pytest.param(*k, id=k[1]) for k in _kernels() if "tcgen05.alloc" in k[2]])
def test_the_next_kernel_is_released_behind_the_allocation_of_tensor_memory(file, kernel, text):
    """A block of the next kernel that came onto the SM first and took the tensor memory would hold it while it waits for
    this kernel, which waits for the memory."""
    alloc = text.index("tcgen05.alloc")
    barrier = text.index("__syncthreads()", alloc)
    for release in ("after_previous_kernel()", "release_next_kernel()", "griddepcontrol.launch_dependents"):
        for m in re.finditer(re.escape(release), text):
            assert m.start() > barrier, (file, kernel, release)


@pytest.mark.parametrize("file,kernel,text", [pytest.param(*k, id=k[1]) for k in _kernels() if "setmaxnreg" in k[2]])
def test_register_splits_are_executed_by_whole_warpgroups(file, kernel, text):
    """setmaxnreg is one instruction for the four warps of a warpgroup: the branch it opens has to hold for all or none."""
    with open(os.path.join(CSRC, file)) as f:
        constants = dict(re.findall(r"\b(k\w+) = (\d+)\b", f.read()))
    for m in re.finditer("setmaxnreg", text):
        branch = text[text.rindex("if (", 0, m.start()):m.start()]
        limit = re.match(r"if \(warp < (\w+)\) \{", branch)
        assert limit and int(constants[limit.group(1)]) % 4 == 0, (file, kernel, branch)
