"""What a kernel that starts while the one before it still runs has to keep to, read from the sources: a fault here shows
on a GPU as a hang or as stale data, and only behind a kernel that lets its dependents in early."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kermac_b200", "csrc")


def _kernels():
    """(name, parameters, body) of the kernels in the files that launch or define overlapped kernels."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for head in re.finditer(r"__global__\s+void(?:\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s+(\w+)\s*\(([^)]*)\)\s*\{", text):
            depth, end = 1, head.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            found.append((os.path.basename(path), head.group(1), head.group(2), text[head.end():end]))
    return [k[1:] for k in found if k[0] != "km_peaks.cu" and k[1] != "wait_expiry_selftest_kernel"]   # launched by <<<>>>


KERNELS = _kernels()


def test_the_kernels_are_found():
    assert {k[0] for k in KERNELS} == {"build_cpasync_kernel", "build_tma_kernel", "build_small_kernel", "pack_kernel", "grad_kernel",
                                       "grad_reduce_kernel", "grad_tensor_kernel", "grad_sign_kernel", "matvec_kernel",
                                       "matvec_tensor_kernel", "matvec_reduce_kernel"}


@pytest.mark.parametrize("name, parameters, body", KERNELS, ids=[k[0] for k in KERNELS])
def test_order_against_the_previous_grid(name, parameters, body):
    before, wait, _ = body.partition("after_previous_grid();")
    assert wait and "return;" not in before           # every block passes the wait
    # tensor memory is taken when the kernel before has given its own back
    assert "tmem_alloc" not in before


@pytest.mark.parametrize("name, parameters, body", KERNELS, ids=[k[0] for k in KERNELS])
def test_nothing_is_promised_to_stay_unwritten(name, parameters, body):
    # the kernel before may still be writing what this one reads: loads must not move in front of the wait
    assert "__restrict__" not in parameters + body and "__ldg" not in body
