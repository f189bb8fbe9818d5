"""What the assembler reports of the kernels whose time the library's calls are made of."""
import os
import re

import pytest

from anemone_b200 import build


@pytest.mark.parametrize("name", ["kernel_exl3_layer", "kernel_exl3_prefill", "kernel_mx_tensor"])
def test_kernels_of_the_layer_calls_spill_no_register(name):
    path = os.path.join(build.BUILD, name + ".ptxas.txt")
    if not os.path.exists(path):
        pytest.skip("the library was not built in this tree")
    found = re.findall(r"Function properties for (\w+)\n\s*(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads",
                       open(path).read())
    assert found and all(stores == loads == "0" for _, _, stores, loads in found), found
