"""Non-coherent loads (__ldg) in the kernels that start in programmatic order:
CUDA allows them only on memory that nothing writes while the kernel lives, so
they may name what is in place before the chain of kernels begins (bitstreams,
input planes, quantiser tables), never what one of its kernels writes
(coefficients and their maxima, lists, counts, sizes)."""

import os
import re

import pytest

from rivet_prores_b200.build import CSRC

# The first name in the load's argument, and what it points into.
ALLOWED = {
    "decode.cu": {"w": "bitstream", "next": "bitstream", "src": "bitstream"},
    "encode.cu": {"line": "input plane", "plane": "alpha plane", "inv": "quantiser table", "cq": "quantiser table"},
}


@pytest.mark.parametrize("file", sorted(ALLOWED))
def test_non_coherent_loads_name_memory_the_chain_never_writes(file):
    text = open(os.path.join(CSRC, file)).read()
    loads = re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*([A-Za-z_0-9]+)", text)
    assert len(loads) == text.count("__ldg(") > 0
    assert set(loads) <= set(ALLOWED[file]), set(loads) - set(ALLOWED[file])
