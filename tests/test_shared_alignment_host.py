"""Shared-memory arrays that the kernels read or write in 16-byte pieces are declared on 16-byte boundaries: an array of floats by
itself is only promised four."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), '..', 'native_sparse_attention_pytorch_b200', 'csrc')


def names(line):
    """The arrays that a declaration of shared memory declares."""
    return re.findall(r'(\w+)(?:\[[^\]]*\])+', line.split('__shared__', 1)[1].split(';')[0])


@pytest.mark.parametrize('source', sorted(f for f in os.listdir(CSRC) if f.endswith(('.cu', '.cuh'))))
def test_pieces_of_sixteen_bytes(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    wide = set(re.findall(r'reinterpret_cast<(?:const )?(?:float4|uint4|int4)\s*\*>\(&?(\w+)', text))
    loose = [(name, line.strip()) for line in text.splitlines() if '__shared__' in line and 'align' not in line.split(';')[0]
             for name in names(line) if name in wide]
    assert not loose
