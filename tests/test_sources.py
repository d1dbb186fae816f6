"""Properties of the CUDA sources that no run can show."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'napmo_b200',
                    'csrc')


@pytest.mark.parametrize('name', ['poisson.cu', 'quad.cu', 'tc.cu'])
def test_dynamic_shared_memory_declares_its_alignment(name):
    """These files read dynamic shared memory in 16-byte words behind static
    shared variables of other sizes; without a declared alignment its base is
    only as aligned as the element type."""
    with open(os.path.join(CSRC, name)) as f:
        arrays = re.findall(r'extern\s+__shared__[^;]*;', f.read())
    assert arrays
    for a in arrays:
        m = re.search(r'__align__\((\d+)\)', a)
        assert m and int(m.group(1)) % 16 == 0, a
