"""Rules of programmatic launches (``csrc/chained_launch.h``), read from the sources: breaking one is a race, which no run shows
reliably."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'asdl_b200', 'csrc')


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r'//[^\n]*', '', fh.read())


@pytest.mark.parametrize('flavour', ['plain', 'wide', 'split3', 'x3wide'])
def test_kernels_that_take_problem_tables_from_memory_are_launched_plainly(flavour):
    """Tensor maps of a table are read through a proxy of their own, which griddepcontrol.wait is not specified to order."""
    launches = re.findall(r'launch_\w+\(([^,]*),', _source(f'gemm2_{flavour}.cu'))
    assert launches == ['g2_may_chain(probs)']
    assert re.search(r'g2_may_chain\(const GemmProblem2\* table\) \{ return table == nullptr; \}', _source('gemm2_host.h'))
