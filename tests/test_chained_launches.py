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
    assert len(launches) == 1 and re.fullmatch(r'g2_may_chain\(probs\)( && !\w+)?', launches[0])
    assert re.search(r'g2_may_chain\(const GemmProblem2\* table\) \{ return table == nullptr; \}', _source('gemm2_host.h'))


#: read-only parameters of kernels that wait on a chain: written before the chain's first kernel, which is launched plainly
OLDER_THAN_THE_CHAIN = {'x', 'dy', 'y', 'res', 'weight', 'bias', 'mean', 'invstd', 'probs', 'work', 'prefix_g', 'tile_prefix'}


def _kernels(name):
    """(name, parameters, body) of the kernels of a file."""
    text = re.sub(r'__(launch_bounds|cluster_dims)__\([^()]*\)', '', _source(name))
    for head in re.finditer(r'__global__\s+void\s+(\w+)\(', text):
        start = text.index('{', head.end())
        depth, end = 1, start + 1
        while depth:
            depth += {'{': 1, '}': -1}.get(text[end], 0)
            end += 1
        yield head.group(1), text[head.end():start], text[start:end]


def test_what_a_chain_has_written_is_read_by_ordinary_loads():
    """The read-only path is for data that nobody writes while the kernel is resident, and a chained kernel is resident early."""
    found = set()
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(('.cu', '.cuh'))):
        for kernel, params, body in _kernels(name):
            if 'chain_wait()' not in body:
                continue
            found.add(kernel)
            read_only = set(re.findall(r'const [\w:]+\* __restrict__ (\w+)', params))
            assert read_only <= OLDER_THAN_THE_CHAIN, (kernel, read_only - OLDER_THAN_THE_CHAIN)
            assert '__ldg(' not in body and '__ldcs(' not in body, kernel
            if '__ldcg(' in body:
                assert 'after_wait(' in body, kernel
    assert found >= {'bn_fwd_finalize', 'bn_apply', 'bn_bwd_finalize', 'bn_dx', 'cg_product_kernel', 'cg_reduce_kernel',
                     'umma_gemm2_kernel', 'umma_gemm2_pair_kernel', 'splitk_reduce2_kernel'}


def test_every_kernel_of_a_chain_waits():
    """A kernel that ends without waiting would let the kernel behind it run ahead of the one in front."""
    chained = set()
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(('.cu', '.cuh'))):
        chained |= {k for k in re.findall(r'launch_chained\((\w+)', _source(name)) if k != 'kernel'}
        chained |= set(re.findall(r'launch_behind\([^,]*, (\w+)', _source(name))) - {'kernel'}
    waiting = {k for name in os.listdir(CSRC) if name.endswith(('.cu', '.cuh')) for k, _, body in _kernels(name)
               if 'chain_wait()' in body}
    assert chained and chained <= waiting


def test_chains_whose_kernels_read_ahead_of_the_wait_begin_with_a_plain_launch():
    """Only the last kernels of BatchNorm do, and what they read there is older than the chain because bn_sums is launched plainly."""
    ahead = {k for name in os.listdir(CSRC) if name.endswith(('.cu', '.cuh')) for k, _, body in _kernels(name)
             if 'chain_wait()' in body and re.search(r'\bfetch\w*\(', body[:body.index('chain_wait()')])}
    assert ahead == {'bn_apply', 'bn_dx'}
    text = _source('batchnorm.cu')
    launches = text[text.index('std::vector<at::Tensor> bn_forward_train('):]
    for use in re.finditer(r'bn_sums<[^>]*>', launches):
        assert launches[use.end():].startswith('<<<') or launches[:use.start()].endswith('sums(')
    assert len(re.findall(r'auto sums = \[&\]\(auto kernel\) \{\s*kernel<<<', launches)) == 1
    for name in ('bn_forward_train', 'bn_backward_train'):
        body = launches[launches.index(name + '('):]
        assert re.search(r'<<<|launch_chained\(', body).group() == '<<<'
