"""The tensor-core inverse is fp32-grade: its bf16 parts carry the whole significand.  The bound that tells three parts from two is
shown on the CPU, where both are restated in tiles, and then asked of the kernel."""
import pytest
import torch

from asdl_b200 import ops

TILE = 128
#: error relative to that of LAPACK's fp32 inverse of the same matrix: three parts stay below 3, two are above 40
GRADE = 6


def _matrix(n, seed=0):
    x = torch.randn(2 * n, n, generator=torch.Generator().manual_seed(seed))
    return x.T @ x / (2 * n)


def _errors(a, damping, *inverses):
    """Errors of inverses of a + damping, relative to that of LAPACK's in fp32."""
    a = a + damping * torch.eye(a.shape[0])
    want = torch.linalg.inv(a.double())

    def error(got):
        return ((got.double() - want).norm() / want.norm()).item()
    lapack = error(torch.cholesky_inverse(torch.linalg.cholesky(a)))
    return [error(got) / lapack for got in inverses]


def _product(a, b, parts):
    """a b of bf16 parts, the part products that matter at that number of them."""
    def split(x):
        out = []
        for _ in range(parts):
            out.append(x.bfloat16().float())
            x = x - out[-1]
        return out
    a, b = split(a), split(b)
    return sum(a[i] @ b[j] for i in range(parts) for j in range(parts) if i + j < parts)


def _tiled_inverse(a, parts):
    """Factor, triangular inverse and product of both in tiles, as ``csrc/chol_inverse_tc.cu`` orders them."""
    n = a.shape[0]
    blocks = [slice(i, min(n, i + TILE)) for i in range(0, n, TILE)]
    low, inv = torch.zeros_like(a), torch.zeros_like(a)
    for j, sj in enumerate(blocks):
        before = slice(0, sj.start)

        def rest(s):
            return a[s, sj] - (_product(low[s, before], low[sj, before].T, parts) if j else 0)
        factor = torch.linalg.cholesky(rest(sj))
        inv[sj, sj] = torch.linalg.solve_triangular(factor, torch.eye(factor.shape[0]), upper=False)
        for si in blocks[j + 1:]:
            low[si, sj] = _product(rest(si), inv[sj, sj].T, parts)
    for j, sj in enumerate(blocks):
        for si in blocks[j + 1:]:
            between = slice(sj.start, si.start)
            inv[si, sj] = -_product(inv[si, si], _product(low[si, between], inv[between, sj], parts), parts)
    return _product(inv.T, inv, parts)


@pytest.mark.parametrize('n', [300, 512, 1153])
def test_the_bound_tells_three_parts_from_two(n):
    a = _matrix(n)
    damped = a + 1e-2 * torch.eye(n)
    three, two = _errors(a, 1e-2, _tiled_inverse(damped, 3), _tiled_inverse(damped, 2))
    assert three < GRADE / 2 and two > 5 * GRADE


@pytest.mark.gpu
@pytest.mark.parametrize('sizes', [(300,), (512, 129, 257), (1153, 640, 700, 385), (2048,)])
def test_the_tensor_core_inverse_is_fp32_grade(sizes):
    mats = [_matrix(n, i) for i, n in enumerate(sizes)]
    outs = [torch.empty(n, n, device='cuda') for n in sizes]
    ops.extension().chol_inverse_tc([m.cuda() for m in mats], outs, torch.full((len(sizes),), 1e-2, device='cuda'))
    ops.check_status()
    for m, out in zip(mats, outs):
        assert _errors(m, 1e-2, out.cpu())[0] < GRADE
