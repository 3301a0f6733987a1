"""What captured CUDA graphs and other streams read stays in place: tables of the grouped inverses, split-K partials."""
import subprocess
import sys
import time

import pytest
import torch

from asdl_b200 import ops

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _spd(n, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    x = torch.randn(2 * n, n, device=DEV, generator=g)
    return x.T @ x / (2 * n)


def _check(mats, outs, damping):
    for m, o in zip(mats, outs):
        d = m.double()
        d.diagonal().add_(damping)
        want = torch.linalg.inv(d)
        # n * 2^-24 times the condition number bounds the error of a Cholesky inverse, relative to the largest entry
        bound = 4 * max(m.shape[0], 8) * 2.0 ** -24 * torch.linalg.cond(d).item() * want.abs().max()
        assert (o.double() - want).abs().max() <= bound


@pytest.mark.parametrize('backend,info,capacity', [('tensor_core', 'chol_inverse_tc_cache_info', 4),
                                                    ('cuda_core', 'chol_inverse_cache_info', 16)])
def test_a_captured_inverse_keeps_its_tables(monkeypatch, backend, info, capacity):
    monkeypatch.setattr(ops, 'CHOLESKY_BACKEND', backend)
    info = getattr(ops.extension(), info)
    sizes, damping = (300, 40, 129), 1e-2
    mats = [_spd(n, 20 + n) for n in sizes]
    outs = [torch.empty_like(m) for m in mats]
    damp = torch.full((len(sizes),), damping, device=DEV)
    ops.spd_inverse_grouped(mats, outs, damp)
    kept_before = info()[1]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.spd_inverse_grouped(mats, outs, damp)
    others = [(_spd(70 + i, i), torch.empty(70 + i, 70 + i, device=DEV)) for i in range(capacity + 2)]
    for m, o in others:
        ops.spd_inverse_grouped([m], [o], damping)
    entries, kept = info()
    assert kept == kept_before + 1      # more sets than the cache holds went by; the captured one is still there
    assert entries - kept <= capacity
    for m, o, n in zip(mats, outs, sizes):
        m.copy_(_spd(n, 40 + n))
        o.zero_()
    graph.replay()
    torch.cuda.synchronize()
    _check(mats, outs, damping)
    _check(*zip(*others), damping)
    ops.check_status()
    graph.reset()
    deadline = time.monotonic() + 10    # the graph gives its references back asynchronously
    while info()[1] > kept_before and time.monotonic() < deadline:
        time.sleep(0.01)
    assert info()[1] == kept_before
    for m, o in others:
        ops.spd_inverse_grouped([m], [o], damping)
    assert info()[0] - info()[1] <= capacity


@pytest.mark.parametrize('backend', ['tensor_core', 'cuda_core'])
def test_tables_evicted_while_another_stream_uses_them(monkeypatch, backend):
    monkeypatch.setattr(ops, 'CHOLESKY_BACKEND', backend)
    mats = [_spd(n, 60 + n) for n in (260, 500, 64)]
    outs = [torch.empty_like(m) for m in mats]
    ops.spd_inverse_grouped(mats, outs, 1e-2)          # the tables belong to this stream
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(8):
            ops.spd_inverse_grouped(mats, outs, 1e-2)  # ... and are still in use there
    for i in range(20):
        m = _spd(90 + i, i)
        ops.spd_inverse_grouped([m], [torch.empty_like(m)], 1e-2)
        torch.empty(64 << 20, device=DEV, dtype=torch.uint8).fill_(255)
    torch.cuda.current_stream().wait_stream(side)
    _check(mats, outs, 1e-2)
    ops.check_status()


_REPLAY_AFTER_GROWTH = """
import torch
from asdl_b200 import ops
x = torch.randn(4096, 200, device='cuda', generator=torch.Generator(device='cuda').manual_seed(0)).to(torch.bfloat16)
want = ops.gram(x)                                     # creates the ring of split-K partials
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = ops.gram(x)
ops.extension().reserve_scratch(0, 64 << 20)           # a larger one takes its place
fillers = [torch.ones(4 << 20, device='cuda') for _ in range(4)]   # ... and others get the memory of the first
out.zero_()
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, want)
assert all(bool((f == 1).all()) for f in fillers), 'the replay wrote to memory that is not its own'
"""


def test_a_replay_leaves_the_former_ring_of_partials_alone():
    done = subprocess.run([sys.executable, '-c', _REPLAY_AFTER_GROWTH], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


_EXIT_AFTER_SIDE_STREAM = """
import torch
from asdl_b200 import ops
ops.extension()                       # loaded before CUDA starts, so its static objects outlive CUDA's
for backend in ('tensor_core', 'cuda_core'):
    ops.CHOLESKY_BACKEND = backend
    a, out = torch.eye(200, device='cuda'), torch.empty(200, 200, device='cuda')
    ops.spd_inverse_grouped([a], [out], 1e-2)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ops.spd_inverse_grouped([a], [out], 1e-2)
torch.cuda.synchronize()
"""


def test_a_process_that_used_two_streams_ends_cleanly():
    done = subprocess.run([sys.executable, '-c', _EXIT_AFTER_SIDE_STREAM], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
