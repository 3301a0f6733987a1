"""Performance cases: the calls that second-order training makes through the public entry points of ``asdl_b200``.

A K-FAC step measures Kronecker factors (``ops.gram``, ``ops.conv_patch_gram``), refreshes damped inverses
(``ops.spd_inverse_grouped``), applies them to gradients (``ops.kron_apply``), and runs the model's normalisation layers
forward and backward together with their 2x2 curvature blocks.  Every listed case is one of these calls at a size that a
configuration, test or benchmark of this repository uses, or a whole cycle of training steps; ``draw`` gives other sizes of
the same ranges, ragged ones among them.

Kinds (``case["kind"]``):
  gram     factor of a linear layer: rows x n samples, fp32 or bf16, moving average folded in when ``beta`` is not 0
  conv     input-side factor of a convolution: channels_last bf16 (the fused models) or NCHW fp32 (plain PyTorch models)
  kron     two-sided product B^-1 G A^-1 of an m x n gradient
  inverse  damped inverses of a set of factors (``sizes``: comma-separated)
  bn       training BatchNorm (+ residual, + ReLU), forward, backward and, with ``curvature``, its 2x2 blocks
  ln       the same for LayerNorm
  cycle    ten K-FAC training steps of a bottleneck ResNet: one that refreshes curvature and inverses, nine that do not
"""
import torch
import torch.nn.functional as F

import asdl_b200 as asdl
from asdl_b200 import ops
from asdl_b200.models import resnet_tiny

DEVICE = 'cuda'
DAMPING = 1e-3
CYCLE = 10   # steps between curvature / inverse updates in 'cycle'


def _resnet50_sizes():
    """Factor sizes (inputs and outputs) of the 53 convolutions and the head of ResNet-50."""
    sizes, cin = [3 * 49, 64], 64
    for width, blocks in ((64, 3), (128, 4), (256, 6), (512, 3)):
        for b in range(blocks):
            sizes += [cin, width, 9 * width, width, width, 4 * width]
            if b == 0:
                sizes += [cin, 4 * width]
            cin = 4 * width
    return sizes + [2048, 1000]


def listed():
    return [
        # smallest call of a training step: the input factor of an MNIST MLP's first layer, batch 128
        {'name': 'mlp_factor', 'kind': 'gram', 'rows': 128, 'n': 784, 'dtype': 'float32', 'beta': 0.0},
        # ViT-B/16 in fp32, 64 images of 197 tokens: a row count that no tile divides
        {'name': 'vit_factor_fp32', 'kind': 'gram', 'rows': 12608, 'n': 768, 'dtype': 'float32', 'beta': 0.95},
        # GPT-2-medium in bf16, 8 x 1024 tokens: the attention width ...
        {'name': 'gpt2_factor', 'kind': 'gram', 'rows': 8192, 'n': 1024, 'dtype': 'bfloat16', 'beta': 0.95},
        # ... and the MLP width, its largest factor
        {'name': 'gpt2_mlp_factor', 'kind': 'gram', 'rows': 8192, 'n': 4096, 'dtype': 'bfloat16', 'beta': 0.95},
        # ResNet-50, 32 images: a 3 x 3 convolution of the third stage in the fused bf16 model
        {'name': 'conv_factor_bf16', 'kind': 'conv', 'batch': 32, 'channels': 256, 'side': 14, 'kernel': 3, 'stride': 1,
         'dtype': 'bfloat16', 'beta': 0.95},
        # CIFAR ResNet-18, batch 128: a first-stage convolution of a plain fp32 NCHW model
        {'name': 'conv_factor_fp32', 'kind': 'conv', 'batch': 128, 'channels': 64, 'side': 32, 'kernel': 3, 'stride': 1,
         'dtype': 'float32', 'beta': 0.95},
        # GPT-2-medium: one MLP weight gradient preconditioned
        {'name': 'precondition', 'kind': 'kron', 'm': 1024, 'n': 4096},
        # inverses of the MLP 784-512-512-10
        {'name': 'inverse_mlp', 'kind': 'inverse', 'sizes': '784,512,512,512,512,10'},
        # inverses of every factor of ResNet-50 on one GPU
        {'name': 'inverse_resnet50', 'kind': 'inverse', 'sizes': ','.join(str(s) for s in _resnet50_sizes())},
        # ResNet-50, 32 images: the last normalisation of a first-stage block (residual add and ReLU inside)
        {'name': 'batchnorm_block', 'kind': 'bn', 'batch': 32, 'channels': 256, 'side': 56, 'residual': True, 'relu': True,
         'curvature': False},
        # GPT-2-medium: a LayerNorm in a step that measures the curvature
        {'name': 'layernorm_curvature', 'kind': 'ln', 'rows': 8192, 'd': 1024, 'curvature': True},
        # whole training steps: 32 images of 224 x 224 through one bottleneck block per stage
        {'name': 'kfac_cycle', 'kind': 'cycle', 'batch': 32, 'image': 224, 'width': 64},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(['gram', 'gram', 'conv', 'conv', 'kron', 'inverse', 'bn', 'bn', 'ln', 'ln', 'cycle'])
    if kind == 'gram':
        dtype = rng.choice(['float32', 'bfloat16'])
        n = _log(rng, 64, 4096 if dtype == 'bfloat16' else 2048)
        if dtype == 'bfloat16' and rng.random() < 0.7:
            n = max(64, n // 64 * 64)   # most hidden sizes are multiples of 64; the others are staged with a pitch
        return {'kind': kind, 'rows': _log(rng, 32, 8192), 'n': n, 'dtype': dtype, 'beta': rng.choice([0.0, 0.95])}
    if kind == 'conv':
        dtype = rng.choice(['float32', 'bfloat16'])
        return {'kind': kind, 'batch': rng.randint(4, 32), 'channels': rng.choice([3, 24, 32, 64, 96, 128, 192]),
                'side': rng.randint(7, 32), 'kernel': rng.choice([1, 3, 3, 5]), 'stride': rng.choice([1, 1, 2]),
                'dtype': dtype, 'beta': rng.choice([0.0, 0.95])}
    if kind == 'kron':
        return {'kind': kind, 'm': _log(rng, 10, 2048), 'n': _log(rng, 32, 2560)}
    if kind == 'inverse':
        return {'kind': kind, 'sizes': ','.join(str(_log(rng, 8, 2304)) for _ in range(rng.randint(1, 24)))}
    if kind == 'bn':
        residual = rng.random() < 0.4
        return {'kind': kind, 'batch': rng.randint(4, 32), 'channels': 8 * _log(rng, 2, 64), 'side': rng.randint(7, 40),
                'residual': residual, 'relu': residual or rng.random() < 0.7, 'curvature': rng.random() < 0.4}
    if kind == 'ln':
        return {'kind': kind, 'rows': _log(rng, 64, 8192), 'd': 256 * rng.choice([1, 2, 3, 4, 6, 8, 12]),
                'curvature': rng.random() < 0.5}
    return {'kind': kind, 'batch': rng.randint(4, 24), 'image': 32 * rng.randint(2, 6), 'width': rng.choice([16, 32, 48])}


def _sizes(case):
    return [int(s) for s in case['sizes'].split(',')]


def _conv_out(case):
    k, s = case['kernel'], case['stride']
    return (case['side'] + 2 * (k // 2) - k) // s + 1


def _spd(n, gen, rows=None):
    """A factor as training sees it: a mean of outer products whose features differ in scale."""
    x = torch.randn(rows or 2 * n, n, generator=gen, device=DEVICE)
    x *= torch.linspace(1.0, 0.1, n, device=DEVICE)
    return x.T @ x / x.shape[0]


def _flat_views(sizes):
    """One buffer with room for all matrices, 64-element aligned, and the matrices as views of it."""
    offsets, total = [], 0
    for n in sizes:
        offsets.append(total)
        total += (n * n + 63) // 64 * 64
    return offsets, total


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed))
    kind = case['kind']

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=DEVICE)

    if kind == 'gram':
        x = randn(case['rows'], case['n']).to(getattr(torch, case['dtype']))
        state = {'x': x, 'scale': (1 - case['beta']) / case['rows']}
        if case['beta']:
            state['factor'] = _spd(case['n'], gen, rows=256)   # every pass adds to the moving average in place
    elif kind == 'conv':
        k = case['kernel']
        x = torch.relu(randn(case['batch'], case['channels'], case['side'], case['side']))
        last = case['dtype'] == 'bfloat16'
        if last:
            x = x.to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        conv = torch.nn.Conv2d(case['channels'], 8, k, stride=case['stride'], padding=k // 2, bias=False).to(DEVICE)
        rows = case['batch'] * _conv_out(case) ** 2
        state = {'x': x, 'conv': conv, 'last': last, 'scale': (1 - case['beta']) / rows}
        if case['beta']:
            state['factor'] = _spd(case['channels'] * k * k, gen, rows=256)
    elif kind == 'kron':
        def inverse_of_factor(n):
            m = _spd(n, gen)
            m.diagonal().add_(0.03)
            return torch.cholesky_inverse(torch.linalg.cholesky(m))
        state = {'left': inverse_of_factor(case['m']), 'right': inverse_of_factor(case['n']),
                 'grad': randn(case['m'], case['n']) * 1e-2}
    elif kind == 'inverse':
        sizes = _sizes(case)
        offsets, total = _flat_views(sizes)
        flat = torch.zeros(total, device=DEVICE)
        state = {'mats': [_spd(n, gen) for n in sizes], 'flat': flat,
                 'outs': [flat[o:o + n * n].view(n, n) for o, n in zip(offsets, sizes)]}
    elif kind == 'bn':
        shape = (case['batch'], case['channels'], case['side'], case['side'])
        c = case['channels']

        def activation(scale=1.0):
            return (randn(*shape) * scale).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        state = {'x': activation().requires_grad_(True), 'dy': activation(1e-2),
                 'residual': activation().requires_grad_(True) if case['residual'] else None,
                 'weight': (1 + 0.1 * randn(c)).requires_grad_(True), 'bias': (0.1 * randn(c)).requires_grad_(True),
                 'mean': torch.zeros(c, device=DEVICE), 'var': torch.ones(c, device=DEVICE),
                 'tracked': torch.zeros((), dtype=torch.int64, device=DEVICE)}
        if case['curvature']:
            state['blocks'] = torch.empty(c, 2, 2, device=DEVICE)
    elif kind == 'ln':
        rows, d = case['rows'], case['d']
        state = {'x': randn(rows, d).to(torch.bfloat16).requires_grad_(True), 'dy': (1e-2 * randn(rows, d)).to(torch.bfloat16),
                 'weight': (1 + 0.1 * randn(d)).requires_grad_(True), 'bias': (0.1 * randn(d)).requires_grad_(True)}
        if case['curvature']:
            state['blocks'] = torch.empty(d, 2, 2, device=DEVICE)
    else:
        with torch.random.fork_rng(devices=[torch.device(DEVICE, torch.cuda.current_device())]):
            torch.manual_seed(int(seed))
            with torch.device(DEVICE):
                model = resnet_tiny(num_classes=1000, width=case['width'], fused=True)
        model = model.to(memory_format=torch.channels_last)
        config = asdl.PreconditioningConfig(data_size=case['batch'], damping=DAMPING, curvature_upd_interval=CYCLE,
                                            preconditioner_upd_interval=CYCLE)
        maker = asdl.FusedKfacGradientMaker(model, config, fisher_type='fisher_emp', cuda_graph=True)
        image = randn(case['batch'], 3, case['image'], case['image']).contiguous(memory_format=torch.channels_last)
        label = torch.randint(0, 1000, (case['batch'],), generator=gen, device=DEVICE)

        def forward(inputs):
            with torch.autocast('cuda', dtype=torch.bfloat16):
                return model(inputs)
        state = {'model': model, 'maker': maker, 'forward': forward, 'image': image, 'label': label}
        state['case'] = dict(case)
        run(state)   # the first cycle: inverses exist and the steps are captured after it
    state['case'] = dict(case)
    return state


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'gram':
        if case['beta']:
            return ops.gram(state['x'], scale=state['scale'], out=state['factor'], beta=case['beta'])
        return ops.gram(state['x'], scale=state['scale'])
    if kind == 'conv':
        if case['beta']:
            return ops.conv_patch_gram(state['x'], state['conv'], scale=state['scale'], out=state['factor'],
                                       beta=case['beta'], channels_last_order=state['last'])
        return ops.conv_patch_gram(state['x'], state['conv'], scale=state['scale'], channels_last_order=state['last'])
    if kind == 'kron':
        return ops.kron_apply(state['left'], state['grad'], state['right'])
    if kind == 'inverse':
        ops.spd_inverse_grouped(state['mats'], state['outs'], DAMPING)
        return state['flat']
    if kind == 'bn':
        x, weight, bias, residual = state['x'], state['weight'], state['bias'], state['residual']
        y, mean, invstd = ops.batch_norm_train(x, weight, bias, state['mean'], state['var'], residual=residual,
                                               relu=case['relu'], num_batches_tracked=state['tracked'], return_stats=True)
        leaves = [x, weight, bias] + ([residual] if residual is not None else [])
        out = {'y': y.detach(), 'mean': mean, 'invstd': invstd}
        out['grads'] = list(torch.autograd.grad(y, leaves, state['dy']))
        if case['curvature']:
            out['blocks'] = ops.batchnorm_unitwise_stats_from_input(
                x.detach(), state['dy'], y.detach() if case['relu'] else None, mean, invstd, state['blocks'])
        return out
    if kind == 'ln':
        x, weight, bias = state['x'], state['weight'], state['bias']
        y = ops.layer_norm(x, weight, bias)
        out = {'y': y.detach(), 'grads': list(torch.autograd.grad(y, [x, weight, bias], state['dy']))}
        if case['curvature']:
            out['blocks'] = ops.layernorm_unitwise_stats(y.detach(), state['dy'], weight, bias, out=state['blocks'])
        return out
    maker = state['maker']
    for _ in range(CYCLE):
        dummy = maker.setup_model_call(state['forward'], state['image'])
        maker.setup_loss_call(F.cross_entropy, dummy, state['label'])
        logits, loss = maker.forward_and_backward()
    return {'logits': logits.detach(), 'loss': loss.detach(), 'grads': [p.grad for p in state['model'].parameters()]}


def work(case):
    kind = case['kind']
    if kind == 'gram':
        size, n = (2 if case['dtype'] == 'bfloat16' else 4), case['n']
        # a symmetric result: half of the products; the moving average reads and writes the factor
        return {'bytes': size * case['rows'] * n + 4 * n * n * (2 if case['beta'] else 1),
                'flops': case['rows'] * n * (n + 1)}
    if kind == 'conv':
        size, n = (2 if case['dtype'] == 'bfloat16' else 4), case['channels'] * case['kernel'] ** 2
        rows = case['batch'] * _conv_out(case) ** 2
        return {'bytes': size * case['batch'] * case['channels'] * case['side'] ** 2 + 4 * n * n * (2 if case['beta'] else 1),
                'flops': rows * n * (n + 1)}
    if kind == 'kron':
        m, n = case['m'], case['n']
        return {'bytes': 4 * (m * m + n * n + 2 * m * n), 'flops': 2 * m * n * (m + n)}
    if kind == 'inverse':
        sizes = _sizes(case)
        # Cholesky factor, triangular inverse and the product of the two triangles: n^3 multiply-adds / 2 in all
        return {'bytes': 8 * sum(n * n for n in sizes), 'flops': sum(n ** 3 for n in sizes)}
    if kind == 'bn':
        size = case['batch'] * case['channels'] * case['side'] ** 2
        # forward: x (and the residual) in, y out; backward: dy and x in, dx (and the residual's gradient) out
        passes = 5 + (2 if case['residual'] else 0) + (2 if case['curvature'] else 0)
        return {'bytes': 2 * size * passes, 'flops': 20 * size}
    if kind == 'ln':
        size = case['rows'] * case['d']
        return {'bytes': 2 * size * (5 + (2 if case['curvature'] else 0)), 'flops': 20 * size}
    width, batch, side = case['width'], case['batch'], case['image'] / 4
    # multiply-adds of the four blocks' convolutions, forward and twice that backward, ten times
    macs, cin, params = batch * 147 * width * (2 * side) ** 2, width, 150 * width
    for stage in range(4):
        planes = width * 2 ** stage
        out = side / 2 ** max(stage, 0)
        weights = cin * planes + 9 * planes * planes + 4 * planes * planes + 4 * cin * planes
        macs += batch * weights * out ** 2
        params += weights
        cin = 4 * planes
    params += 1000 * cin
    activations = batch * width * (2 * side) ** 2 + batch * sum(
        (2 + 4 + 4) * width * 2 ** s * (side / 2 ** s) ** 2 for s in range(4))
    return {'bytes': CYCLE * (4 * params * 3 + 2 * activations * 10), 'flops': CYCLE * 6 * macs}


def tolerance(case):
    kind = case['kind']
    if kind in ('gram', 'conv'):
        if case['dtype'] == 'bfloat16':
            return {'rel': 5e-6, 'max': 2e-4}   # exact products, fp32 sums
        return {'rel': 4e-5, 'max': 1e-3}       # fp32 inputs enter as bf16 pairs (2^-16 of a product)
    if kind == 'kron':
        return {'rel': 4e-5, 'max': 1e-3}       # two chained products of bf16 pairs
    if kind == 'inverse':
        return {'rel': 5e-6, 'max': 2e-4}       # fp32 arithmetic times the condition number
    if kind in ('bn', 'ln'):
        return {'rel': 4e-3, 'max': 0.99}       # bf16 activations; a ReLU mask may flip where the output is zero
    return {'rel': 0.03, 'max': 0.99}           # bf16 roundings travel through the model and the inverses


def exact(case, seed):
    kind = case['kind']
    if kind == 'cycle':
        return None
    s = prepare(case, seed)
    if kind in ('gram', 'conv'):
        x = s['x'].double()
        if kind == 'conv':
            x = F.unfold(x, case['kernel'], padding=case['kernel'] // 2, stride=case['stride'])
            if s['last']:   # (c, kh, kw) -> (kh, kw, c)
                b, _, pixels = x.shape
                x = x.view(b, case['channels'], case['kernel'] ** 2, pixels).transpose(1, 2).reshape(b, -1, pixels)
            x = x.transpose(1, 2).reshape(-1, x.shape[1])
        out = x.T @ x * s['scale']
        return out + case['beta'] * s['factor'].double() if case['beta'] else out
    if kind == 'kron':
        return s['left'].double() @ s['grad'].double() @ s['right'].double()
    if kind == 'inverse':
        flat = torch.zeros(s['flat'].numel(), dtype=torch.float64, device=DEVICE)
        offsets, _ = _flat_views(_sizes(case))
        for o, m in zip(offsets, s['mats']):
            d = m.double()
            d.diagonal().add_(DAMPING)
            flat[o:o + m.numel()] = torch.cholesky_inverse(torch.linalg.cholesky(d)).reshape(-1)
        return flat
    w, b, dy = s['weight'].detach().double(), s['bias'].detach().double(), s['dy'].double()
    x = s['x'].detach().double()
    if kind == 'ln':
        mean = x.mean(1, keepdim=True)
        rstd = (x.var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
        xh, g = (x - mean) * rstd, dy * w
        dx = rstd * (g - g.mean(1, keepdim=True) - xh * (g * xh).mean(1, keepdim=True))
        out = {'y': xh * w + b, 'grads': [dx, (dy * xh).sum(0), dy.sum(0)]}
        if case['curvature']:
            out['blocks'] = None   # measured from the rounded output: no value of its own in 64 bits
        return out
    dims, view = (0, 2, 3), (1, -1, 1, 1)
    mean, var = x.mean(dims), x.var(dims, unbiased=False)
    invstd = (var + 1e-5).rsqrt()
    xh = (x - mean.view(view)) * invstd.view(view)
    y = xh * w.view(view) + b.view(view)
    if case['residual']:
        y = y + s['residual'].detach().double()
    g = dy
    if case['relu']:
        g = dy * (y > 0)
        y = y.relu()
    dw, db = (g * xh).sum(dims), g.sum(dims)
    count = x.numel() // x.shape[1]
    dx = (w * invstd).view(view) * (g - (db / count).view(view) - xh * (dw / count).view(view))
    out = {'y': y, 'mean': mean, 'invstd': invstd, 'grads': [dx, dw, db] + ([g] if case['residual'] else [])}
    if case['curvature']:
        gw, gb = (g * xh).sum((2, 3)), g.sum((2, 3))
        ww, wb, bb = (gw * gw).sum(0), (gw * gb).sum(0), (gb * gb).sum(0)
        out['blocks'] = torch.stack([torch.stack([ww, wb], 1), torch.stack([wb, bb], 1)], 1)
    return out
