"""Staging, reduction, normalisation and factorisation kernels at the sizes where their tiles, vectors and lanes end."""
import pytest
import torch
import torch.nn.functional as F

from asdl_b200 import ops
from asdl_b200.models.layers import FusedMaxPool2d

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.fixture(scope='module')
def ext():
    e = ops.extension()
    yield e
    ops.check_status()


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('rows,n,ld,offset', [(1, 1, 8, 0), (3, 7, 8, 0), (37, 64, 64, 0), (130, 65, 72, 0), (2, 2057, 2064, 0),
                                              (1300, 24, 24, 0), (9, 40, 40, 1), (5, 9, 12, 0)])
def test_cast_parts(ext, dtype, rows, n, ld, offset):
    x = torch.randn(rows, n + offset, device=DEV, generator=_gen(0)).to(dtype)[:, offset:]
    hi = torch.full((rows, ld), float('nan'), device=DEV, dtype=torch.bfloat16)
    lo = torch.full_like(hi, float('nan'))
    ext.cast_pad_bf16(x, hi, lo, 1.0)
    want = F.pad(x.float(), (0, ld - n))
    assert torch.equal(hi, want.to(torch.bfloat16))
    assert torch.equal(lo, (want - hi.float()).to(torch.bfloat16))
    one = torch.empty_like(hi)
    ext.cast_pad_bf16(x, one, None, 0.5)
    assert torch.equal(one, (want * 0.5).to(torch.bfloat16))


@pytest.mark.parametrize('scale', [float('inf'), float('nan'), -1.0])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
def test_cast_pads_with_zeros_whatever_the_scale(ext, dtype, scale):
    x = torch.ones(5, 11, device=DEV, dtype=dtype)
    hi, lo = (torch.full((5, 24), float('nan'), device=DEV, dtype=torch.bfloat16) for _ in range(2))
    ext.cast_pad_bf16(x, hi, lo, scale)
    assert torch.equal(hi[:, :11], torch.full((5, 11), scale, device=DEV).to(torch.bfloat16)) or scale != scale
    for part in (hi, lo):
        assert not part[:, 11:].view(torch.int16).any()


@pytest.mark.parametrize('rows', [1, 3])
def test_cast_of_more_columns_than_a_grid_has_blocks_on_y(ext, rows):
    n = 65535 * 2048 + 11
    x = torch.randn(rows, n, device=DEV, generator=_gen(20))
    hi, lo = (torch.full((rows, (n + 7) // 8 * 8), float('nan'), device=DEV, dtype=torch.bfloat16) for _ in range(2))
    ext.cast_pad_bf16(x, hi, lo, 1.0)
    assert torch.equal(hi[:, :n], x.to(torch.bfloat16)) and not hi[:, n:].any()
    assert torch.equal(lo[:, :n], (x - hi[:, :n].float()).to(torch.bfloat16)) and not lo[:, n:].any()


def test_batch_norm_of_more_channels_than_a_grid_has_blocks_on_y():
    c = 65535 * 2048 + 8
    x = torch.randn(2, c, 1, 1, device=DEV, generator=_gen(21), dtype=torch.bfloat16)
    x = x.contiguous(memory_format=torch.channels_last).requires_grad_(True)
    weight, bias = torch.full((c,), 0.5, device=DEV), torch.full((c,), 0.25, device=DEV)
    y = ops.batch_norm_train(x, weight, bias)
    dx, = torch.autograd.grad(y, x, torch.ones_like(y))
    d = (x[0] - x[1]).detach().float().flatten() / 2
    want = 0.25 + 0.5 * d * torch.rsqrt(d * d + 1e-5)
    assert (y[0].flatten() - want).abs().max() <= 2.0 ** -8     # one bf16 rounding of values below 1
    assert dx.abs().max() <= 1e-3                               # a constant gradient has no component along x or 1


def test_outputs_without_columns_are_refused(ext):
    parts = [torch.empty(3, 0, device=DEV, dtype=torch.bfloat16) for _ in range(3)]
    with pytest.raises(RuntimeError, match='no columns'):
        ext.cast_split3(torch.empty(3, 0, device=DEV), *parts)
    x = torch.empty(1, 0, 4, 4, device=DEV, dtype=torch.bfloat16).as_strided((1, 0, 4, 4), (0, 1, 0, 0))
    with pytest.raises(RuntimeError, match='no columns'):
        ext.im2col_bf16(x, torch.empty(16, 0, device=DEV, dtype=torch.bfloat16), None, [1, 1], [1, 1], [0, 0], [1, 1], False)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('cfg', [  # n, c, h, w, kernel, stride, padding, dilation
    (2, 8, 9, 7, 3, 1, 1, 1), (1, 3, 12, 11, 7, 2, 3, 1), (2, 24, 8, 8, 3, 2, 1, 1), (1, 5, 13, 13, 3, 1, 2, 2),
    (1, 300, 9, 9, 5, 1, 2, 1), (3, 16, 5, 5, 1, 2, 0, 1), (1, 1, 3, 40, 3, 1, 1, 1)])
@pytest.mark.parametrize('layout', ['nchw', 'nhwc', 'sliced'])
def test_im2col_layouts(ext, cfg, dtype, layout):
    n, c, h, w, k, s, p, d = cfg
    x = torch.randn(n, c, h, w + 1, device=DEV, generator=_gen(1)).to(dtype)
    x = x[..., 1:] if layout == 'sliced' else x[..., :w].contiguous()
    if layout == 'nhwc':
        x = x.contiguous(memory_format=torch.channels_last)
    cols = F.unfold(x.float(), k, padding=p, stride=s, dilation=d)                 # n x (c kh kw) x pixels
    ld = (c * k * k + 7) // 8 * 8
    for c_major in (True, False):
        want = cols if c_major else cols.view(n, c, k * k, -1).transpose(1, 2).reshape(n, c * k * k, -1)
        want = F.pad(want.transpose(1, 2).reshape(-1, c * k * k), (0, ld - c * k * k))
        for with_lo in (False, True):
            out = torch.full((want.shape[0], ld), float('nan'), device=DEV, dtype=torch.bfloat16)
            lo = torch.full_like(out, float('nan')) if with_lo else None
            ext.im2col_bf16(x, out, lo, [k, k], [s, s], [p, p], [d, d], c_major)
            assert torch.equal(out, want.to(torch.bfloat16))
            if with_lo:
                assert torch.equal(lo, (want - out.float()).to(torch.bfloat16))


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('cfg', [  # rows of pixels enough for the tile kernel: full and part-filled rounds of loads, both chunkings
    (24, 16, 9, 40, 3, 1, 1, 1), (160, 6, 14, 14, 5, 1, 0, 1), (32, 300, 9, 9, 3, 1, 1, 1), (256, 64, 8, 8, 8, 1, 0, 1),
    (16, 24, 30, 31, 2, 2, 0, 1), (40, 33, 12, 12, 3, 1, 2, 2), (512, 1, 28, 28, 5, 1, 0, 1)])
@pytest.mark.parametrize('layout', ['nchw', 'nhwc', 'sliced'])
def test_im2col_tiles(ext, cfg, dtype, layout):
    test_im2col_layouts(ext, cfg, dtype, layout)


@pytest.mark.parametrize('rows,n', [(700, 33), (3000, 130), (2048, 257), (5000, 64)])
@pytest.mark.parametrize('nsplit', [2, 5, 9])
@pytest.mark.parametrize('beta', [0.0, 0.9])
def test_split_k_reduction(ext, rows, n, nsplit, beta):
    x = torch.randn(rows, (n + 7) // 8 * 8, device=DEV, generator=_gen(2)).to(torch.bfloat16)[:, :n]
    old = torch.randn(n, n, device=DEV, generator=_gen(3))
    old = old + old.T
    c = old.clone() if beta else torch.full((n, n), float('nan'), device=DEV)
    ext.umma_gemm([x], [x], False, False, c, 0.25, beta, True, None, None, nsplit)
    want = 0.25 * (x.double().T @ x.double()) + beta * old.double()
    # exact products; every one of the `rows` additions loses at most 2^-22 of the running sum (truncating accumulator)
    bound = rows * 2.0 ** -22 * 0.25 * (x.double().abs().T @ x.double().abs()) + 2.0 ** -22 * beta * old.double().abs()
    assert ((c.double() - want).abs() <= bound).all()
    assert torch.equal(c, c.T)


@pytest.mark.parametrize('rows,n', [(20000, 40), (9000, 200), (4000, 400), (4000, 513)])   # 16- and 32-row patches
@pytest.mark.parametrize('nsplit', [0, 3, 8, 17, 32])
def test_split_k_reduction_patches(ext, rows, n, nsplit):
    test_split_k_reduction(ext, rows, n, nsplit, 0.9)


@pytest.mark.parametrize('m,n,ldc', [(70, 72, 72), (40, 65, 68), (130, 63, 63), (300, 258, 260)])
@pytest.mark.parametrize('nsplit', [1, 3, 17])
def test_split_k_reduction_replicates_its_result(ext, m, n, ldc, nsplit):
    k = 64 * 20
    a, b = (torch.randn(k, (c + 7) // 8 * 8, device=DEV, generator=_gen(30 + c)).to(torch.bfloat16)[:, :c] for c in (m, n))
    outs = [torch.full((m + 1, ldc), 7.0, device=DEV) for _ in range(3)]
    ext.umma_gemm_to_ptr([a], [b], False, False, outs[0].data_ptr(), ldc, 2.0, False, 0, [t.data_ptr() for t in outs[1:]],
                         nsplit, False)
    want = 2.0 * (a.double().T @ b.double())
    # every one of the k additions loses at most 2^-22 of the running sum (truncating accumulator)
    bound = k * 2.0 ** -22 * 2.0 * (a.double().abs().T @ b.double().abs())
    assert ((outs[0][:m, :n].double() - want).abs() <= bound).all()
    for t in outs:
        assert torch.equal(t[:m, :n], outs[0][:m, :n])
        assert (t[m:] == 7).all() and (t[:, n:] == 7).all()      # nothing outside of the matrix is written


def test_kron_apply_reads_either_order_of_a_symmetric_factor():
    left, right = (torch.randn(n, n, device=DEV, generator=_gen(4 + n)) for n in (72, 130))
    left, right = left + left.T, right + right.T
    mid = torch.randn(72, 130, device=DEV, generator=_gen(4))
    row = ops.kron_apply(left, mid, right)
    col = ops.kron_apply(left.T.contiguous().T, mid, right.T.contiguous().T)
    assert torch.equal(row, col)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('m,n', [(1, 1), (8, 24), (72, 130), (257, 129), (129, 640)])
def test_kron_apply_gives_the_same_bits_for_either_order_of_storage(m, n, dtype):
    # not symmetric, so that a factor read as its transpose shows: inverses are symmetric up to their last bits only
    left, right = (torch.randn(k, k, device=DEV, generator=_gen(4 + k)).to(dtype) for k in (m, n))
    mid = torch.randn(m, n, device=DEV, generator=_gen(4)).to(dtype)
    row = ops.kron_apply(left, mid, right)
    for a in (left, left.T.contiguous().T):
        for b in (right, right.T.contiguous().T):
            assert torch.equal(ops.kron_apply(a, mid, b), row)


@pytest.mark.parametrize('n', [1, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 160, 225, 257])
def test_inverse_at_the_edges_of_the_diagonal_stages(n):
    x = torch.randn(2 * n, n, device=DEV, generator=_gen(19))
    a = x.T @ x / (2 * n)
    before = a.clone()
    got = ops.spd_inverse(a, 1e-2)
    d = a.double()
    d.diagonal().add_(1e-2)
    want = torch.linalg.inv(d)
    # n * 2^-24 times the condition number bounds the error of a Cholesky inverse, relative to the largest entry
    cond = torch.linalg.cond(d).item()
    assert (got.double() - want).abs().max() <= 4 * max(n, 8) * 2.0 ** -24 * cond * want.abs().max()
    assert torch.equal(a, before)
    ops.check_status()


@pytest.mark.parametrize('n', [1537, 1601, 2000, 2001, 2100, 2101, 2177])
def test_factors_of_about_as_many_tiles_as_sms(n):
    """Both sides of the rule that launches products of unaligned outputs plainly, and the CTAs of one wave and a little more."""
    x = torch.randn(70, n, device=DEV, generator=_gen(16)).to(torch.bfloat16)
    want = x.double().T @ x.double()
    out = torch.eye(n, device=DEV)
    for turn in (1, 2):
        ops.gram(x, out=out, beta=0.5)
        assert (out.double() - want - 0.5 * (torch.eye(n, device=DEV) if turn == 1 else before)).abs().max() <= 1e-6 * want.abs().max()
        before = out.clone()
    ops.check_status()


@pytest.mark.parametrize('m,n', [(129, 129), (256, 300), (257, 640), (1000, 520)])
@pytest.mark.parametrize('k', [2, 64, 200, 1600])
def test_bf16x3_products_on_pairs(m, n, k):
    """Odd and even counts of 128-row tiles, ragged edges, one K block, several K ranges, operands of either order, hi and lo images."""
    a, b = torch.randn(k, m, device=DEV, generator=_gen(1)), torch.randn(k, n, device=DEV, generator=_gen(2))
    (ah, al), (bh, bl) = ops._stage_bf16(a, True), ops._stage_bf16(b, True)
    (akh, akl), (bkh, bkl) = ops._stage_bf16(a.T.contiguous(), True), ops._stage_bf16(b.T.contiguous(), True)
    want = a.double().T @ b.double()
    # 2^-16 of each product from the bf16 pairs, fp32 sums
    bound = (a.abs().double().T @ b.abs().double()) * (2.0 ** -15 + k * 2.0 ** -24) + 1e-6
    for (p, pk), (q, qk) in [(((ah, al), False), ((bh, bl), False)), (((akh, akl), True), ((bkh, bkl), True))]:
        for nsplit in (0, 1, 3):
            out = torch.full((m, n), float('nan'), device=DEV)
            ops.extension().umma_gemm(list(p), list(q), pk, qk, out, 1.0, 0.0, False, None, None, nsplit, None, False, True)
            assert ((out.double() - want).abs() <= bound).all()
            hi = torch.empty(m, (n + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)
            lo = torch.empty_like(hi)
            ops.extension().umma_gemm(list(p), list(q), pk, qk, None, 1.0, 0.0, False, hi, lo, nsplit, None, False, True)
            assert ((hi[:, :n].double() + lo[:, :n].double() - want).abs() <= bound + 2.0 ** -15 * want.abs()).all()
    ops.check_status()


@pytest.mark.parametrize('shape', [(8,), (2, 8, 8)])
def test_a_two_sided_product_of_something_else_than_a_matrix_is_a_value_error(shape):
    eye = torch.eye(8, device=DEV)
    with pytest.raises(ValueError):
        ops.kron_apply(eye, torch.zeros(*shape, device=DEV), eye)


@pytest.mark.parametrize('rows', [1535, 1536, 4001])
@pytest.mark.parametrize('n', [128, 200, 256, 385, 520, 1000])
def test_fp32_factor_on_pairs(rows, n):
    """Both sides of the rule that takes a symmetric bf16x3 product to CTA pairs, also while a batch is recorded."""
    x = torch.randn(rows, n, device=DEV, generator=_gen(5))
    before = torch.eye(n, device=DEV)
    want = x.double().T @ x.double() / rows + 0.5 * before.double()
    bound = 2.0 ** -15 + 3 * rows * 2.0 ** -24 + 1e-6
    out = before.clone()
    ops.gram(x, scale=1 / rows, out=out, beta=0.5)
    assert (out.double() - want).abs().max() <= bound * want.abs().max() and torch.equal(out, out.T)
    out = before.clone()
    ops.extension().gemm_batch_begin()
    ops.gram(x, scale=1 / rows, out=out, beta=0.5)
    ops.extension().gemm_batch_end()
    assert (out.double() - want).abs().max() <= bound * want.abs().max() and torch.equal(out, out.T)
    ops.check_status()


def test_batches_whose_tables_take_each_others_place(ext):
    """Problem tables of one batch after another lie at the same address and hold other tensor maps."""
    for turn in range(6):
        n = 64 + 72 * turn
        xs = [torch.randn(300 + 50 * i, n, device=DEV, generator=_gen(10 * turn + i)).to(torch.bfloat16) for i in range(8)]
        outs = [torch.empty(n, n, device=DEV) for _ in xs]
        ext.gemm_batch_begin()
        for x, out in zip(xs, outs):
            ops.gram(x, out=out)
        ext.gemm_batch_end()
        del x
        for x, out in zip(xs, outs):
            want = x.double().T @ x.double()
            # products of bf16 values are exact in fp32; the sums are not
            assert (out.double() - want).abs().max() <= x.shape[0] * 2.0 ** -24 * want.abs().max()
    ops.check_status()


@pytest.mark.parametrize('kernel,padding', [((3, 3), (1, 1)), ((3, 3), (0, 0)), ((5, 5), (2, 2)), ((5, 5), (0, 0)), ((5, 5), (1, 0)),
                                            ((4, 3), (1, 2)), ((2, 2), (1, 0))])
@pytest.mark.parametrize('shape', [(1, 64, 7, 7), (3, 24, 9, 6), (70, 65, 8, 8), (2, 192, 12, 13), (5, 128, 10, 10)])
@pytest.mark.parametrize('dtype,layout', [(torch.float32, 'nchw'), (torch.bfloat16, 'nhwc'), (torch.float16, 'view')])
def test_factor_by_tap_differences(kernel, padding, shape, dtype, layout):
    """One, two and more chunks of channels, ragged ones, windows that cut both sides of the image, both column orders."""
    n, c, h, w = shape
    x = torch.randn(n, c + 1, h, w + 2, device=DEV, generator=_gen(3)).to(dtype)[:, 1:, :, 1:-1]
    if layout != 'view':
        x = x.contiguous(memory_format=torch.channels_last if layout == 'nhwc' else torch.contiguous_format)
    taps = kernel[0] * kernel[1]
    x3 = dtype == torch.float32
    seen = (x if x3 else x.to(torch.bfloat16)).double()
    patches = F.unfold(seen, kernel, padding=padding).transpose(1, 2).reshape(-1, c * taps)
    for khwc in (True, False):
        m = patches.view(-1, c, taps).transpose(1, 2).reshape(patches.shape) if khwc else patches
        before = torch.randn(c * taps, c * taps, device=DEV, generator=_gen(4))
        before += before.T.clone()
        out = torch.full((c * taps, c * taps + 3), 2.0, device=DEV)[:, :c * taps]   # rows of any alignment
        out.copy_(before)
        done = ops.extension().conv_gram(x, out, *kernel, *padding, 1 / n, 0.5, khwc, x3)
        # no plan where an image row or column would be among the first and among the last that a window leaves out
        assert done == (h >= 2 * (kernel[0] - 1 - padding[0]) and w >= 2 * (kernel[1] - 1 - padding[1]))
        if not done:
            assert torch.equal(out, before)
            return
        want = m.T @ m / n + 0.5 * before.double()
        # 2^-16 of a product of bf16 pairs (exact ones for bf16) and an ulp for every sixteen rows of a sum; the products of an entry
        # add up to at most the root of its two diagonal entries
        energy = m.square().sum(0).sqrt() / n ** 0.5
        bound = ((2.0 ** -15 + 3 / 16 * len(m) * 2.0 ** -23 if x3 else 1 / 16 * len(m) * 2.0 ** -23) + 2.0 ** -20) * torch.outer(energy, energy) + 2.0 ** -22 * before.abs()
        assert ((out.double() - want).abs() <= bound).all()
        assert torch.equal(out, out.T)
        got = ops.extension().conv_gram(x, out, *kernel, *padding, 1 / n, 0.0, khwc, x3)
        assert got and ((out.double() - m.T @ m / n).abs() <= bound).all()
    ops.check_status()


@pytest.mark.parametrize('dtype,last', [(torch.float32, False), (torch.bfloat16, True)])
def test_a_factor_of_one_image_row_has_the_zeros_and_signs_of_a_gram_matrix(ext, dtype, last):
    """Taps whose window leaves the only non-zero row out have exact zeros, and no diagonal entry is negative."""
    x = torch.zeros(4, 64, 12, 12, device=DEV)
    x[:, :, -1] = 100 * torch.randn(4, 64, 12, device=DEV, generator=_gen(11))
    x = x.to(dtype)
    out = torch.full((576, 576), float('nan'), device=DEV)
    assert ext.conv_gram(x, out, 3, 3, 1, 1, 1.0, 0.0, last, dtype == torch.float32)
    taps = out if last else out.view(64, 9, 64, 9).permute(1, 0, 3, 2).reshape(576, 576)
    assert (taps[:192] == 0).all() and (taps[:, :192] == 0).all()
    assert (out.diagonal() >= 0).all() and (taps.diagonal()[192:] > 0).all()


@pytest.mark.parametrize('at', [(0, 0), (5, 0), (11, 7), (6, 6)])
@pytest.mark.parametrize('value', [float('inf'), float('nan')])
def test_a_value_that_is_not_finite_stays_in_its_channel(ext, at, value):
    """Taps that see the value have diagonal entries that are not finite, and other channels have what they have without it."""
    x = torch.randn(3, 70, 12, 12, device=DEV, generator=_gen(12))
    clean, out = torch.empty(630, 630, device=DEV), torch.empty(630, 630, device=DEV)
    ext.conv_gram(x, clean, 3, 3, 1, 1, 1.0, 0.0, False, True)
    x[1, 20, at[0], at[1]] = value
    ext.conv_gram(x, out, 3, 3, 1, 1, 1.0, 0.0, False, True)
    seen = ~F.unfold(x, 3, padding=1).isfinite().all(2).all(0)
    assert 4 <= seen.sum() <= 9 and not out.diagonal()[seen].isfinite().any()
    others = torch.arange(630, device=DEV) // 9 != 20
    assert torch.equal(out[others][:, others], clean[others][:, others])


@pytest.mark.parametrize('shape,k', [((32, 96, 32, 32), 5), ((32, 256, 28, 28), 3), ((16, 130, 30, 31), 5)])
def test_long_sums_of_fp32_factors_by_tap_differences(ext, shape, k):
    """K ranges of hundreds of blocks: the tensor core truncates with each of its additions of 16 rows."""
    n, c, h, w = shape
    x = torch.relu(torch.randn(*shape, device=DEV, generator=_gen(17)))
    out = torch.empty(c * k * k, c * k * k, device=DEV)
    assert ext.conv_gram(x, out, k, k, k // 2, k // 2, 1.0, 0.0, False, True)
    want = torch.zeros(c * k * k, c * k * k, device=DEV, dtype=torch.float64)
    for part in x.split(4):
        m = F.unfold(part.double(), k, padding=k // 2).transpose(1, 2).reshape(-1, c * k * k)
        want += m.T @ m
    (_, _, n_grids, *_), words, _ = ext.conv_gram_plan(n, c, h, w, k, k, k // 2, k // 2, torch.cuda.get_device_properties(0).multi_processor_count, True)
    blocks = max(-(-words[8 * g + 2] // words[8 * g + 3]) for g in range(n_grids))
    # 2^-16 of a product, and half a last bit of half the sum, on average, for each addition to the large accumulator; a third accumulating
    # product in it would be three times that
    assert (out - want).norm() <= (2.0 ** -16 + 4 * blocks * 2.0 ** -25) * want.norm()


@pytest.mark.parametrize('rows,n', [(60000, 2048), (20000, 1100)])
def test_long_sums_of_fp32_factors_on_pairs(rows, n):
    x = torch.randn(rows, n, device=DEV, generator=_gen(18))
    want = x.double().T @ x.double()
    # 2^-16 of a product, and a last bit of half the sum for each of the additions of a range of 256 K blocks
    assert (ops.gram(x) - want).norm() <= (2.0 ** -16 + 4 * 256 * 2.0 ** -24) * want.norm()


@pytest.mark.parametrize('k', [3, 5])
def test_a_captured_factor_by_tap_differences_replays_on_new_inputs(ext, k):
    """Tables that are kernel parameters (3 x 3) and tables that a kernel writes first (5 x 5)."""
    x = torch.randn(4, 64, 16, 16, device=DEV, generator=_gen(13))
    out, want = (torch.zeros(64 * k * k, 64 * k * k, device=DEV) for _ in range(2))
    args = (k, k, k // 2, k // 2, 1.0, 0.0, False, True)
    ext.conv_gram(x, out, *args)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):
            ext.conv_gram(x, out, *args)
    for seed in (14, 15):
        x.copy_(torch.randn(4, 64, 16, 16, device=DEV, generator=_gen(seed)))
        ext.conv_gram(x, want, *args)
        out.fill_(float('nan'))
        graph.replay()
        assert torch.equal(out, want)
    ops.check_status()


def test_a_refused_factor_by_tap_differences_launches_nothing(ext):
    """5 x 5 filters have tables that a kernel writes first; a refused call stops ahead of it."""
    x, out = torch.zeros(2, 8, 9, 9, device=DEV, dtype=torch.float64), torch.zeros(200, 200, device=DEV)
    before = ext.launch_count()
    with pytest.raises(RuntimeError, match='fp32, bf16 or fp16'):
        ext.conv_gram(x, out, 5, 5, 2, 2, 1.0, 0.0, True, False)
    assert ext.launch_count() == before


def test_the_rule_for_tap_differences_gives_what_patches_give(monkeypatch):
    for shape, k, p, mode, dtype in [((4, 64, 7, 7), 3, 1, 'zeros', torch.float32), ((8, 32, 16, 16), 3, 1, 'reflect', torch.float32),
                                     ((32, 64, 14, 14), 5, 2, 'zeros', torch.bfloat16), ((4, 128, 9, 9), 3, 0, 'zeros', torch.bfloat16)]:
        x = torch.randn(*shape, device=DEV, generator=_gen(8)).to(dtype)
        last = dtype == torch.bfloat16
        x = x.contiguous(memory_format=torch.channels_last) if last else x
        conv = torch.nn.Conv2d(shape[1], 4, k, padding=p, padding_mode=mode, bias=False).to(DEV)
        with monkeypatch.context() as m:
            m.setattr(ops, 'tap_difference_eligible', lambda *args: True)   # whatever is the faster one
            got = ops.conv_patch_gram(x, conv, scale=1e-3, channels_last_order=last)
            m.setattr(ops, 'tap_difference_eligible', lambda *args: False)
            want = ops.conv_patch_gram(x, conv, scale=1e-3, channels_last_order=last)
        assert (got - want).norm() <= (4e-5 if dtype == torch.float32 else 5e-6) * want.norm()


@pytest.mark.parametrize('threshold,implicit', [(None, False), (0.0, True), (64.0, True), (63.9, True), (200.0, False)])
def test_a_threshold_that_is_set_asks_for_implicit_im2col(ext, monkeypatch, threshold, implicit):
    """110 MiB of patches, which both ways can take: a number asks for one of them, also the number that holds by default."""
    conv = torch.nn.Conv2d(64, 8, 3, padding=1, bias=False).to(DEV)
    x = torch.randn(32, 64, 56, 56, device=DEV, generator=_gen(9)).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    monkeypatch.setattr(ops, 'IMPLICIT_IM2COL_MIN_MB', threshold)
    monkeypatch.setattr(ops, 'TAP_DIFFERENCES', True)
    before = ext.launch_count()
    ops.conv_patch_gram(x, conv, channels_last_order=True)
    assert (ext.launch_count() - before <= 2) == implicit   # the product and its split-K reduction


@pytest.mark.parametrize('sizes', [(1, 128, 129, 256, 384, 385), (640, 8, 513, 64, 257, 191, 1), (1153, 1024), (130,) * 90 + (400,) * 40])
def test_grouped_inverse_of_mixed_sizes(sizes):
    """Tiles at and past the edges, chains of several lengths side by side, more tasks than CTAs; inputs with a row pitch."""
    mats, damp = [], torch.rand(len(sizes), device=DEV, generator=_gen(6)) * 1e-2 + 1e-2
    for i, n in enumerate(sizes):
        x = torch.randn(2 * n, n, device=DEV, generator=_gen(30 + i))
        wide = torch.full((n, n + 1 + i % 3), float('nan'), device=DEV)
        wide[:, :n] = x.T @ x / (2 * n)
        mats.append(wide[:, :n])
    outs = [torch.full((n, n), float('nan'), device=DEV) for n in sizes]
    for _ in range(3):
        ops.spd_inverse_grouped(mats, outs, damp)
    ops.check_status()
    for m, o, d, n in zip(mats, outs, damp, sizes):
        want = m.double()
        want.diagonal().add_(d.double())
        cond = torch.linalg.cond(want).item()
        want = torch.linalg.inv(want)
        # n * 2^-24 times the condition number bounds the error of a Cholesky inverse, relative to the largest entry
        assert (o.double() - want).abs().max() <= 4 * max(n, 8) * 2.0 ** -24 * cond * want.abs().max()
        assert torch.equal(o, o.T)


def test_a_set_of_small_inverses_keeps_one_tile_for_each(ext):
    """Up to 128 rows there is nothing below the diagonal: three 32 KiB parts of the inverse's factor, and the tables."""
    ext.chol_inverse_tc_clear_cache()
    mats = [torch.eye(10, device=DEV) * (i + 1) for i in range(200)]
    outs = [torch.empty_like(m) for m in mats]
    damp = torch.zeros(200, device=DEV)
    ext.read_status(0)
    before = torch.cuda.memory_allocated()
    ext.chol_inverse_tc(mats, outs, damp)
    assert torch.cuda.memory_allocated() - before <= 200 * (96 * 1024 + 512) + 4096
    for i, out in enumerate(outs):
        assert (out - torch.eye(10, device=DEV) / (i + 1)).abs().max() <= 2.0 ** -21
    ops.check_status()
    ext.chol_inverse_tc_clear_cache()


@pytest.mark.parametrize('n,at', [(40, 35), (128, 0), (128, 100), (200, 150)])
def test_a_negative_pivot_in_any_stage_is_reported(n, at):
    a = torch.eye(n, device=DEV)
    a[at, at] = -1.0
    got = ops.spd_inverse(a, 0.0)
    with pytest.raises(RuntimeError, match='not positive definite'):
        ops.check_status()
    assert torch.isfinite(got).all()


@pytest.mark.parametrize('d', [256, 512, 768, 1024, 1536, 2048, 4096])
@pytest.mark.parametrize('rows', [1, 7, 148 * 8 + 1, 148 * 16 + 5])
def test_layer_norm_backward_rows(rows, d):
    x = torch.randn(rows, d, device=DEV, generator=_gen(10)).to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(rows, d, device=DEV, generator=_gen(11)).to(torch.bfloat16)
    weight = (1 + 0.1 * torch.randn(d, device=DEV, generator=_gen(12))).requires_grad_(True)
    bias = torch.randn(d, device=DEV, generator=_gen(13)).requires_grad_(True)
    got = torch.autograd.grad(ops.layer_norm(x, weight, bias), [x, weight, bias], dy)
    leaves = [t.detach().double().requires_grad_(True) for t in (x, weight, bias)]
    want = torch.autograd.grad(F.layer_norm(leaves[0], (d,), leaves[1], leaves[2]), leaves, dy.double())
    assert ((got[0].double() - want[0]).abs() <= 2.0 ** -8 * want[0].abs() + 1e-4).all()   # bf16 result, fp32 row sums
    for a, b in zip(got[1:], want[1:]):   # fp32 sums of `rows` terms of size ~ 1: at most rows * 2^-24 of sqrt(rows) * few
        assert (a.double() - b).abs().max() <= 1e-5 * max(1.0, rows ** 0.5) + 1e-5


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('rows,d', [(1, 8), (31, 64), (33, 72), (700, 12), (3001, 1024), (257, 1001), (5000, 256)])
def test_layer_norm_curvature_chunks(dtype, rows, d):
    y = torch.randn(rows, d, device=DEV, generator=_gen(14)).to(dtype)
    g = torch.randn(rows, d, device=DEV, generator=_gen(15)).to(dtype)
    weight = 1 + 0.1 * torch.randn(d, device=DEV, generator=_gen(16))
    bias = 0.1 * torch.randn(d, device=DEV, generator=_gen(17))
    gw, gb = (y.double() - bias.double()) / weight.double() * g.double(), g.double()
    want = torch.stack([torch.stack([(gw * gw).sum(0), (gw * gb).sum(0)], 1),
                        torch.stack([(gw * gb).sum(0), (gb * gb).sum(0)], 1)], 1)
    size = torch.stack([torch.stack([(gw * gw).sum(0), (gw * gb).abs().sum(0)], 1),
                        torch.stack([(gw * gb).abs().sum(0), (gb * gb).sum(0)], 1)], 1)
    old = torch.randn(d, 2, 2, device=DEV, generator=_gen(18))
    got = ops.layernorm_unitwise_stats(y, g, weight, bias, out=old.clone(), alpha=0.5, beta=0.25)
    # a few fp32 roundings per term and a sum of at most 64 per lane before double precision takes over
    assert ((got.double() - (0.25 * old.double() + 0.5 * want)).abs() <= 64 * 2.0 ** -24 * size + 1e-6).all()


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('rows,d', [(1, 16384), (112, 64), (113, 64), (999, 512), (1000, 512), (1031, 72), (513, 16384)])
def test_layer_norm_curvature_rows(dtype, rows, d):
    test_layer_norm_curvature_chunks(dtype, rows, d)


@pytest.mark.parametrize('relu,residual', [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize('n,c,h,w', [(2, 8, 1, 1), (3, 16, 5, 7), (1, 2056, 3, 3), (5, 264, 11, 9), (16, 64, 40, 40)])
def test_batch_norm_row_walk(n, c, h, w, relu, residual):
    def act(seed):
        return torch.randn(n, c, h, w, device=DEV, generator=_gen(seed)).to(torch.bfloat16).contiguous(
            memory_format=torch.channels_last)
    x, dy, res = act(5).requires_grad_(True), act(6), act(7).requires_grad_(True) if residual else None
    weight = (1 + 0.1 * torch.randn(c, device=DEV, generator=_gen(8))).requires_grad_(True)
    bias = (0.1 * torch.randn(c, device=DEV, generator=_gen(9))).requires_grad_(True)
    y = ops.batch_norm_train(x, weight, bias, None, None, residual=res, relu=relu)
    grads = torch.autograd.grad(y, [x, weight, bias] + ([res] if residual else []), dy)
    xd, wd, bd = (t.detach().double().requires_grad_(True) for t in (x, weight, bias))
    rd = res.detach().double().requires_grad_(True) if residual else None
    pre = F.batch_norm(xd, None, None, wd, bd, training=True)
    pre = pre + rd if residual else pre
    yd = pre * (y > 0) if relu else pre        # the mask of the stored output: a value may round to zero
    want = torch.autograd.grad(yd, [xd, wd, bd] + ([rd] if residual else []), dy.double())
    # bf16 results: 2^-8 of the value; of the largest value where terms cancel (y near 0, dx of two rows)
    for got, ref in zip((y,) + grads, (yd,) + want):
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * (ref.abs() + ref.abs().max()) + 1e-5).all()


@pytest.mark.parametrize('relu,residual', [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize('n,c,h,w', [(1, 8, 1, 384), (1, 136, 1, 385), (2, 72, 3, 64), (1, 24, 7, 55), (1, 40, 16, 32), (3, 16, 19, 27)])
def test_batch_norm_rows_around_a_ring(n, c, h, w, relu, residual):
    """12 rows per lane fill the ring of the forward pass, 6 that of the backward pass; 512 rows are one split."""
    test_batch_norm_row_walk(n, c, h, w, relu, residual)


@pytest.mark.parametrize('c', [8, 72])
def test_batch_norm_mask_of_special_values(c):
    """The gradient passes where the stored output is above zero: not at zeros of either sign, nor where it is NaN."""
    values = torch.tensor([0.0, -0.0, 1.0, -1.0, float('inf'), float('-inf'), float('nan'), 2.0 ** -133], device=DEV)
    res = values.repeat(64 * c // 8 * 3)[:64 * c].view(1, 64, 1, c).roll(1, 1).permute(0, 3, 1, 2).to(torch.bfloat16).requires_grad_(True)
    x = torch.zeros_like(res)                  # normalised to zeros: the output is the ReLU of the residual
    y = ops.batch_norm_train(x, torch.ones(c, device=DEV), torch.zeros(c, device=DEV), residual=res, relu=True)
    dy = torch.randn_like(y)
    grad, = torch.autograd.grad(y, res, dy)
    assert torch.equal(y.float(), torch.nan_to_num(res.detach().float(), posinf=float('inf'), neginf=0.0).clamp(min=0))
    assert torch.equal(grad, torch.where(y > 0, dy, torch.zeros_like(dy)))


@pytest.mark.parametrize('padding', [0, 1])
@pytest.mark.parametrize('n,c,h,w', [(2, 64, 17, 18), (1, 8, 3, 3), (3, 24, 16, 33), (2, 264, 15, 40), (1, 16, 32, 4)])
def test_max_pool_gives_the_bits_of_pytorch(padding, n, c, h, w):
    kernel, stride = 3, 2
    pool = FusedMaxPool2d(kernel, stride=stride, padding=padding)
    x = torch.randn(n, c, h, w, device=DEV, generator=_gen(32)).mul_(2).round_().to(torch.bfloat16)   # many equal values
    x.view(-1)[::97] = float('nan')
    x.view(-1)[::61] = float('-inf')
    x[0, :, :8, :8] = float('-inf')   # whole windows
    x = x.contiguous(memory_format=torch.channels_last).requires_grad_(True)
    assert pool._native(x)
    y, want = pool(x), F.max_pool2d(x, kernel, stride, padding)
    assert y.shape == want.shape and y.is_contiguous(memory_format=torch.channels_last)
    assert torch.equal(y.nan_to_num(nan=1e4), want.nan_to_num(nan=1e4))
    dy = torch.randn_like(want)
    got, ref = torch.autograd.grad(y, x, dy, retain_graph=True)[0], torch.autograd.grad(want, x, dy)[0]
    assert torch.equal(got, ref)
    # twice differentiable: the second pass is the gather of what the first one scatters
    g = dy.clone().requires_grad_(True)
    back, = torch.autograd.grad(y, x, g, create_graph=True)
    v = torch.randn_like(back)
    again, = torch.autograd.grad(back, g, v)
    _, where = F.max_pool2d(x.detach(), kernel, stride, padding, return_indices=True)
    assert torch.equal(again, v.flatten(2).gather(2, where.flatten(2)).view_as(again))


@pytest.mark.parametrize('m,n', [(1, 1), (2, 1), (129, 1), (1, 2), (2, 2), (8, 8), (7, 9), (1, 300), (129, 2049), (640, 24)])
def test_two_sided_product_stages_its_operands_together(m, n):
    """Pitches that are padded or not, rows that are aligned or not, strided and transposed operands."""
    def spd(k, seed):
        x = torch.randn(2 * k, k, device=DEV, generator=_gen(seed))
        return x.T @ x / (2 * k)
    left, right = spd(m, 50), spd(n, 51)
    for mid in (torch.randn(m, n, device=DEV, generator=_gen(52)), torch.randn(n, m, device=DEV, generator=_gen(53)).T,
                torch.randn(m, 2 * n + 1, device=DEV, generator=_gen(54))[:, 1::2], torch.randn(m, n + 3, device=DEV, generator=_gen(55))[:, 3:]):
        want = left.double() @ mid.double() @ right.double()
        for r in (right, right.T.contiguous().T):
            got = ops.kron_apply(left, mid, r)
            # hi and lo parts carry 2^-16 of every operand of the two products
            assert (got.double() - want).norm() <= 4 * 2.0 ** -16 * want.norm()


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('rows', [1, 7, 200])
def test_one_column_of_any_stride(rows, dtype):
    """contiguous() returns a column as it is, whatever the stride of its columns."""
    wide = torch.randn(rows, 5, device=DEV, generator=_gen(56)).to(dtype)
    other = torch.randn(rows, 3, device=DEV, generator=_gen(57)).to(dtype)
    for x in (wide.T.contiguous().T[:, :1], wide[:, 1::5], wide[:, 3:]):
        x = x[:, :1]
        want, bound = x.double().T @ x.double(), 2.0 ** -15 * x.double().square().sum()   # hi and lo parts carry 2^-16 of every operand
        assert ((ops.gram(x).double() - want).abs() <= bound).all()
        with torch.no_grad():
            got, ref = ops.matmul_tn(x, other).double(), x.double().T @ other.double()
        assert ((got - ref).abs() <= 2.0 ** -15 * x.double().norm() * other.double().norm(dim=0)).all()
        if dtype == torch.float32:
            assert torch.equal(sum(p.float() for p in ops.split3(x)), x)
            one = torch.ones(1, 1, device=DEV).T
            assert (ops.kron_apply(torch.eye(rows, device=DEV), x, one).double() - x.double()).norm() <= 2.0 ** -14 * x.double().norm()


@pytest.mark.parametrize('up', [False, True])
def test_casts_of_many_tensors(up):
    """Sizes around a vector and a piece of 8192, layouts that are alike or not, unaligned views, more tensors than a table holds."""
    src_type, dst_type = (torch.bfloat16, torch.float32) if up else (torch.float32, torch.bfloat16)
    shapes = [(1,), (7,), (8,), (8191,), (8192,), (8193,), (3, 5, 7, 9), (64, 16, 1, 1), (0, 4), (40, 24, 3, 3), (100, 300)]
    src, dst = [], []
    for i, shape in enumerate(shapes * 13):
        s = torch.randn(shape, device=DEV, generator=_gen(40 + i)).to(src_type)
        if len(shape) == 4 and i % 2:
            s = s.contiguous(memory_format=torch.channels_last)
        if i % 5 == 4:   # a base that is not 16-byte aligned
            s = torch.cat([s.new_zeros(1), s.flatten()])[1:].view(shape)
        d = torch.full(shape, float('nan'), device=DEV, dtype=dst_type)
        if len(shape) == 4 and i % 3:
            d = d.contiguous(memory_format=torch.channels_last)
        if len(shape) == 2 and i % 7 == 3:
            s = s.T.contiguous().T
        src.append(s)
        dst.append(d)
    src.append(torch.arange(9, device=DEV, dtype=torch.float32))
    dst.append(torch.zeros(9, device=DEV, dtype=torch.float64))
    ops.extension().cast_many(dst, src)
    for s, d in zip(src, dst):
        assert torch.equal(d, s.to(d.dtype))


@pytest.mark.parametrize('scale', [1.0, -0.375])
@pytest.mark.parametrize('count', [1, 3, 64, 131])
def test_stage_gradients(ext, count, scale):
    shapes = [(1, 1), (64, 3, 7, 7), (37, 65), (130, 8), (3, 2056), (5, 24, 3, 3), (2, 16, 1, 1), (700, 40)]
    grads, staged, want = [], [], []
    for i in range(count):
        shape = shapes[i % len(shapes)]
        numel = torch.Size(shape).numel()
        rows, last = shape[0], i % 3 == 1 and len(shape) == 4                 # in the factor's order, or copied into it
        fmt = torch.channels_last if len(shape) == 4 else torch.contiguous_format
        v = torch.zeros(shape, device=DEV).contiguous(memory_format=fmt)
        flat = torch.randn(numel + 1, device=DEV, generator=_gen(i))[i % 2:i % 2 + numel]   # on and off 16 bytes
        if last or len(shape) == 2:
            g = flat.view(shape)
        else:
            g = flat.as_strided(v.shape, v.stride())
        grads.append(g.half() if i % 11 == 10 else g)
        staged.append(v)
        x = grads[-1].float().mul(scale)
        want.append((x.permute(0, 2, 3, 1) if len(shape) == 4 else x).reshape(rows, -1))
    hi, lo = ([torch.full((w.shape[0], (w.shape[1] + 7) // 8 * 8), 9.0, device=DEV, dtype=torch.bfloat16) for w in want] for _ in range(2))
    kept = [g.clone() for g in grads]
    ext.stage_gradients(grads, staged, hi, lo, scale)
    for w, h, l, g, k in zip(want, hi, lo, grads, kept):
        w = F.pad(w, (0, h.shape[1] - w.shape[1]))
        assert torch.equal(h, w.bfloat16()) and torch.equal(l, (w - w.bfloat16().float()).bfloat16())
        assert torch.equal(g, k)


@pytest.mark.parametrize('n', [1, 31, 33, 511, 513, 1000, 1031])
def test_bias_products(ext, n):
    inverse, bias, scratch = (torch.randn(shape, device=DEV, generator=_gen(n)) for shape in ((n, n), (n,), (n,)))
    want = 0.5 * (inverse.double() @ bias.double())
    bound = 0.5 * (inverse.double().abs() @ bias.double().abs()) * (n / 32 + 7) * 2.0 ** -24   # a lane's chain, then the lanes' sums
    ext.bias_precondition_mt([[inverse.data_ptr(), bias.data_ptr(), scratch.data_ptr(), n]], 0.5)
    assert bool(((bias.double() - want).abs() <= bound).all())


def test_max_pool_takes_gradients_at_any_address():
    x = torch.randn(2, 8, 9, 9, device=DEV, generator=_gen(33)).to(torch.bfloat16).contiguous(memory_format=torch.channels_last).requires_grad_(True)
    y, want = FusedMaxPool2d(3, stride=2, padding=1)(x), F.max_pool2d(x, 3, 2, 1)
    dy = torch.randn(y.numel() + 1, device=DEV, generator=_gen(34)).to(torch.bfloat16)[1:].view(2, 5, 5, 8).permute(0, 3, 1, 2)
    assert dy.data_ptr() % 16 and dy.is_contiguous(memory_format=torch.channels_last)
    assert torch.equal(torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(want, x, dy)[0])


def test_max_pool_gradients_that_pytorch_has_to_look_into():
    """Batches of gradients, gradients with a tangent, negative views: the results of the parent."""
    x = torch.randn(2, 8, 9, 9, device=DEV, generator=_gen(35)).to(torch.bfloat16).contiguous(memory_format=torch.channels_last).requires_grad_(True)
    y, want = FusedMaxPool2d(3, stride=2, padding=1)(x), F.max_pool2d(x, 3, 2, 1)
    dy, tangent = (torch.randn_like(want) for _ in range(2))

    def back(out, g, **options):
        return torch.autograd.grad(out, x, g, retain_graph=True, **options)[0]

    batch = torch.stack([dy, tangent])
    assert torch.equal(back(y, batch, is_grads_batched=True), back(want, batch, is_grads_batched=True))
    assert torch.equal(torch.func.vmap(lambda g: back(y, g))(batch), torch.func.vmap(lambda g: back(want, g))(batch))
    assert torch.equal(back(y, torch._neg_view(dy)), back(want, -dy))
    ad = torch.autograd.forward_ad
    with ad.dual_level():
        got, ref = (ad.unpack_dual(back(out, ad.make_dual(dy, tangent))) for out in (y, want))
        assert torch.equal(got.primal, ref.primal) and torch.equal(got.tangent, ref.tangent)


def test_max_pool_gradient_has_a_derivative_of_zeros_by_the_input():
    """As nn.MaxPool2d's, also where the gradient that comes in does not require one."""
    x = torch.randn(2, 8, 9, 9, device=DEV, generator=_gen(37)).to(torch.bfloat16).contiguous(memory_format=torch.channels_last).requires_grad_(True)
    for y in (FusedMaxPool2d(3, stride=2, padding=1)(x), F.max_pool2d(x, 3, 2, 1)):
        dx, = torch.autograd.grad(y.sum(), x, create_graph=True)
        assert dx.requires_grad
        again, = torch.autograd.grad((dx * dx).sum(), x)
        assert torch.equal(again, torch.zeros_like(x))
    y = FusedMaxPool2d(3, stride=2, padding=1)(x)
    with torch.no_grad():
        x.mul_(2)
    with pytest.raises(RuntimeError, match='inplace'):   # the input is saved
        y.sum().backward()


def test_max_pool_leaves_tensors_without_memory_to_pytorch():
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        x = torch.empty(2, 8, 9, 9, device=DEV, dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last)
        assert FusedMaxPool2d(3, stride=2, padding=1)(x).shape == (2, 8, 5, 5)


def _norm_calls():
    def act(*shape):
        return torch.randn(*shape, device=DEV, generator=_gen(30)).to(torch.bfloat16)
    x, res = (act(4, 16, 5, 5).contiguous(memory_format=torch.channels_last).requires_grad_(True) for _ in range(2))
    weight, bias = (torch.rand(16, device=DEV, generator=_gen(31)).requires_grad_(True) for _ in range(2))
    wide, gain, shift = act(6, 256).requires_grad_(True), torch.ones(256, device=DEV).requires_grad_(True), torch.zeros(256, device=DEV)
    return [(lambda x, w, b: ops.batch_norm_train(x, w, b, relu=True), (x, weight, bias)),
            (lambda x, w, b, r: ops.batch_norm_train(x, w, b, residual=r, relu=True), (x, weight, bias, res)),
            (lambda x, w, b, r: ops.batch_norm_train(x, w, b, residual=r), (x, weight, bias, res)),
            (lambda x, w, b: ops.layer_norm(x, w, b), (wide, gain, shift))]


@pytest.mark.parametrize('which', range(4))
def test_native_norm_functions_keep_the_rules_of_autograd(which):
    fn, args = _norm_calls()[which]
    leaves = [a for a in args if a.requires_grad]
    y = fn(*args)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy)
    # saved tensors go through hooks, and are gone after the first pass
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or len(packed) - 1, lambda i: packed[i].clone()):
        y2 = fn(*args)
    assert packed
    for a, b in zip(torch.autograd.grad(y2, leaves, dy), want):
        assert torch.equal(a, b)
    with pytest.raises(RuntimeError, match='second time'):
        torch.autograd.grad(y2, leaves, dy)
    # a trace runs the kernels again instead of returning what its allocations hold
    if which < 3:   # sizes are tensors in a trace, so that a LayerNorm goes to PyTorch's, which refuses bf16 with fp32 parameters
        traced = torch.jit.trace(fn, tuple(a.detach() for a in args), check_trace=False)
        assert torch.equal(traced(*(2 * a.detach() for a in args)), fn(*(2 * a.detach() for a in args)))
    # transforms that a kernel has no rule for are refused
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda x: fn(x, *args[1:]).float().sum())(args[0])
    with pytest.raises(RuntimeError), torch.autograd.forward_ad.dual_level():
        fn(torch.autograd.forward_ad.make_dual(args[0].detach(), torch.ones_like(args[0])), *args[1:])
    with torch.no_grad():
        assert not fn(*args).requires_grad and torch.equal(fn(*args), y)
    args[0].data.add_(0)   # not seen by autograd
    y3 = fn(*args)
    with torch.no_grad():
        args[0].mul_(1)
    with pytest.raises(RuntimeError, match='inplace'):
        torch.autograd.grad(y3, leaves, dy)


def test_batch_norm_with_running_statistics_that_require_a_gradient():
    """They make the output part of a graph, whose backward pass has a mask to read and no gradient for them."""
    x = torch.randn(2, 8, 5, 5, device=DEV, generator=_gen(36)).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    weight, bias, mean, var = (torch.ones(8, device=DEV) for _ in range(4))
    y = ops.batch_norm_train(x, weight, bias, mean.requires_grad_(True), var, residual=x, relu=True)
    assert y.requires_grad
    y.float().sum().backward()
    assert mean.grad is None


class _Cut(torch.autograd.Function):
    """Identity whose backward gives no gradient."""

    @staticmethod
    def forward(ctx, x):
        return x.view_as(x)

    @staticmethod
    def backward(ctx, dy):
        return None


@pytest.mark.parametrize('relu', [False, True])
def test_batch_norm_counts_an_undefined_gradient_as_zeros(relu):
    def act(seed):
        x = torch.randn(2, 16, 3, 3, device=DEV, generator=_gen(seed)).to(torch.bfloat16)
        return x.contiguous(memory_format=torch.channels_last).requires_grad_(True)
    x, res = act(22), act(23)
    weight, bias = (torch.ones(16, device=DEV, requires_grad=True) for _ in range(2))
    _Cut.apply(ops.batch_norm_train(x, weight, bias, residual=res, relu=relu)).sum().backward()
    for leaf in (x, res, weight, bias):
        assert leaf.grad is not None and not leaf.grad.any()


@pytest.mark.parametrize('masked', [False, True])
@pytest.mark.parametrize('n,c,h,w', [(600, 8, 1, 31), (600, 8, 3, 53), (600, 8, 10, 16), (600, 8, 7, 23), (600, 8, 18, 18), (3, 72, 29, 31)])
def test_batch_norm_curvature_positions(n, c, h, w, masked):
    def act(seed):
        return torch.randn(n, c, h, w, device=DEV, generator=_gen(seed)).to(torch.bfloat16).contiguous(
            memory_format=torch.channels_last)
    x, dy, y = act(24), act(25), act(26) if masked else None
    mean, invstd = (0.1 * torch.randn(c, device=DEV, generator=_gen(27)), 0.5 + torch.rand(c, device=DEV, generator=_gen(28)))
    old = torch.randn(c, 2, 2, device=DEV, generator=_gen(29))
    got = ops.batchnorm_unitwise_stats_from_input(x, dy, y, mean, invstd, old.clone(), alpha=0.5, beta=0.25)
    g = dy.double() * (y > 0) if masked else dy.double()
    terms = (x.double() - mean.double().view(1, -1, 1, 1)) * invstd.double().view(1, -1, 1, 1) * g
    sums = [terms.sum((2, 3)), g.sum((2, 3))]                                     # per sample and channel
    sizes = [terms.abs().sum((2, 3)), g.abs().sum((2, 3))]
    pairs = [(0, 0), (0, 1), (1, 0), (1, 1)]
    want = torch.stack([(sums[a] * sums[b]).sum(0) for a, b in pairs], 1).view(c, 2, 2)
    size = torch.stack([(sizes[a] * sizes[b]).sum(0) for a, b in pairs], 1).view(c, 2, 2)
    # both factors of a product lose at most 2^-24 of their absolute sum per addition: h w / 32 per lane, 32 lanes, the splits;
    # the samples add another 2^-24 each (n / 32 per lane of a warp, then five steps)
    steps = 2 * (h * w / 32 + 32 + 8) + n / 32 + 8
    assert ((got.double() - (0.25 * old.double() + 0.5 * want)).abs() <= steps * 2.0 ** -24 * size + 1e-6).all()
