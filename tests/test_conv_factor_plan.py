"""The plan of a convolution factor by tap difference (``csrc/conv_gram.cu``): which rows are staged, which products are formed of them and
which of those make up the block of two taps.  The kernels are restated here in whole numbers, so equality is exact."""
import random

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from asdl_b200.ops import _build

GRID = 8   # words: first item, first row of B, K blocks, K ranges, tiles along B, first tile, first partial tile, first slot


def _plan(n, c, h, w, kh, kw, ph, pw, x3, sms=148):
    return _build.load().conv_gram_plan(n, c, h, w, kh, kw, ph, pw, sms, x3)


def _factor(x, kh, kw, ph, pw, plan):
    """Runs a plan on x [n, c, h, w], order (kh, kw, c).  Also: every term that went into an entry, for what depends on signs."""
    n, c, h, w = x.shape
    (total, cc, n_grids, assembly, n_products, n_terms, n_tiles, split_tiles, n_partial, items), words, staged = plan
    words = np.array(words, dtype=np.int32)
    rows = np.zeros((total + 64 * 64, 64 * (cc + 1)), dtype=x.dtype)   # behind the last row and channel: the zeros of a load out of range
    at = np.array(staged).reshape(-1, 4)
    assert (np.sort(at[:, 0]) == np.arange(total)).all()   # every row is written, once
    at = at[at[:, 1] >= 0]
    rows[at[:, 0], :c] = x[at[:, 1], :, at[:, 2], at[:, 3]]
    grids = words[:(n_grids + 1) * GRID].reshape(-1, GRID)
    slot_rows = words[(n_grids + 1) * GRID:assembly]
    n_b = 2 if cc == 1 else 1
    partial = np.full((n_partial, 128, 128), np.nan)
    tiles = np.full((n_tiles, 128, 128), np.nan)
    for g, grid in enumerate(grids[:-1]):
        first, rows_b, nkb, nsplit, tiles_b, tile0, part0, slot0 = grid
        slots = slot_rows[slot0:grids[g + 1, 7]]
        for item in range(grids[g + 1, 0] - first):
            tile, split = divmod(item, nsplit)
            ia, ib = divmod(tile, tiles_b)
            kb0, kb1 = split * nkb // nsplit, (split + 1) * nkb // nsplit
            assert kb1 > kb0
            a, b = [], []
            for u in range(2):
                sa, ca = divmod(2 * ia + u, cc)
                row, ch = (slots[sa], ca) if sa < len(slots) else (rows_b, cc)
                assert row + kb0 * 64 >= 0
                a.append(rows[row + kb0 * 64:row + kb1 * 64, 64 * ch:64 * ch + 64])
                sb, cb = divmod(2 * ib + u, cc)
                row, ch = (rows_b - sb, cb) if sb < n_b else (rows_b, cc)
                assert row + kb0 * 64 >= 0
                b.append(rows[row + kb0 * 64:row + kb1 * 64, 64 * ch:64 * ch + 64])
            out = np.concatenate(a, 1).T @ np.concatenate(b, 1)
            if nsplit > 1:
                assert tile0 + tile < split_tiles
                partial[part0 + item] = out
            else:
                assert tile0 + tile >= split_tiles
                tiles[tile0 + tile] = out
    assert grids[-1, 0] == items
    for t in range(split_tiles):
        g = np.searchsorted(grids[:-1, 5], t, side='right') - 1
        _, _, _, nsplit, _, tile0, part0, _ = grids[g]
        tiles[t] = partial[part0 + (t - tile0) * nsplit:part0 + (t - tile0 + 1) * nsplit].sum(0)
    assert not np.isnan(tiles).any() and not np.isnan(partial).any()
    products = words[assembly:assembly + 3 * n_products].view(np.int16).reshape(-1, 6)
    tile0s = words[assembly:assembly + 3 * n_products].reshape(-1, 3)[:, 0]
    taps = kh * kw
    firsts = words[assembly + 3 * n_products:][:taps * (taps + 1) // 2 + 1]
    terms = words[assembly + 3 * n_products + len(firsts):].view(np.uint16)
    assert firsts[-1] == n_terms
    result = np.zeros((taps, c, taps, c))
    for t in range(taps):
        for u in range(t + 1):
            pair = t * (t + 1) // 2 + u
            for term in terms[firsts[pair]:firsts[pair + 1]]:
                assert term < n_products
                tiles_b, a0, b0 = products[term, 2:5]
                for i in range(cc):
                    for j in range(cc):
                        ca, cb = a0 + i, b0 + j
                        block = tiles[tile0s[term] + (ca >> 1) * tiles_b + (cb >> 1)][(ca & 1) * 64:, (cb & 1) * 64:]
                        ni, nj = min(64, c - 64 * i), min(64, c - 64 * j)
                        part = block[:ni, :nj]
                        if t == u and i == j:
                            assert (np.diagonal(part) >= 0).all()   # sums of squares: nothing is taken off
                        result[t, 64 * i:64 * i + ni, u, 64 * j:64 * j + nj] += part
            if t != u:
                result[u, :, t, :] = result[t, :, u, :].T
    return result.reshape(taps * c, taps * c)


def _patches(x, kh, kw, ph, pw):
    n, c = x.shape[:2]
    m = F.unfold(torch.from_numpy(x), (kh, kw), padding=(ph, pw)).numpy()
    m = m.reshape(n, c, kh * kw, -1).transpose(0, 3, 2, 1).reshape(-1, kh * kw * c)
    return m.T @ m


def _check(n, c, h, w, kh, kw, ph, pw, x3):
    plan = _plan(n, c, h, w, kh, kw, ph, pw, x3)
    assert plan
    x = np.random.default_rng(n * h + w).integers(-3, 4, (n, c, h, w)).astype(np.float64)
    assert (_factor(x, kh, kw, ph, pw, plan) == _patches(x, kh, kw, ph, pw)).all()


@pytest.mark.parametrize('kernel', [(3, 3), (5, 5), (2, 2), (4, 3), (3, 5), (1, 3), (3, 1), (5, 2)])
def test_products_by_difference_add_up_to_the_factor(kernel):
    """Every padding, images down to the smallest that a window fits, one and several images."""
    rng = random.Random(sum(kernel))
    for ph in range(kernel[0]):
        for pw in range(kernel[1]):
            for _ in range(3):
                h = rng.randint(max(1, 2 * (kernel[0] - 1 - ph), kernel[0] - 2 * ph), 10)
                w = rng.randint(max(1, 2 * (kernel[1] - 1 - pw), kernel[1] - 2 * pw), 10)
                _check(rng.choice([1, 2, 3, 9]), rng.choice([1, 2]), h, w, *kernel, ph, pw, rng.random() < 0.5)


@pytest.mark.parametrize('shape', [(1, 65, 7, 7), (2, 129, 6, 9), (70, 64, 8, 8), (3, 192, 5, 11), (130, 3, 12, 16)])
@pytest.mark.parametrize('kernel,padding', [((3, 3), (1, 1)), ((3, 3), (0, 2)), ((5, 5), (2, 2))])
def test_several_chunks_of_channels_and_k_ranges(shape, kernel, padding):
    for x3 in (False, True):
        _check(*shape, *kernel, *padding, x3)


def test_a_window_that_leaves_the_energy_out_sees_exact_zeros():
    """Only the last image row is not zero: the first tap row of a padded 3 x 3 filter never meets it."""
    x = np.zeros((3, 5, 8, 8))
    x[:, :, -1] = np.random.default_rng(1).standard_normal((3, 5, 8))
    got = _factor(x, 3, 3, 1, 1, _plan(3, 5, 8, 8, 3, 3, 1, 1, True))
    assert (got[:15, :15] == 0).all() and (np.diagonal(got) >= 0).all()


def test_shapes_that_the_tables_do_not_hold_have_no_plan():
    for shape in [(1, 8, 9, 9, 6, 3, 1, 1), (1, 8, 9, 9, 3, 3, 3, 1), (1, 8, 7, 9, 5, 3, 0, 1), (1, 5000, 9, 9, 3, 3, 1, 1),
                  (1 << 22, 8, 64, 64, 3, 3, 1, 1), (1, 8, 9, 9, 1, 1, 0, 0), (0, 8, 9, 9, 3, 3, 1, 1)]:
        assert not _plan(*shape, True)
