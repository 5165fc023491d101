"""Whole columns in one CTA (2^9 .. 2^14 words): every size, one column and enough that the blown-up copies of a
column share its CTA, blow-ups 2 and 4, in place, padded and unaligned columns; and the sizes on either side."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
P = 2**31 - 1


def _buf(cols, stride, offset=0):
    import torch
    flat = np.full(offset + cols.shape[0] * stride, 0x5A5A5A5A, dtype=np.uint32)
    flat[offset:].reshape(cols.shape[0], stride)[:, : cols.shape[1]] = cols
    return torch.from_numpy(flat.view(np.int32)).cuda()[offset:]


def _get(t, n, stride):
    return t.cpu().numpy().view(np.uint32)[: n * stride].reshape(n, stride)


@pytest.mark.parametrize("log", [8, 9, 10, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("n,blowup", [(1, 1), (3, 2), (149, 1), (80, 2), (37, 4)])
def test_interpolate_and_extend(ctx, log, n, blowup):
    import torch
    cols = np.random.default_rng(log + n).integers(0, P, size=(n, 1 << log), dtype=np.uint32)
    cols[0] = P - 1
    co, lde = torch.empty(n << log, dtype=torch.int32, device="cuda"), torch.empty(n << (log + blowup), dtype=torch.int32, device="cuda")
    ev = _buf(cols, 1 << log)
    ctx.interpolate_and_extend(ev, co, lde, log, blowup, n)
    same = _buf(cols, 1 << log)  # coefficients in place of the evaluations
    lde2 = torch.empty_like(lde)
    ctx.interpolate_and_extend(same, same, lde2, log, blowup, n)
    ext = torch.empty_like(lde)
    ctx.extend(co, ext, log, blowup, n)
    assert torch.equal(co, same) and torch.equal(lde, lde2) and torch.equal(lde, ext)
    assert np.array_equal(_get(ev, n, 1 << log), cols)
    for c in {0, n // 2, n - 1}:
        ref = oracle.interpolate(cols[c])
        assert np.array_equal(_get(co, n, 1 << log)[c], ref)
        assert np.array_equal(_get(lde, n, 2 << (log + blowup - 1))[c], oracle.extend(ref, blowup))


@pytest.mark.parametrize("log,pad,offset", [(9, 0, 1), (11, 3, 0), (13, 5, 2), (14, 1, 3), (12, 64, 0)])
def test_in_place(ctx, log, pad, offset):
    cols = np.random.default_rng(log).integers(0, P, size=(3, 1 << log), dtype=np.uint32)
    stride = (1 << log) + pad
    t = _buf(cols, stride, offset)
    ctx.interpolate(t, log, 3, stride)
    got = _get(t, 3, stride)
    for c in range(3):
        assert np.array_equal(got[c, : 1 << log], oracle.interpolate(cols[c]))
    assert (got[:, 1 << log :] == 0x5A5A5A5A).all()
    ctx.evaluate(t, log, 3, stride)
    got = _get(t, 3, stride)
    assert np.array_equal(got[:, : 1 << log], cols) and (got[:, 1 << log :] == 0x5A5A5A5A).all()


@pytest.mark.parametrize("log,blowup", [(8, 1), (9, 1), (10, 2), (11, 1), (12, 2), (13, 1), (14, 1), (14, 2), (15, 1)])
@pytest.mark.parametrize("place", ["front", "middle", "back"])
def test_evaluations_in_the_lde_buffer(ctx, log, blowup, place):
    """Evaluations packed anywhere in the buffer that receives their extension, more columns than CTAs run at once."""
    import torch
    n, size, words = 700, 1 << log, 700 << (log + blowup)
    cols = torch.from_numpy(np.random.default_rng(log).integers(0, P, size=(n, size), dtype=np.uint32).view(np.int32)).cuda()
    co, ref = torch.empty_like(cols), torch.empty(words, dtype=torch.int32, device="cuda")
    ctx.interpolate_and_extend(cols, co, ref, log, blowup, n)
    lde, co2 = torch.empty_like(ref), torch.empty_like(co)
    at = {"front": 0, "middle": (words - cols.numel()) // 2 + 4, "back": words - cols.numel()}[place]
    evals = lde[at : at + cols.numel()]
    evals.copy_(cols.view(-1))
    ctx.interpolate_and_extend(evals, co2, lde, log, blowup, n)
    assert torch.equal(co, co2) and torch.equal(ref, lde)


@pytest.mark.parametrize("log", [11, 12, 13, 14])
def test_coefficients_in_the_lde_buffer(ctx, log):
    """One column whose coefficients go where its second blown-up block comes: the extension stands at the end."""
    import torch
    ev = _buf(np.random.default_rng(log).integers(0, P, size=(1, 1 << log), dtype=np.uint32), 1 << log)
    co, ref = torch.empty_like(ev), torch.empty(2 << log, dtype=torch.int32, device="cuda")
    ctx.interpolate_and_extend(ev, co, ref, log, 1, 1)
    lde = torch.empty_like(ref)
    ctx.interpolate_and_extend(ev, lde[1 << log :], lde, log, 1, 1)
    assert torch.equal(ref, lde)
