"""The column sums on the tensor cores (composition, quotients) at the edges of their blocks: the
smallest domains that take them and those below, column counts around a group of eight and around the
narrow ones that the composition sums row by row, columns and outputs that are not 16-byte aligned;
against the definitions in Python integers."""
import numpy as np
import pytest

import oracle
import verifier as V

pytestmark = pytest.mark.gpu
P = 2**31 - 1


def _dev(a, offset):
    import torch
    flat = np.zeros(a.size + offset, dtype=np.uint32)
    flat[offset:] = a.reshape(-1)
    return torch.from_numpy(flat.view(np.int32)).cuda()[offset:]


def _out(words, offset):
    import torch
    return torch.full((words + offset,), -1, dtype=torch.int32, device="cuda")[offset:]


def _words(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("log_n,W,offset", [(3, 3, 0), (4, 9, 0), (5, 3, 0), (5, 8, 0), (6, 9, 0), (7, 16, 2), (6, 17, 3),
                                            (14, 24, 0), (1, 51, 3), (3, 26, 0), (4, 27, 1), (4, 100, 2), (6, 15, 0), (6, 14, 1),
                                            (6, 16, 0), (7, 20, 2), (6, 20, 3), (6, 21, 0)])
def test_composition(ctx, log_n, W, offset):
    rng = np.random.default_rng(10 * log_n + W)
    rows = 2 << log_n
    cols = rng.integers(0, P, size=(W, rows), dtype=np.uint32)
    cols[:, 0], cols[:, 1] = P - 1, 0  # the largest limbs, and none
    co = rng.integers(0, P, size=(W - 2, 4), dtype=np.uint32)
    co[0] = P - 1
    den = [int(x) for x in rng.integers(1, P, size=2)]
    out = _out(4 * rows, offset)
    ctx.wide_fib_composition(_dev(cols, offset), log_n, W, _dev(co, 0), *den, out)
    c = cols.astype(object)
    cons = [(c[k + 2] - c[k] ** 2 - c[k + 1] ** 2) for k in range(W - 2)]
    d = np.array([den[r >> log_n] for r in range(rows)], dtype=object)
    ref = np.array([(sum(int(co[k, i]) * cons[k] for k in range(W - 2)) * d) % P for i in range(4)]).astype(np.uint32)
    assert np.array_equal(_words(out).reshape(4, rows), ref)


@pytest.mark.parametrize("log,n,offset", [(5, 9, 0), (6, 1, 0), (6, 8, 0), (7, 13, 0), (6, 17, 1), (7, 24, 2), (2, 24, 0),
                                          (3, 25, 0), (5, 49, 1), (5, 27, 2)])
def test_quotients(ctx, log, n, offset):
    import torch
    rng = np.random.default_rng(10 * log + n)
    cols = rng.integers(0, P, size=(n, 1 << log), dtype=np.uint32)
    cols[:, 3] = P - 1
    c, pts = rng.integers(0, P, size=(n, 4)), rng.integers(0, P, size=(4, 4)).tolist()
    dc, out = _dev(cols, offset), _out(4 << log, offset)
    ptrs = torch.tensor([dc.data_ptr() + 4 * (i << log) for i in range(n)], dtype=torch.int64, device="cuda")
    ctx.accumulate_quotients(log, ptrs, _dev(c.astype(np.uint32), 0), *pts, out, n)
    got = _words(out).reshape(4, -1)
    px, py, sa, sb = (V.qfrom(p) for p in pts)
    for row in range(1 << log):
        x, y = V.index_point(V.domain_index(log, V.bitrev(row, log)))
        num = V.q(0)
        for i in range(n):
            num = V.qadd(num, V.qmulm(V.qfrom(c[i].tolist()), int(cols[i, row])))
        num = V.qsub(num, V.qadd(V.qmulm(sa, y), sb))
        den = V.csub(V.cmul(V.csub(px[0], (x, 0)), py[1]), V.cmul(V.csub(py[0], (y, 0)), px[1]))
        assert got[:, row].tolist() == list(V.qflat(V.qmulc(num, V.cinv(den)))), row


@pytest.mark.parametrize("log,n", [(0, 3), (3, 2), (11, 5), (12, 1), (13, 33), (14, 600), (16, 160), (18, 38), (16, 3000),
                                   (17, 1500)])
def test_openings(ctx, log, n):
    """Below the tensor-core kernel's 2^12, with a chunk per CTA (n few) and per warp, and four chunks a warp in one and
    two CTAs a column (the last two)."""
    import torch
    rng = np.random.default_rng(log)
    cols = rng.integers(0, P, size=(n, 1 << log), dtype=np.uint32)
    cols[0] = P - 1
    px, py = rng.integers(0, P, size=(2, 4)).tolist()
    out = torch.empty(4 * n, dtype=torch.int32, device="cuda")
    ctx.eval_at_point(_dev(cols, 0), log, n, 1 << log, px, py, out)
    got = _words(out).reshape(n, 4)
    for c in {0, n // 2, n - 1}:
        assert np.array_equal(got[c], oracle.eval_at_point(cols[c], px, py)), c


def test_openings_of_more_chunks_than_the_factor_table(ctx):
    """One CTA a column of 2^25 coefficients: 2048 chunks a warp, whose factors beyond the table's 1024 are multiplied
    in. Every column is the same one (stride 0), as so many would not fit the device."""
    import torch
    log, n = 25, 2960
    col = np.random.default_rng(log).integers(0, P, size=1 << log, dtype=np.uint32)
    px, py = np.random.default_rng(log).integers(0, P, size=(2, 4)).tolist()
    out = torch.empty(4 * n, dtype=torch.int32, device="cuda")
    ctx.eval_at_point(_dev(col, 0), log, n, 0, px, py, out)
    got = _words(out).reshape(n, 4)
    assert (got == oracle.eval_at_point(col, px, py)).all()
