"""bd_cell_sort_static against a numpy sort, exact: grids whose cells are not
a multiple of the warps' 32, cells of 31 to 34 records (ordered in a row of
lanes up to 32, by a block above), records with equal x, y or z words and
identical ones, input in random and in cell order, cell starts at an address
that is not a multiple of 16 bytes."""
import ctypes as C

import numpy as np
import pytest

from gpusmoldyn_gb300 import _lib as L
from gpusmoldyn_gb300.configs import rng

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def expected(rec, dims):
    """Box [0, dims): cell edge 1, so the key's float operations are exact."""
    c = np.clip(np.floor(rec[:, :3]).astype(np.int64), 0, np.asarray(dims) - 1)
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    w = rec.view(np.uint32)
    order = np.lexsort((w[:, 3], w[:, 2], w[:, 1], w[:, 0], key))
    start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=int(np.prod(dims))))])
    return rec[order], start


def sort(rec, dims, shift=0):
    d_in = torch.from_numpy(rec).cuda()
    d_out = torch.empty_like(d_in)
    cells = int(np.prod(dims))
    d_start = torch.full((cells + 1 + shift,), -1, dtype=torch.int32, device="cuda")[shift:]
    lo, hi = (C.c_float * 3)(0, 0, 0), (C.c_float * 3)(*[float(d) for d in dims])
    rc = L.load().bd_cell_sort_static(C.c_void_p(d_in.data_ptr()), len(rec), lo, hi, (C.c_uint32 * 3)(*dims),
                                      C.c_void_p(d_out.data_ptr()), C.c_void_p(d_start.data_ptr()),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == L.BD_OK
    return d_out.cpu().numpy(), d_start.cpu().numpy()


def records(n, dims, seed):
    g = rng(seed)
    rec = (g.random((n, 4), dtype=np.float32) * np.append(np.asarray(dims, np.float32), 1.0).astype(np.float32))
    rec[:, 3] = g.integers(0, 3, n).astype(np.uint32).view(np.float32)
    return rec


@pytest.mark.parametrize("n,dims", [(1, (1, 1, 1)), (3, (5, 1, 1)), (100, (33, 1, 1)), (5000, (11, 13, 9)),
                                    (40000, (31, 33, 7)), (200000, (40, 41, 43)), (3000, (1, 2, 1))])
@pytest.mark.parametrize("ordered", [False, True])
def test_random_records(n, dims, ordered):
    rec = records(n, dims, n)
    if ordered:
        rec = expected(rec, dims)[0][::-1].copy()
    want, start = expected(rec, dims)
    got, got_start = sort(rec, dims, shift=n % 4)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    np.testing.assert_array_equal(got_start, start)


@pytest.mark.parametrize("sizes", [(31, 32, 33, 34, 1, 0, 30), (32,) * 40, (33,) * 40, (0, 5, 2, 7, 33, 1, 16, 17, 15)])
def test_cell_sizes_and_ties(sizes):
    dims = (len(sizes), 1, 1)
    g = rng(sum(sizes))
    rows = []
    for c, m in enumerate(sizes):
        r = np.zeros((m, 4), np.float32)
        r[:, 0] = c + g.choice([0.25, 0.5, 0.75], m)
        r[:, 1:3] = g.choice([0.125, 0.5], (m, 2))
        r[:, 3] = g.integers(0, 2, m).astype(np.uint32).view(np.float32)
        rows.append(r)
    rec = np.concatenate(rows)
    rec = rec[g.permutation(len(rec))]
    want, start = expected(rec, dims)
    got, got_start = sort(rec, dims)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    np.testing.assert_array_equal(got_start, start)
