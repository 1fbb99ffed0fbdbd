"""A joint trial point's parameters and costs, one launch each per group (bmc_joint_params, bmc_segment_costs), against
NumPy: the parameters exactly, the costs to the rounding of their sums."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,nf,rows,shared", [(1, 13, [0], -1), (33, 23, [3, -1, 22], 1), (257, 38, [], 37),
                                               (64, 38, [5, 6, 7, 8, 9, 10, 11, 12], 0)])
def test_parameters_at_a_point(cuda, nv, nf, rows, shared):
    import torch
    from bmc_b200 import _lib
    rng = np.random.default_rng(nv)
    base, x, scl = rng.random((nf, nv)), rng.random((2 * nv, max(1, len(rows)))), rng.random(len(rows)) + 0.5
    idx = rng.permutation(2 * nv)[:nv].astype(np.int64)
    want = base.copy()
    for j, r in enumerate(rows):
        if r >= 0:
            want[r] = x[idx, j] * scl[j]
    if shared >= 0:
        want[shared] = 0.75 * 1.5
    up = lambda a: torch.as_tensor(a).cuda()
    db, di, dx, ds, out = up(base), up(idx), up(x), up(np.array([0.75])), torch.empty((nf, nv), dtype=torch.float64, device="cuda")
    n = len(rows)
    _lib.check(_lib.lib().bmc_joint_params(nv, nf, _lib.ptr(db), _lib.ptr(di), _lib.ptr(dx), n, (C.c_int32 * n)(*rows),
                                           (C.c_double * n)(*scl), shared, 1.5, _lib.ptr(ds), _lib.ptr(out),
                                           _lib.stream_handle()))
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("lengths", [[1], [0, 31, 32, 33], [1000, 1, 0, 64, 5]])
def test_costs_of_segments(cuda, lengths):
    """A sum of n non-negative terms rounds by at most n x 2^-53, a term (difference, square) by 3 x 2^-53."""
    import torch
    from bmc_b200 import _lib
    rng = np.random.default_rng(len(lengths))
    seg = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    z, zm = rng.random((2, max(1, seg[-1])))
    idx = rng.permutation(len(lengths)).astype(np.int64)
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    dseg, dz, dm, di = up(seg), up(z), up(zm), up(idx)
    out = torch.full((len(lengths),), -1.0, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().bmc_segment_costs(len(lengths), _lib.ptr(dseg), _lib.ptr(dz), _lib.ptr(dm), _lib.ptr(di),
                                            _lib.ptr(out), _lib.stream_handle()))
    got = out.cpu().numpy()
    for v, n in enumerate(lengths):
        want = float(np.sum((z[seg[v]:seg[v + 1]] - zm[seg[v]:seg[v + 1]]) ** 2, dtype=np.longdouble))
        assert abs(got[idx[v]] - want) <= (n + 3) * 2.0 ** -53 * want
