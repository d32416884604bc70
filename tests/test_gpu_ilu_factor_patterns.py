"""The block-ILU(0) factorisation on block patterns that no quadrilateral grid
makes: elements whose lower neighbours are adjacent to one another (a neighbour's
update then falls on a block of the row that is needed next, not only on the
diagonal one). Against block elimination in NumPy at 1e-11 of the largest entry
(chains of 5 products of at most 100 terms, diagonally dominant blocks of
condition below 10: 5 x 100 x 10 x 1.1e-16 leaves a margin above 10)."""
import ctypes as C

import numpy as np
import pytest
import torch

from linalg_calls import lib, ptr

pytestmark = pytest.mark.gpu

PATTERNS = {
    "complete": [list(range(5))] * 5,
    "triangles": [[0, 1, 2], [0, 1, 2, 3], [0, 1, 2, 3, 4], [1, 2, 3, 4], [2, 3, 4]],
    "ring of three": [[0, 1, 2], [0, 1, 2], [0, 1, 2]],
    "grid": [[0, 1, 2], [0, 1, 3], [0, 2, 3], [1, 2, 3]],
}


@pytest.mark.parametrize("bs", [4, 9, 16, 25, 36, 64, 100])
@pytest.mark.parametrize("name", PATTERNS)
def test_factors(name, bs):
    cols = PATTERNS[name]
    E = len(cols)
    rng = np.random.default_rng(bs)
    at = {(e, k): rng.standard_normal((bs, bs)) * (0.2 / bs ** 0.5) + (2.0 * np.eye(bs) if e == k else 0.0)
          for e in range(E) for k in cols[e]}
    lu = torch.from_numpy(np.stack([at[e, k] for e in range(E) for k in cols[e]])).cuda()
    uinv = torch.full((E, bs, bs), float("nan"), dtype=torch.float64, device="cuda")
    # L_ek and the updates of row e in ascending order of k; then inv(U_ee) U_ek above the diagonal
    inv = {}
    for e in range(E):
        for k in [c for c in cols[e] if c < e]:
            at[e, k] = at[e, k] @ inv[k]
            for j in [c for c in cols[k] if c > k and c in cols[e]]:
                at[e, j] = at[e, j] - at[e, k] @ at[k, j]
        inv[e] = np.linalg.inv(at[e, e])
    level = []
    for e in range(E):
        level.append(max([level[k] + 1 for k in cols[e] if k < e], default=0))
    order = sorted(range(E), key=lambda e: (level[e], e))
    off = np.concatenate([[0], np.cumsum(np.bincount(level))]).astype(np.int32)
    d = [torch.tensor(v, dtype=torch.int32, device="cuda")
         for v in (np.concatenate([[0], np.cumsum([len(c) for c in cols])]), sum(cols, []), order, [0])]
    st = lib().ilu_factor(C.c_int(E), C.c_int(bs), C.c_int(len(sum(cols, []))), ptr(d[0]), ptr(d[1]), ptr(d[2]),
                          off.ctypes.data_as(C.c_void_p), C.c_int(len(off) - 1), ptr(lu), ptr(uinv), ptr(d[3]))
    assert st == 0
    torch.cuda.synchronize()
    assert int(d[3][0]) == 0
    got, want = lu.cpu().numpy(), []
    for e in range(E):
        for k in cols[e]:
            want.append(at[e, k] if k <= e else inv[e] @ at[e, k])
    want = np.stack(want)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
    ui = np.stack([inv[e] for e in range(E)])
    assert np.abs(uinv.cpu().numpy() - ui).max() <= 1e-11 * np.abs(ui).max()
