"""Weighted dots at the edges of their chunks and vector groups, and the small
symmetric eigensolver, against numpy.

A dot of n terms summed in any order is within n rounding errors of sum |w V y|;
here the sum runs in chunks and warps, well below that.  Jacobi eigenvalues and
eigenvectors reconstruct the matrix to some 100 m rounding errors of its norm.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# sector sizes (rows x cols) around the 2048-element chunk, vectors around groups of four
@pytest.mark.parametrize("dims", [[(1, 1)], [(32, 64), (1, 2047), (683, 3)], [(90, 91), (17, 1), (64, 65)]])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 64])
def test_wdot_matches_numpy(dims, k):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule = tb.SU2FusionRule()
    sp = rt.space(rule, [tb.GradedSpace(rule, [(j, d[0]) for j, d in enumerate(dims)])],
                  [tb.GradedSpace(rule, [(j, d[1]) for j, d in enumerate(dims)])])
    plan = rt.fplan(sp)
    n = sp.size
    rng = np.random.default_rng(n + k)
    V, y = rng.standard_normal((k, n + 1)), rng.standard_normal(n)  # odd row stride: rows alternate in alignment
    w = np.concatenate([np.full(r * c, lab[0] + 1.0) for lab, r, c, _ in sp.sectors()])
    dV, dy, out = torch.as_tensor(V, device="cuda"), torch.as_tensor(y, device="cuda"), torch.empty(
        k, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    _lib.call("tnt_wdot", rt._h, plan._h, k, p(dV), n + 1, p(dy), p(out), rt.stream())
    bound = n * 2.0 ** -53 * (np.abs(V[:, :n]) @ (w * np.abs(y))) + 1e-300
    assert np.all(np.abs(out.cpu().numpy() - V[:, :n] @ (w * y)) <= bound)


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 48])
def test_symeig_matches_numpy(m):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rng = np.random.default_rng(m)
    T = np.diag(rng.standard_normal(m)) + np.diag(rng.standard_normal(m - 1), 1)
    for A in (T + T.T, np.eye(m), np.zeros((m, m))):
        dA = torch.as_tensor(np.ascontiguousarray(A).ravel(), device="cuda")
        w = torch.empty(m, dtype=torch.float64, device="cuda")
        v = torch.empty(m * m, dtype=torch.float64, device="cuda")
        p = lambda t: C.c_void_p(t.data_ptr())
        _lib.call("tnt_symeig", rt._h, m, p(dA), p(w), p(v), rt.stream())
        w, v = w.cpu().numpy(), v.cpu().numpy().reshape(m, m).T
        tol = 100 * m * 2.0 ** -53 * max(1.0, np.linalg.norm(A))
        assert np.all(np.abs(w - np.linalg.eigvalsh(A)) <= tol)
        assert np.abs((v * w) @ v.T - A).max() <= tol and np.abs(v.T @ v - np.eye(m)).max() <= tol
