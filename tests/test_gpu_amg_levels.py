"""The AMG hierarchy's numeric kernels (sparse products by row length, power
iteration, prolongator, coarsest inverse) and V-cycle against a plain
scipy restatement of the same smoothed-aggregation method."""

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import has_cuda

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not has_cuda(), reason="needs a CUDA device")]


def _aggregate(A, skip):
    """Three-pass standard aggregation, every off-diagonal entry strong."""
    n, ip, ix = A.shape[0], A.indptr, A.indices
    agg, na = np.full(n, -1), 0
    nbrs = [[c for c in ix[ip[r]:ip[r + 1]] if c != r and not skip[c]] for r in range(n)]
    for r in range(n):
        if not skip[r] and agg[r] < 0 and nbrs[r] and all(agg[c] < 0 for c in nbrs[r]):
            agg[r] = agg[nbrs[r]] = na
            na += 1
    first = agg.copy()
    for r in range(n):
        if not skip[r] and agg[r] < 0:
            agg[r] = next((first[c] for c in nbrs[r] if first[c] >= 0), -1)
    for r in range(n):
        if not skip[r] and agg[r] < 0 and nbrs[r]:
            agg[r] = na
            agg[[c for c in nbrs[r] if agg[c] < 0]] = na
            na += 1
    return agg, na


def _power_start(n, skip):
    x, h, mask = np.empty(n), 0x9E3779B97F4A7C15, (1 << 64) - 1
    for r in range(n):
        h ^= (h << 13) & mask
        h ^= h >> 7
        h ^= (h << 17) & mask
        x[r] = 0.0 if skip[r] else 0.5 + (h % 1000003) / 1000003.0
    return x


def _hierarchy(A, skip, max_coarse, max_levels=10):
    levels = []
    while True:
        n = A.shape[0]
        if n <= max_coarse or len(levels) + 1 >= max_levels:
            break
        agg, na = _aggregate(A, skip)
        if na == 0 or na >= n:
            break
        d = A.diagonal()
        dinv = np.where(d != 0, 1.0 / np.where(d != 0, d, 1.0), 1.0)
        s = np.sqrt(np.abs(dinv))
        x, lam = _power_start(n, skip), 0.0
        for _ in range(20):
            y = np.where(skip, 0.0, s * (A @ (s * x)))
            lam = (x @ y) / (x @ x)
            x = y / np.linalg.norm(y)
        omega = (4.0 / 3.0) / (1.05 * lam if lam > 0 else 2.0)
        on = agg >= 0
        size = np.bincount(agg[on], minlength=na)
        T = sp.csr_matrix((1.0 / np.sqrt(size[agg[on]]), (np.nonzero(on)[0], agg[on])), shape=(n, na))
        P = (T - omega * (sp.diags(dinv) @ (A @ T))).tocsr()
        levels.append((A, dinv, omega, P))
        # structural pattern: with strictly positive copies nothing cancels
        Q = (abs(A) @ T + T).tocsr()
        S = (Q.T @ (abs(A) @ Q)).tocsr()
        C = (P.T @ (A @ P)).tocsr()
        S.data[:] = 0.0
        A, skip = (C + S).tocsr(), np.zeros(na, dtype=bool)
        A.sort_indices()
    return levels, np.linalg.inv(A.toarray())


def _vcycle(levels, inv, b, k=0, pre=2, post=2):
    if k == len(levels):
        return inv @ b
    A, dinv, w, P = levels[k]
    x = w * dinv * b
    for _ in range(pre - 1):
        x = x + w * dinv * (b - A @ x)
    x = x + P @ _vcycle(levels, inv, P.T @ (b - A @ x), k + 1)
    for _ in range(post):
        x = x + w * dinv * (b - A @ x)
    return x


def _graph(kind, rng):
    """(lower, upper) index pairs of a symmetric pattern and its size."""
    if kind == "p1":            # rows of 15: A P rows of at most 15 entries
        from up3d_b200.mesh.kuhn import kuhn_box
        nodes, el = kuhn_box(16, 7, 5)
        return len(nodes), np.vstack([el[:, [i, j]] for i in range(4) for j in range(i)])
    if kind.startswith("path"):        # one-dimensional, odd size: rows of 2 and 3
        n = {"path": 2057, "path512": 1536}[kind]
        return n, np.column_stack([np.arange(n - 1), np.arange(1, n)])
    if kind == "band":          # neighbours up to 14 away: long A P and Galerkin rows
        n = 6000
        return n, np.vstack([np.column_stack([np.arange(n - k), np.arange(k, n)]) for k in (1, 2, 3, 5, 9, 14)])
    if kind == "grid":          # far neighbours: A P rows of about a dozen
        n = 9000
        return n, np.vstack([np.column_stack([np.arange(n - k), np.arange(k, n)]) for k in (1, 21, 22, 440, 443)])
    n = 40000                   # an expander: Galerkin rows past the shared-memory staging
    return n, rng.integers(0, n, size=(6 * n, 2))


CASES = [("p1", 500, False), ("p1", 30, True), ("path", 10, False), ("path", 600, True), ("path", 700, False),
         ("path512", 512, False), ("band", 40, True), ("band", 500, False), ("grid", 400, False), ("expander", 500, False)]


@pytest.mark.parametrize("kind,max_coarse,dirichlet", CASES)
def test_vcycle_matches_scipy(kind, max_coarse, dirichlet):
    import torch
    from up3d_b200.solve.linear import as_device_csr, build_amg_preconditioner, with_dirichlet
    rng = np.random.default_rng(3)
    n, e = _graph(kind, rng)
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    w = rng.uniform(0.5, 2.0, len(e))
    A = sp.coo_matrix((np.r_[-w, -w], (np.r_[e[:, 0], e[:, 1]], np.r_[e[:, 1], e[:, 0]])), shape=(n, n)).tocsr()
    A = (A + sp.diags(0.05 - np.asarray(A.sum(axis=1)).ravel())).tocsr()
    A.sort_indices()
    skip = np.zeros(n, dtype=bool)
    if dirichlet:
        skip[rng.choice(n, size=n // 20, replace=False)] = True
    Ad = as_device_csr(A)
    if dirichlet:
        Ad = with_dirichlet(Ad, torch.from_numpy(skip.astype(np.uint8)).cuda())
    ml, M = build_amg_preconditioner(Ad, max_coarse=max_coarse)
    keep = sp.diags((~skip).astype(float))
    levels, inv = _hierarchy((keep @ A @ keep + sp.diags(skip.astype(float))).tocsr(), skip, max_coarse)
    assert ml.n_levels == len(levels) + 1 and ml.n_coarse == len(inv)
    b = rng.standard_normal(n)
    z = M.matvec(torch.from_numpy(b).cuda()).cpu().numpy()
    ref = _vcycle(levels, inv, b)
    # rounding only: 1e-15 per operation, amplified by the coarsest inverse
    # (condition below 1e5 for the 0.05 shift)
    assert np.linalg.norm(z - ref) < 1e-10 * np.linalg.norm(ref)
