"""The disk's and the annulus's phi stage on pairs of rows against the oracle (oracle/grid.py): odd and even
N around the rows a block of the kernels takes, matrices 16- and only 8-byte aligned, both directions and
both TRANS values, within 1e-14 relative 2-norm as in the tests of whole grids; and all families with rows
and columns many decades apart.  Two rows, and on the sphere the two columns of a frequency, share a complex
DFT, so what rounds in one reaches its partner.  Every output of the two stages is a sum over all rows and
columns, so no output row or column is far smaller than its neighbour: each pair of them is within the same
1e-14 of the pair's own norm."""
import numpy as np
import pytest

from conftest import rel2

pytestmark = pytest.mark.gpu

RHO = float(np.sqrt(1.0 / 3.0))


def run_at(torch, call, P, analysis, tr, X, offset):
    n, m = X.shape
    t = torch.full((n * m + 4,), 7.0, dtype=torch.float64, device="cuda")
    t[offset:offset + n * m] = torch.from_numpy(np.asfortranarray(X).ravel(order="F").copy())
    call(P, analysis, tr, t.data_ptr() + 8 * offset, n, m, torch.cuda.current_stream().cuda_stream)
    h = t.cpu().numpy()
    assert (h[:offset] == 7.0).all() and (h[offset + n * m:] == 7.0).all()
    return h[offset:offset + n * m].reshape((n, m), order="F")


def families(ft, G, N, M):
    return [(ft.plan_disk_synthesis(N, M), ft.plan_disk_analysis(N, M), ft.execute_disk_grid_dev, "disk",
             lambda op, tr, X: G.execute_disk(op, tr, op, X)),
            (ft.plan_annulus_synthesis(N, RHO, M), ft.plan_annulus_analysis(N, RHO, M), ft.execute_annulus_grid_dev, "annulus",
             lambda op, tr, X: G.execute_annulus(op, tr, op, X, RHO))]


@pytest.mark.parametrize("N,M", [(1, 5), (2, 1), (4, 5), (127, 5), (128, 9), (512, 5), (513, 9), (600, 13), (1025, 5)])
def test_rows_vs_oracle(N, M):
    import torch
    import fasttransforms_b200 as ft
    from oracle import grid as G
    X = np.random.default_rng(N * 1000 + M).uniform(-1, 1, (N, M))
    for S, A, call, name, oracle in families(ft, G, N, M):
        for P, analysis, op in ((S, False, name + "_synthesis"), (A, True, name + "_analysis")):
            for tr in "NT":
                want = oracle(op, tr, X)
                for offset in (0, 1):
                    got = run_at(torch, call, P, analysis, tr, X, offset)
                    assert rel2(got, want) <= 1e-14, (op, tr, offset, rel2(got, want))
        S.close()
        A.close()


def pairs_within(got, want, tol):
    """Rows 2p, 2p + 1 and columns 2j - 1, 2j: error against the pair's norm."""
    e2, w2 = (got - want) ** 2, want ** 2
    for axis, first in ((1, 0), (0, 1)):
        e, w = e2.sum(axis), w2.sum(axis)
        at = list(range(first, len(e), 2))
        e, w = np.add.reduceat(e, at), np.add.reduceat(w, at)
        assert np.all(e <= tol ** 2 * w), (axis, float(np.sqrt((e / w).max())))


@pytest.mark.parametrize("scaling", ["rows", "columns", "zero columns", "falling rows", "falling columns"])
@pytest.mark.parametrize("N", [33, 64])
def test_rows_and_columns_decades_apart(N, scaling):
    import torch
    import fasttransforms_b200 as ft
    from oracle import grid as G

    def data(M):
        X = np.random.default_rng(N).uniform(-1, 1, (N, M))
        if scaling == "rows":
            X[1::2] *= 1e-12
        elif scaling == "columns":
            X[:, 2::2] *= 1e-12
        elif scaling == "zero columns":
            X[:, 1::2] = 0.0
        elif scaling == "falling rows":
            X *= (10.0 ** (-14 * np.arange(N) / N))[:, None]
        else:
            X *= (10.0 ** (-14 * np.arange(M) / M))[None, :]
        return X

    M = 2 * N - 1
    X = data(M)
    for op in ("sph_synthesis", "sph_analysis", "sphv_synthesis", "sphv_analysis"):
        P = getattr(ft, "plan_" + op)(N, M)
        for tr in "NT":
            call = lambda P, analysis, tr, p, n, m, st: ft.execute_sph_grid_dev(P, op, tr, p, n, m, st)
            got, want = run_at(torch, call, P, False, tr, X, 0), G.execute(op, tr, op, X)
            assert rel2(got, want) <= 1e-14, (op, tr)
            pairs_within(got, want, 1e-14)
        P.close()
    X = data(4 * N - 3)
    for S, A, call, name, oracle in families(ft, G, N, 4 * N - 3):
        for P, analysis, op in ((S, False, name + "_synthesis"), (A, True, name + "_analysis")):
            for tr in "NT":
                assert rel2(run_at(torch, call, P, analysis, tr, X, 0), oracle(op, tr, X)) <= 1e-14, (op, tr)
        S.close()
        A.close()
