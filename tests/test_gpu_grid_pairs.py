"""The grid stages' row pairs and complex columns at their edges: odd and even N around the rows a block
of the kernels takes, and a matrix that is 8- but not 16-byte aligned, whose rows cannot be read as
pairs in place.  Against the oracle (oracle/grid.py), within 1e-14 relative 2-norm as in the tests of
whole grids (about log2(NM) eps, 20 eps, with a factor of two); what lies around the matrix stays."""
import numpy as np
import pytest

from conftest import rel2

pytestmark = pytest.mark.gpu

OPS = ["sph_synthesis", "sph_analysis", "sphv_synthesis", "sphv_analysis"]


def run_at(ft, torch, call, X, offset):
    n, m = X.shape
    t = torch.full((n * m + 4,), 7.0, dtype=torch.float64, device="cuda")
    t[offset:offset + n * m] = torch.from_numpy(np.asfortranarray(X).ravel(order="F").copy())
    call(t.data_ptr() + 8 * offset, n, m, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    h = t.cpu().numpy()
    assert (h[:offset] == 7.0).all() and (h[offset + n * m:] == 7.0).all()
    return h[offset:offset + n * m].reshape((n, m), order="F")


@pytest.mark.parametrize("N,M", [(2, 1), (4, 3), (127, 5), (128, 9), (512, 5), (513, 7), (600, 13), (1025, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_pairs_and_alignment(N, M, offset):
    import torch
    import fasttransforms_b200 as ft
    from oracle import grid as G
    X = np.random.default_rng(N * 1000 + M).uniform(-1, 1, (N, M))
    for op in OPS:
        P = getattr(ft, "plan_" + op)(N, M)
        for tr in "NT":
            got = run_at(ft, torch, lambda p, n, m, st: ft.execute_sph_grid_dev(P, op, tr, p, n, m, st), X, offset)
            assert rel2(got, G.execute(op, tr, op, X)) <= 1e-14, (op, tr)
        P.close()
    rho = float(np.sqrt(1.0 / 3.0))
    for fn, call, args in ((ft.plan_disk_synthesis, ft.execute_disk_grid_dev, (N, M)),
                           (ft.plan_annulus_synthesis, ft.execute_annulus_grid_dev, (N, rho, M))):
        P = fn(*args)
        outs = [[run_at(ft, torch, lambda p, n, m, st: call(P, False, tr, p, n, m, st), X, o) for tr in "NT"] for o in (0, offset)]
        for a, b in zip(*outs):
            assert rel2(b, a) <= 1e-14
        P.close()
