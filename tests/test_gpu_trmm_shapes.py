"""The connection multiply's tile shapes (128 x 64, 64 x 64, 32 x 32, chosen by the size of a launch) give
the same bits: a field around the tiles' edges alone (small launches take 32 x 32) and in a batch with a
large field, whose launch takes the larger tiles.  Sums are cut at multiples of 256 in k whatever the tile,
so sizes around 256 and 512 are among them.  The fields alone are within 1e-14 of the oracle (as in the
tests of the transforms; tri amplifies rounding and is compared bit for bit only)."""
import numpy as np
import pytest

from conftest import rel2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,params,degrees,large", [
    ("sph", (), [31, 32, 33, 64, 65, 129, 256, 257, 513], [700, 1500, 2600]),
    ("disk", (0.0, 0.0), [31, 33, 65, 257], [500, 1100]),
    ("tri", (0.0, 0.0, 0.0), [31, 32, 33, 65, 129, 257, 513], [1200, 2200]),
])
def test_shapes_agree(kind, params, degrees, large):
    import torch
    import fasttransforms_b200 as ft
    from oracle.bind import Oracle
    O = Oracle()
    O.set_fused(True)
    st = torch.cuda.current_stream().cuda_stream
    planner = {"sph": ft.plan_sph2fourier, "tri": ft.plan_tri2cheb, "disk": ft.plan_disk2cxf}[kind]
    plans = [planner(n, *params) for n in degrees]
    fields = [ft.rand_layout(kind, n, 70 + i) for i, n in enumerate(degrees)]
    def on_device(A):
        return torch.from_numpy(A.ravel(order="F").copy()).cuda()
    alone = {}
    for fwd in (True, False):
        for i, (P, A) in enumerate(zip(plans, fields)):
            t = on_device(A)
            ft.execute_dev(P, fwd, "N", t.data_ptr(), P.n, P.M, st)
            alone[fwd, i] = t.cpu().numpy()
            if kind == "tri" or P.n > 257:
                continue
            want = A.copy(order="F")
            PO = O.plan(kind, P.n, *params)
            O.execute(PO, fwd, "N", want)
            O.destroy(PO)
            assert rel2(alone[fwd, i].reshape(A.shape, order="F"), want) <= 1e-14, (P.n, fwd)
    for n in large:
        L = planner(n, *params)
        for fwd in (True, False):
            ts = [on_device(A) for A in fields] + [on_device(ft.rand_layout(kind, n, 5))]
            ps = plans + [L]
            ft.execute_batched_dev(ps, fwd, "N", [t.data_ptr() for t in ts], [p.n for p in ps], [p.M for p in ps], st)
            single = on_device(ft.rand_layout(kind, n, 5))
            ft.execute_dev(L, fwd, "N", single.data_ptr(), L.n, L.M, st)
            assert torch.equal(ts[-1], single), (n, fwd)
            for i, t in enumerate(ts[:-1]):
                assert np.array_equal(t.cpu().numpy(), alone[fwd, i]), (n, degrees[i], fwd)
        L.close()
    for P in plans:
        P.close()
