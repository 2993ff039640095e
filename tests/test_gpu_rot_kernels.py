"""The two rotation kernels at the edges of their tiles: every launch shape and pass-pipeline mode
against the oracle's sequential sweeps, bit for bit.  Sizes: single positions, the block of 8 sweeps
and the chunks of 8 and 16 positions with a remainder either side, more than one pass, and either
side of the largest columns that the resident kernel holds (sph 1360, tri and disk 768)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = ([("sph", n) for n in (2, 3, 9, 16, 17, 18, 33, 129, 1360, 1361)] +
         [("tri", n) for n in (2, 8, 9, 15, 17, 65, 768, 769)] +
         [("disk", n) for n in (2, 8, 9, 17, 63, 768, 769)] +
         [("rect", n) for n in (3, 17, 18, 131)])
PARAMS = {"sph": (), "tri": (0.0, 0.5, -0.25), "disk": (0.0, 0.25), "rect": (0.5,)}


@pytest.fixture(scope="module")
def env():
    import torch
    import fasttransforms_b200 as ft
    from oracle.bind import Oracle
    torch.cuda.set_device(0)
    O = Oracle()
    O.set_fused(True)
    yield ft, torch, O
    ft.set_rotation_config(-1)


@pytest.mark.parametrize("kind,n", CASES, ids=[f"{k}{n}" for k, n in CASES])
def test_every_shape_matches_the_sequential_sweeps(env, kind, n):
    ft, torch, O = env
    par = PARAMS[kind]
    RP = {"sph": ft.plan_rotsphere, "tri": ft.plan_rottriangle, "disk": ft.plan_rotdisk, "rect": ft.plan_rotrectdisk}[kind](n, *par)
    PO = O.plan(kind, n, **({"beta": par[0]} if kind == "rect" else dict(zip(("alpha", "beta", "gamma"), par))), rotations_only=True)
    A = np.asfortranarray(np.random.default_rng(n).standard_normal((n, ft.layout_cols(kind, n))))   # every entry, not the triangle alone
    M = A.shape[1]
    want = {}
    for hi2lo in (True, False):
        want[hi2lo] = A.copy(order="F")
        (O.hi2lo if hi2lo else O.lo2hi)(PO, want[hi2lo])
    try:
        for cfg in [-1] + [s + 8 * p for p in range(3) for s in range(6)]:
            ft.set_rotation_config(cfg)
            for hi2lo in (True, False):
                d = torch.from_numpy(A.ravel(order="F").copy()).cuda()
                ft.rotations_dev(RP, hi2lo, d.data_ptr(), M, torch.cuda.current_stream().cuda_stream)
                got = d.cpu().numpy().reshape((n, M), order="F")
                assert np.array_equal(got, want[hi2lo]), (kind, n, cfg, hi2lo)
    finally:
        ft.set_rotation_config(-1)
        O.destroy(PO)
        RP.close()
