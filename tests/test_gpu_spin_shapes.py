"""The spin sweeps at the edges of the kernels, bit for bit against the oracle's sequential sweeps: every
launch shape and pass-pipeline mode (interleaved parts, the columns of orders -m and m in tasks of their
own, one column in the task of order 0), sizes around the block of 8 sweeps, the chunks of 8 and 16
positions and more than one pass; widths other than 2n - 1; stage 1 in one and in several passes of four
sweeps (|s| = 4 .. 9); and the sizes at which the launch rule takes one sequence a lane (801, 832)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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


def data(n, M, seed):
    """Every entry, not the triangle alone."""
    r = np.random.default_rng(seed)
    return np.asfortranarray(r.standard_normal((n, M)) + 1j * r.standard_normal((n, M)))


def compare(env, n, s, M, cfgs):
    ft, torch, O = env
    A = data(n, M, 100 * n + s)
    R, PO = ft.plan_rotspinsphere(n, s), O.spin_plan(n, s, False)
    try:
        for hi2lo in (True, False):
            want = A.copy(order="F")
            (O.spin_hi2lo if hi2lo else O.spin_lo2hi)(PO, want)
            for cfg in cfgs:
                ft.set_rotation_config(cfg)
                t = torch.from_numpy(A.ravel(order="F").view(np.float64).copy()).cuda()
                ft.spin_rotations_dev(R, hi2lo, t.data_ptr(), M, torch.cuda.current_stream().cuda_stream)
                got = t.cpu().numpy().view(np.complex128).reshape((n, M), order="F")
                assert np.array_equal(got, want), (n, s, M, cfg, hi2lo)
    finally:
        ft.set_rotation_config(-1)
        O.spin_destroy(PO)
        R.close()


EVERY = [-1] + [s + 8 * p for p in range(3) for s in range(6)]


@pytest.mark.parametrize("n", [1, 2, 3, 9, 16, 17, 18, 33, 65, 131, 200])
@pytest.mark.parametrize("s", [-3, 0, 1, 2])
def test_every_shape(env, n, s):
    compare(env, n, s, 2 * n - 1, EVERY)


@pytest.mark.parametrize("n,M", [(17, 1), (17, 3), (40, 31), (33, 35), (70, 69)])
def test_other_widths(env, n, M):
    compare(env, n, 2, M, EVERY)


@pytest.mark.parametrize("n", [5, 8, 31, 33, 100])
@pytest.mark.parametrize("s", [4, -5, 6, 7, -8, 9])
def test_several_passes_of_stage_1(env, n, s):
    compare(env, n, s, 2 * n - 1, [-1, 0, 8])


@pytest.mark.parametrize("n,s", [(801, 2), (832, -3)])
def test_one_sequence_a_lane_by_rule(env, n, s):
    compare(env, n, s, 2 * n - 1, [-1, 3, 11, 19])
