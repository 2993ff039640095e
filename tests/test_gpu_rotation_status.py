"""The rotation kernels' status word (ft_b200_rotation_status) is a report: a launch after one that gave
up runs as usual, whichever kernel and queue it uses.  The word is set from the host to what a bounded
wait that ran out leaves there; the outputs are compared bit for bit with those of a clear word."""
import numpy as np
import pytest

HARMONIC = [("sph", 64, 0), ("sph", 700, 0), ("sph", 700, 8), ("sph", 700, 16), ("sph", 700, 11), ("disk", 600, 12), ("tri", 900, 8),
            ("tri", 900, -1)]


def test_negative_value_is_refused():
    import fasttransforms_b200 as ft
    assert ft.lib.ft_b200_rotation_status(-1) == -1
    assert ft.lib.ft_b200_last_status() == 1
    with pytest.raises(ft.FTB200Error):
        ft.rotation_status(-3)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,cfg", HARMONIC)
def test_later_launches_run_as_usual(kind, n, cfg):
    import torch
    import fasttransforms_b200 as ft
    st = torch.cuda.current_stream().cuda_stream
    P = {"sph": ft.plan_sph2fourier, "tri": lambda n: ft.plan_tri2cheb(n, 0.0, 0.0, 0.0), "disk": lambda n: ft.plan_disk2cxf(n, 0.0, 0.0)}[kind](n)
    A = ft.rand_layout(kind, n, 4)
    outs = []
    try:
        ft.set_rotation_config(cfg)
        ft.rotation_status(0)
        for status in (0, 3):
            ft.rotation_status(status)
            t = torch.from_numpy(A.ravel(order="F").copy()).cuda()
            for fwd in (True, False):
                ft.execute_dev(P, fwd, "N", t.data_ptr(), n, A.shape[1], st)
                outs.append(t.cpu().numpy())
            assert ft.rotation_status(status) == status
        assert np.array_equal(outs[0], outs[2]) and np.array_equal(outs[1], outs[3])
        assert ft.device_status(P) == 3      # reads and clears
        assert ft.device_status(P) == 0 and ft.rotation_status() == 0
    finally:
        ft.set_rotation_config(-1)
        ft.rotation_status(0)
        P.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [200, 815, 1024])
def test_spin_launches_run_as_usual(n):
    import torch
    import fasttransforms_b200 as ft
    st = torch.cuda.current_stream().cuda_stream
    R = ft.plan_rotspinsphere(n, 2)
    A = ft.spinsphrand(n, 2, 4)
    outs = []
    try:
        for status in (0, 5):
            ft.rotation_status(status)
            t = torch.from_numpy(A.ravel(order="F").view(np.float64).copy()).cuda()
            for hi2lo in (True, False):
                ft.spin_rotations_dev(R, hi2lo, t.data_ptr(), A.shape[1], st)
                outs.append(t.cpu().numpy())
            assert ft.rotation_status(status) == status
        assert np.array_equal(outs[0], outs[2]) and np.array_equal(outs[1], outs[3])
    finally:
        ft.rotation_status(0)
        R.close()
