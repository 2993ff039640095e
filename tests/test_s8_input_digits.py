"""The connection multiply's input digits (fasttransforms_b200/csrc/trmm_mixed.cu, slice_input_s8_kernel):
a CPU restatement of the column scale and of the digits cut by adding 1.5 * 2^52 in units of 2^(-7 a), equal
to the rint sequence and rebuilding the scaled value within half a unit of the last digit; and, on the
GPU, columns near the bottom of the double range, whose scale must stay finite.

Bound of the last: an entry's digits leave half a unit of the last one, 2^-22 of 2^-1022 (four digits), the
matrix's digits half of 2^-28 of a row's largest entry below 2^6, i.e. at most 2^-34 of twice that entry,
the dropped levels less; the result is rounded to a multiple of 2^-1074 twice."""
import numpy as np
import pytest

from test_s8_digits import digits


def column_scale(amax):
    """(1 / s, s) as the kernel takes them."""
    ex = max(int(np.frexp(amax)[1]) if amax > 0 else 0, -1016)
    inv = float(np.ldexp(1.0, ex - 6)) if amax > 0 else 1.0
    return inv, 1.0 / inv


def cut(t, nd):
    """The kernel's digits: signed bytes from the low word of t + unit."""
    out = np.zeros(t.shape + (nd,), dtype=np.int64)
    t, unit = t.astype(np.float64).copy(), 1.5 * 2.0 ** 52
    for a in range(nd):
        u = t + unit
        out[..., a] = (u.view(np.uint64) & np.uint64(0xFF)).astype(np.uint8).view(np.int8)
        t = t - (u - unit)
        unit *= 0.0078125
    return out


@pytest.mark.parametrize("nd", [4, 5])
def test_cut_is_the_rint_sequence(nd):
    r = np.random.default_rng(1)
    ties = np.array([k + 0.5 for k in range(-64, 64)]) * (1 - 2.0 ** -53)
    steps = np.arange(-64 * 256 + 1, 64 * 256) / 256.0      # halves of the second digit among them
    t = np.concatenate([r.uniform(-64, 64, 20000), r.standard_normal(20000) * 2.0 ** r.integers(-40, 4, 20000), ties,
                        np.arange(-63, 64) + 0.5, steps, steps / 128, [0.0, -0.0, np.nextafter(64, 0), -np.nextafter(64, 0), 2.0 ** -52]])
    t = t[np.abs(t) < 64]
    d = cut(t, nd)
    assert np.array_equal(d, digits(t, nd))
    assert d.min() >= -64 and d.max() <= 64
    rec = sum(d[:, a] * 2.0 ** (-7 * a) for a in range(nd))
    assert np.abs(rec - t).max() <= 2.0 ** (-7 * (nd - 1) - 1)


@pytest.mark.parametrize("amax", [0.0, 5e-324, 1e-312, 2.0 ** -1022, 2.0 ** -1017, 2.0 ** -1016, 1e-300, 1.0, 63.9, 64.0, 1.7e308])
def test_scale_is_finite_and_exact(amax):
    inv, s = column_scale(amax)
    assert np.isfinite(s) and inv * s == 1.0 and amax * s < 64.0
    assert amax < 2.0 ** -1016 or amax * s >= 32.0


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["MIXED_BF16", "MIXED_BF16X4"])
def test_columns_of_tiny_values(precision):
    import torch
    import fasttransforms_b200 as ft
    n = 64
    M = 2 * n - 1
    st = torch.cuda.current_stream().cuda_stream
    P = ft.plan_sph2fourier(n)
    U = np.zeros((n, n))                       # column 0 (order 0) meets no sweep: out = U x
    for k in range(n):
        t = torch.zeros(M, n, dtype=torch.float64, device="cuda")
        t[0, k] = 1.0
        ft.execute_dev(P, True, "N", t.data_ptr(), n, M, st)
        U[:, k] = t[0].cpu().numpy()
    r = np.random.default_rng(3)
    for scale in (1e-312, 1e-318, 1e-307):
        x = r.uniform(-1, 1, n) * scale
        t = torch.from_numpy(r.uniform(-1, 1, (M, n))).cuda()
        t[0] = torch.from_numpy(x).cuda()
        ft.execute_shared_dev(P, True, "N", [t.data_ptr()], getattr(ft, precision), st)
        got = t[0].cpu().numpy() * 2.0 ** 1000
        big = x * 2.0 ** 1000                  # exact
        last = max(2.0 ** -22 * 2.0 ** -22, np.abs(big).max() * 2.0 ** -26)
        bound = np.abs(U).sum(1) * last + 2 * np.abs(U).max(1) * np.abs(big).sum() * 2.0 ** -34 + 2 * 2.0 ** -74
        assert np.all(np.abs(got - U @ big) <= 1.01 * bound), (scale, np.abs(got - U @ big).max(), bound.min())
    P.close()
