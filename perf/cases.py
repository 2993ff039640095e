"""Workloads of the harmonic transforms as a program calls them: coefficients in, function data
out, and back again.

Every case runs both directions through the public entry points: the forward transform on a copy
of the coefficients, then the backward transform on a copy of its result; both results are
returned.  (The transforms work in place, so a program that keeps its coefficients copies them.)
Coefficients are U(-1, 1) in the family's triangular layout, drawn on the GPU from the seed.

A case names its entry point in "call":

  single   execute_dev: one field on device memory (families sph, tri, disk)
  host     execute_<transform>: one field in host memory, the drop-in C call
  batched  execute_batched_dev: sph fields of several degrees in one call
  shared   execute_shared_dev: fields of one plan in one call, at a stated precision
  sht      execute_dev and execute_sph_grid_dev: coefficients to values on the sphere's grid and back
  spin     execute_spin_dev: spin-weighted coefficients (complex)
"""
import math
import random

import numpy as np
import torch

import fasttransforms_b200 as ft

PRECISION = {"fp64": ft.FP64, "mixed_bf16": ft.MIXED_BF16, "mixed_bf16x4": ft.MIXED_BF16X4}
STEP = {"sph": 2, "tri": 1, "disk": 4}    # columns a row of the triangular layout loses


def listed():
    return [
        # the smallest calls: a low-degree field transformed in every step of an outer loop, where
        # the calls themselves are most of the time
        {"name": "sph_63", "call": "single", "family": "sph", "n": 64},
        # a climate or gravity model's degree, not a power of two
        {"name": "sph_300", "call": "single", "family": "sph", "n": 301},
        # an ordinary field whose matrix stays in L2
        {"name": "sph_1023", "call": "single", "family": "sph", "n": 1024},
        # the largest single field, plain double precision
        {"name": "sph_4095", "call": "single", "family": "sph", "n": 4096},
        # polynomials on a triangle element, odd size
        {"name": "tri_1000", "call": "single", "family": "tri", "n": 1001, "alpha": 0.0, "beta": 0.0, "gamma": 0.0},
        # an existing C program relinked: host matrices, copies inside the call
        {"name": "host_sph_511", "call": "host", "family": "sph", "n": 512},
        # many fields of uneven degree in one call
        {"name": "batch_sph", "call": "batched", "family": "sph", "fields": 24, "sizes": 6, "n_min": 100, "n_max": 1500, "spread": 3},
        # a stack of levels or time steps sharing a plan on the tensor cores
        {"name": "shared_sph_4095", "call": "shared", "family": "sph", "n": 4096, "fields": 16, "precision": "mixed_bf16"},
        # the same for the disk, with the four-slice form
        {"name": "shared_disk_1500", "call": "shared", "family": "disk", "n": 1501, "fields": 6, "precision": "mixed_bf16x4", "alpha": 0.0, "beta": 0.0},
        # a mesh's elements sharing a plan, where the triangle's conditioning asks for double precision
        {"name": "shared_tri_767", "call": "shared", "family": "tri", "n": 768, "fields": 12, "precision": "fp64", "alpha": -0.5, "beta": -0.5, "gamma": -0.5},
        # a whole spherical harmonic transform: coefficients to point values and back, odd size
        {"name": "sht_1500", "call": "sht", "family": "sph", "n": 1501},
        # polarisation maps and wind fields: spin-weighted coefficients
        {"name": "spin2_1023", "call": "spin", "family": "spin", "n": 1024, "s": 2},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["single", "single", "single", "host", "batched", "shared", "sht", "spin"])
    c = {"call": call, "family": "sph"}
    if call in ("single", "shared"):
        c["family"] = rng.choice(["sph", "sph", "tri", "disk"])
    if call == "single":
        c["n"] = size(32, {"sph": 4096, "tri": 3000, "disk": 2048}[c["family"]])
    elif call == "host":
        c["n"] = size(32, 1200)
    elif call == "batched":
        c.update(fields=rng.randint(4, 28), sizes=rng.randint(2, 6), n_min=size(32, 200), n_max=size(300, 1600), spread=rng.randint(0, 999))
    elif call == "shared":
        c["n"] = size(200, {"sph": 3000, "tri": 1500, "disk": 1600}[c["family"]])
        c["fields"] = rng.randint(2, 12)
        c["precision"] = rng.choice(["fp64", "mixed_bf16", "mixed_bf16x4"])
    elif call == "sht":
        c["n"] = size(32, 2500)
    else:
        c["family"] = "spin"
        c["n"] = size(32, 2000)
        c["s"] = rng.choice([-2, -1, 0, 1, 2])
    if c["family"] == "tri":
        p = rng.choice([0.0, -0.5])
        c.update(alpha=p, beta=p, gamma=p)
    elif c["family"] == "disk":
        c.update(alpha=0.0, beta=0.0)
    return c


def columns(family, n):
    return {"sph": 2 * n - 1, "tri": n, "disk": 4 * n - 3, "spin": 2 * n - 1}[family]


def field_sizes(case):
    """n of each field."""
    if case["call"] == "batched":
        r = random.Random(case["spread"])
        sizes = [int(round(math.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"]))))) for _ in range(case["sizes"])]
        return [sizes[f % len(sizes)] for f in range(case["fields"])]
    return [case["n"]] * case.get("fields", 1)


def coefficients(case, seed):
    """The fields' coefficients on the GPU, as (M, n) tensors (column-major N x M matrices);
    (M, n, 2) for the complex spin coefficients."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    fields = []
    for n in field_sizes(case):
        M = columns(case["family"], n)
        row = torch.arange(n, device="cuda")[None, :]
        col = torch.arange(M, device="cuda")[:, None]
        if case["family"] == "spin":
            A = torch.rand(M, n, 2, generator=g, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
            A.mul_(((row < n - abs(case["s"])) & (col < M - 2 * row))[:, :, None])
        else:
            A = torch.rand(M, n, generator=g, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
            A.mul_(col < M - STEP[case["family"]] * row)
        fields.append(A)
    return fields


def make_plan(case, n):
    if case["family"] == "tri":
        return ft.plan_tri2cheb(n, case["alpha"], case["beta"], case["gamma"])
    if case["family"] == "disk":
        return ft.plan_disk2cxf(n, case["alpha"], case["beta"])
    if case["family"] == "spin":
        return ft.plan_spinsph2fourier(n, case["s"])
    return ft.plan_sph2fourier(n)


def prepare(case, seed):
    A = coefficients(case, seed)
    sizes = field_sizes(case)
    plans = {n: make_plan(case, n) for n in set(sizes)}
    state = {"case": case, "sizes": sizes, "plans": plans, "A": A}
    if case["call"] == "host":
        state["A"] = [a.cpu().numpy().T for a in A]               # Fortran order, n x M
        state["forward"] = [np.empty_like(a, order="F") for a in state["A"]]
        state["back"] = [np.empty_like(a, order="F") for a in state["A"]]
        return state
    state["forward"] = [torch.empty_like(a) for a in A]
    state["back"] = [torch.empty_like(a) for a in A]
    if case["call"] == "sht":
        state["synthesis"] = ft.plan_sph_synthesis(case["n"])
        state["analysis"] = ft.plan_sph_analysis(case["n"])
    return state


def run(state):
    case, sizes, plans = state["case"], state["sizes"], state["plans"]
    A, F, B = state["A"], state["forward"], state["back"]
    call, n = case["call"], sizes[0]
    if call == "host":
        np.copyto(F[0], A[0])
        ft.execute_sph2fourier("N", plans[n], F[0])
        np.copyto(B[0], F[0])
        ft.execute_fourier2sph("N", plans[n], B[0])
        return {"forward": F, "back": B}
    stream = torch.cuda.current_stream().cuda_stream
    M = columns(case["family"], n)
    if len(A) == 1:
        F[0].copy_(A[0])
    else:
        torch._foreach_copy_(F, A)
    if call == "single":
        ft.execute_dev(plans[n], True, "N", F[0].data_ptr(), n, M, stream)
        B[0].copy_(F[0])
        ft.execute_dev(plans[n], False, "N", B[0].data_ptr(), n, M, stream)
    elif call == "spin":
        ft.execute_spin_dev(plans[n], True, "N", F[0].data_ptr(), n, M, stream)
        B[0].copy_(F[0])
        ft.execute_spin_dev(plans[n], False, "N", B[0].data_ptr(), n, M, stream)
    elif call == "sht":
        ft.execute_dev(plans[n], True, "N", F[0].data_ptr(), n, M, stream)
        ft.execute_sph_grid_dev(state["synthesis"], "sph_synthesis", "N", F[0].data_ptr(), n, M, stream)
        B[0].copy_(F[0])
        ft.execute_sph_grid_dev(state["analysis"], "sph_analysis", "N", B[0].data_ptr(), n, M, stream)
        ft.execute_dev(plans[n], False, "N", B[0].data_ptr(), n, M, stream)
    elif call == "shared":
        precision = PRECISION[case["precision"]]
        ft.execute_shared_dev(plans[n], True, "N", [f.data_ptr() for f in F], precision, stream)
        torch._foreach_copy_(B, F)
        ft.execute_shared_dev(plans[n], False, "N", [b.data_ptr() for b in B], precision, stream)
    else:
        P = [plans[k] for k in sizes]
        Ms = [columns("sph", k) for k in sizes]
        ft.execute_batched_dev(P, True, "N", [f.data_ptr() for f in F], sizes, Ms, stream)
        torch._foreach_copy_(B, F)
        ft.execute_batched_dev(P, False, "N", [b.data_ptr() for b in B], sizes, Ms, stream)
    return {"forward": F, "back": B}


def rotations(family, n, s=0):
    """Givens rotations of one direction of one field."""
    if family == "tri":
        return sum((n - 1 - j) * (n - 1 - j) for j in range(n - 1))       # sweep j: columns j + 1 .. n - 1
    if family == "disk":
        last = 2 * n - 2                                                  # the highest order
        return sum(2 * max(0, n - 1 - (j + 1) // 2) * ((last - j) // 2) for j in range(last))
    if family == "spin":
        count = 0
        for m in range(n):
            d = abs(m - abs(s))
            low = (m + abs(s)) % 2
            part = sum(n - 2 - j for j in range(d - 2, low - 1, -2))
            part += sum(max(0, n - 1 - d - j) for j in range(min(m, abs(s))))
            count += (2 if m == 0 else 4) * part                          # orders -m and m, both parts
        return count
    return sum(2 * (n - 2 - j) * ((n - 1 - j) // 2) for j in range(n - 2))


def work(case):
    """Both directions: six flops a rotation, the triangular multiplies, (sht) the grid's FFTs; each
    direction's matrix read and written once, with one copy each, its tables and matrices read once."""
    flops, moved = 0.0, 0.0
    counts = {}
    for n in field_sizes(case):
        counts[n] = counts.get(n, 0) + 1
    for n, fields in counts.items():
        M = columns(case["family"], n)
        parts = 2 if case["family"] == "spin" else 1
        multiply = float(n) * (n + 1) * M * parts * (2 if case["family"] == "tri" else 1)
        if case["family"] == "tri" and case["alpha"] == case["beta"] == case["gamma"] == -0.5:
            multiply = float(n) * (n + 1) * M       # the second multiply is the identity
        flops += 2.0 * fields * (6.0 * rotations(case["family"], n, case.get("s", 0)) + multiply)
        matrix = 8.0 * n * M * parts
        plan = 8.0 * n * (n + 1) + 8.0 * n * (n + 1)        # (sin, cos) table; two triangles a direction
        moved += fields * 8 * matrix + 2 * plan
        if case["call"] == "sht":
            moved += 4 * matrix
            flops += 2 * 2.5 * n * M * (math.log2(n) + math.log2(M))
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------------
# The values of the transforms in 64 bits: the basis functions by their three-term recurrences,
# and the Fourier or Chebyshev coefficients by the discrete orthogonality of the cosines.
# ---------------------------------------------------------------------------

def jacobi_start(a, b):
    """log2 of the orthonormal constant polynomial of the weight (1 - x)^a (1 + x)^b."""
    h = (a + b + 1) * math.log(2) + torch.lgamma(a + 1) + torch.lgamma(b + 1) - torch.lgamma(a + b + 2)
    return -h / (2 * math.log(2))


def jacobi_step(k, a, b):
    """x p_k = A_{k-1} p_{k-1} + B_k p_k + A_k p_{k+1}: B_k and A_k."""
    t = 2 * k + a + b
    if k == 0:
        return (b - a) / (t + 2), torch.sqrt(4 * (1 + a) * (1 + b) / ((t + 2) ** 2 * (t + 3)))
    B = (b - a) * (b + a) / (t * (t + 2))
    return B, torch.sqrt(4 * (k + 1) * (k + 1 + a) * (k + 1 + b) * (k + 1 + a + b) / ((t + 2) ** 2 * (t + 1) * (t + 3)))


def jacobi_sums(C, a, b, start, x, live):
    """sum_k C[:, m, k] w_m(x) p_k(x), p_k the orthonormal Jacobi polynomials of (a[m], b[m]), as
    (sets, orders, points).  start[m, i] is log2 of w_m(x_i) p_0, which spans more than the exponent
    range, so the recurrence runs on values scaled by powers of two; the first live(k) orders have
    coefficients from k on."""
    G = torch.zeros(C.shape[0], C.shape[1], x.numel(), device=x.device, dtype=torch.float64)
    E = torch.floor(start / 256) * 256                      # value = p 2^E
    p, q = torch.exp2(start - E), torch.zeros_like(start)
    a, b, before = a[:, None], b[:, None], torch.zeros_like(a)[:, None]
    for k in range(C.shape[2]):
        m = live(k)
        if m < 1:
            break
        a, b, before, E, p, q = a[:m], b[:m], before[:m], E[:m], p[:m], q[:m]
        if k % 8 == 0:
            up = (p.abs() > 2.0 ** 128) | (q.abs() > 2.0 ** 128)
            down = torch.exp2(up.double() * -256)
            p, q, E = p * down, q * down, E + up.double() * 256
            F = torch.exp2(E.clamp(min=-2000))
        value = p * F[:m]
        for g, c in zip(G, C):
            g[:m].addcmul_(c[:m, k, None], value)
        B, A = jacobi_step(k, a, b)
        p, q = (x * p - B * p - before * q) / A, p
        before = A
    return G


def cosine_analysis(n, dev):
    """Matrices from values at phi_i = (i + 1/2) pi / n to the coefficients of cos(k phi), of
    sin((k + 1) phi) and of cos((k + 1/2) phi), k = 0 .. n - 1."""
    k = torch.arange(n, device=dev)[:, None]
    i = torch.arange(n, device=dev)[None, :]

    def angle(u):                                           # u pi / (4 n), reduced exactly
        return (u % (8 * n)).double() * (math.pi / (4 * n))

    cosine = torch.cos(angle(2 * k * (2 * i + 1))) * (2.0 / n)
    cosine[0] *= 0.5
    sine = torch.sin(angle(2 * (k + 1) * (2 * i + 1))) * (2.0 / n)
    sine[n - 1] *= 0.5
    half = torch.cos(angle((2 * k + 1) * (2 * i + 1))) * (2.0 / n)
    return cosine, sine, half


def column_values(case, n, fields):
    """The forward transform's columns as functions at phi_i = (i + 1/2) pi / n: (sets, orders, n) with
    two sets a field (columns 2m - 1 and 2m; order 0 in the second), four for spin, one for tri."""
    family, dev = case["family"], fields[0].device
    phi = (torch.arange(n, device=dev).double() + 0.5) * (math.pi / n)
    x = torch.cos(phi)
    if family == "tri":
        m = torch.arange(n, device=dev).double()
        a, b = 2 * m + case["beta"] + case["gamma"] + 1, torch.full_like(m, case["alpha"])
        start = m[:, None] * (torch.log2(torch.sin(phi / 2)) * 2 + 1) + jacobi_start(a, b)[:, None]
        return jacobi_sums(torch.stack(fields), a, b, start, x, lambda k: n - k)
    orders = (columns(family, n) + 1) // 2
    m = torch.arange(orders, device=dev).double()
    sets = []
    for A in fields:
        for part in ([A[..., 0], A[..., 1]] if family == "spin" else [A]):
            first = torch.zeros(orders, n, device=dev, dtype=torch.float64)
            first[1:] = part[1::2]
            sets += [first, part[0::2]]
    if family == "disk":
        a, b = torch.zeros_like(m) + case["beta"], m + case["alpha"]
        start = (m[:, None] * torch.log2(torch.cos(phi / 2)) + (case["alpha"] + case["beta"] + m + 2)[:, None] / 2 +
                 jacobi_start(a, b)[:, None])
        return jacobi_sums(torch.stack(sets), a, b, start, x, lambda k: 2 * (n - k) - 1)
    if family == "spin":
        G = [None] * len(sets)
        for side, s in ((0, case["s"]), (1, -case["s"])):   # orders -m, then m
            a, b = (m - s).abs(), (m + s).abs()
            half = torch.log2(torch.sin(phi / 2)) + 0.5, torch.log2(torch.cos(phi / 2)) + 0.5
            start = a[:, None] * half[0] + b[:, None] * half[1] + jacobi_start(a, b)[:, None]
            got = jacobi_sums(torch.stack(sets[side::2]), a, b, start, x, lambda k: n - k)
            G[side::2] = list(got)
        return torch.stack(G)
    start = m[:, None] * torch.log2(torch.sin(phi)) + jacobi_start(m, m)[:, None]
    return jacobi_sums(torch.stack(sets), m, m, start, x, lambda k: n - k)


def interleave(G, n, M):
    """Sets (columns 2m - 1, columns 2m) of one field back to its M columns."""
    out = torch.empty(M, n, device=G.device, dtype=torch.float64)
    out[1::2], out[0::2] = G[0][1:], G[1]
    return out


def forward_values(case, n, fields):
    """The forward transforms of fields of one size."""
    dev, family, M = fields[0].device, case["family"], columns(case["family"], n)
    G = column_values(case, n, fields)
    cosine, sine, half = cosine_analysis(n, dev)
    if family == "tri":
        x = torch.cos((torch.arange(n, device=dev).double() + 0.5) * (math.pi / n))
        a, b = torch.tensor([case["gamma"]], device=dev).double(), torch.tensor([case["beta"]], device=dev).double()
        p, q, before, rows = torch.exp2(jacobi_start(a, b)).expand(n), torch.zeros_like(x), 0.0, []
        for k in range(n):
            rows.append(p)
            B, A = jacobi_step(k, a, b)
            p, q, before = ((x - B) * p - before * q) / A, p, A
        right = torch.stack(rows) @ cosine.T                # [m, j]: p_m in the T_j
        return [right.T @ (g @ cosine.T) for g in G]
    if case["call"] == "sht":
        sets = [interleave(G[2 * f:2 * f + 2], n, M) for f in range(len(fields))]
        j = torch.arange(M, device=dev)
        phase = (((j + 1) // 2)[:, None] * j[None, :] % M).double() * (2 * math.pi / M)
        trig = torch.where((j % 2 == 1)[:, None], torch.sin(phase), torch.cos(phase)) / math.sqrt(math.pi)
        trig[0] *= math.sqrt(0.5)
        return [trig.T @ g for g in sets]
    odd = {"sph": sine, "spin": sine, "disk": half}[family]
    H = torch.empty_like(G)
    s = abs(case.get("s", 0)) % 2
    H[:, s::2] = G[:, s::2] @ cosine.T
    H[:, 1 - s::2] = G[:, 1 - s::2] @ odd.T
    if family == "spin":
        return [torch.stack([interleave(H[4 * f + 2 * p:4 * f + 2 * p + 2], n, M) for p in (0, 1)], dim=2).contiguous() for f in range(len(fields))]
    return [interleave(H[2 * f:2 * f + 2], n, M) for f in range(len(fields))]


def exact(case, seed):
    """run()'s results in 64 bits; the backward transform undoes the forward one."""
    A = coefficients(case, seed)
    sizes = field_sizes(case)
    F = [None] * len(A)
    for n in set(sizes):
        which = [f for f, k in enumerate(sizes) if k == n]
        for f, v in zip(which, forward_values(case, n, [A[f] for f in which])):
            F[f] = v
    if case["call"] == "host":
        A, F = [a.cpu().numpy().T for a in A], [f.cpu().numpy().T for f in F]
    return {"forward": F, "back": A}
