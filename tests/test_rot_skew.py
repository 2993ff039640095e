"""CPU restatement of the rotation kernels' index arithmetic (fasttransforms_b200/csrc/ft_internal.h:
Geo::skew_*, fasttransforms_b200/csrc/rotations.cu: skew_table_kernel, Pass, TaskGeo, Mover, stage_steps,
rot_kernel, rot_resident_kernel, with the kernels' own formulas):

* the skewed table's blocks lie one after the other and fill it, and every bulk copy of a stage stays
  inside its block (the chunk of identities at the block's end included);
* the copies of a chunk touch every double of a group's columns once, inside the matrix, and put it where
  the lane that carries the sequence reads it;
* columns run through the stages, chunk by chunk with these copies and the circular window, come out as
  the sequential sweeps leave them, bit for bit, in both directions, for whole columns and for the
  blocked paths' heads, in every launch shape, and so do resident columns, whose accesses stay inside
  the shared array."""
import numpy as np
import pytest

SPH, TRI, DISK, SPIN, RECT = 0, 1, 2, 3, 4
ROWS, LEN = 8, 8                    # Geo::kSkewRows, Geo::kSkewLen
# W, B, E, one sequence a lane (launch shapes 0 .. 4)
SHAPES = [(8, 8, 16, False), (8, 8, 8, False), (4, 8, 8, False), (8, 8, 8, True), (4, 8, 16, True)]


def sphlike(k): return k in (SPH, SPIN, RECT)
def chains(k): return 2 if sphlike(k) else 1
def step(k): return 1 if k == TRI else 2
def sequences(k): return 1 if k in (TRI, RECT) else 2
def elem(k): return 2 if k == SPIN else 1
def parities(k): return 1 if k == TRI else 2
def table_cols(k, N): return 2 * N - 1 if k == DISK else N
def chain_len(k, N, c): return (N - c + 1) // 2 if sphlike(k) else N
def task_orders(k): return 16 if sphlike(k) else 32
def last_order(k, M): return M - 1 if k in (TRI, RECT) else M // 2
def default_M(k, n): return {SPH: 2 * n - 1, TRI: n, DISK: 4 * n - 3, SPIN: 2 * n - 1, RECT: n}[k]


def top(k, N, j, c):
    if sphlike(k):
        return (N - 3 - j - c) // 2
    return N - 2 - j if k == TRI else N - 2 - (j + 1) // 2


def table_base(k, N, j):
    return j * N - (j // 2) * ((j + 1) // 2) if k == DISK else j * (2 * N + 1 - j) // 2


def skew_chunk(k): return ROWS * LEN * chains(k)
def skew_blocks(k, N, p): return 0 if top(k, N, p, 0) < 0 else top(k, N, p, 0) // ROWS + 1
def skew_chunks(k, N, p, beta): return (top(k, N, p, 0) + ROWS + 1) // LEN + 1 - beta
def skew_first(k, N, p, beta): return beta * (skew_chunks(k, N, p, 0) + 1) - beta * (beta - 1) // 2


def skew_at(k, N, p, beta):
    before = skew_first(k, N, 0, skew_blocks(k, N, 0)) if p else 0
    return (before + skew_first(k, N, p, beta)) * skew_chunk(k)


def skew_len(k, N):
    p = parities(k) - 1
    return skew_at(k, N, p, skew_blocks(k, N, p))


def packed_table(k, N):
    """(sin, cos) of the packed table; any values do, the rotations are compared bit for bit."""
    n = N * N if k == DISK else N * (N + 1) // 2
    a = np.random.default_rng(N).uniform(0.1, 1.4, n + 2 * N + 2)
    return np.stack([np.sin(a), np.cos(a)], 1)


def skew_table(k, N, sc):
    out = np.full((max(1, skew_len(k, N)), 2), np.nan)
    C = chains(k)
    for p in range(parities(k)):
        for beta in range(skew_blocks(k, N, p)):
            at = skew_at(k, N, p, beta)
            for e in range((skew_chunks(k, N, p, beta) + 1) * skew_chunk(k)):
                kappa, i, jj = e // skew_chunk(k), e % skew_chunk(k) // (LEN * C), e % (LEN * C)
                j, pos, c = p + step(k) * (ROWS * beta + i), LEN * kappa - 2 - 2 * i + jj // C, jj % C
                rotates = j < table_cols(k, N) and 0 <= pos <= top(k, N, j, c)
                assert np.isnan(out[at + e, 0])          # no block overlaps another
                out[at + e] = sc[table_base(k, N, j) + C * pos + c] if rotates else (0.0, 1.0)
    return out


def task_sweeps(k, M, mbase, blk, spin, orders):
    st, mlast = step(k), last_order(k, M)
    omax = mbase + st * (orders - 1)
    if omax > mlast:
        omax = mbase + st * ((mlast - mbase) // st)
    if k == SPIN:
        jlo, jhi = (mbase + spin) & 1, max([0] + [abs(m - spin) for m in range(mbase, omax + 1, st)]) - st
    else:
        jpar = 0 if k == TRI else mbase & 1
        jlo, jhi = jpar, omax - st
        if blk:
            jlo = min(m - st * (((m - jpar) // st) % blk) for m in range(mbase, omax + 1, st))
    return (0 if jhi < jlo else (jhi - jlo) // st + 1), jlo


def groups(k, M, orders):
    """Lowest orders of the groups of one launch."""
    span, mlast = step(k) * task_orders(k), last_order(k, M)
    first = [1] if k == TRI else ([0, 1] if k == SPIN else [2, 3])
    for f in first:
        for mb in range(f, mlast + 1, span):
            for g in range(task_orders(k) // orders):
                m = mb + step(k) * orders * g
                if m <= mlast:
                    yield m


def rotate(hi2lo, x, y, s, c):
    return (c * x + s * y, c * y - s * x) if hi2lo else (c * x - s * y, c * y + s * x)


def order_sweeps(k, m, jpar, blk, spin):
    """Sweeps of order m, lowest first."""
    me = abs(m - spin) if k == SPIN else m
    jcut = m - step(k) * (((m - jpar) // step(k)) % blk) if blk else jpar
    return [j for j in range(jpar, me - step(k) + 1, step(k)) if j >= jcut]


def sequential(k, N, col, js, hi2lo, sc):
    """The sweeps js of one order on its column, one rotation after the other."""
    C = chains(k)
    x = col.copy()
    for j in reversed(js) if hi2lo else js:
        if j >= table_cols(k, N):
            continue
        for c in range(C):
            t = top(k, N, j, c)
            for i in (range(t, -1, -1) if hi2lo else range(t + 1)):
                a, b = C * i + c, C * (i + 1) + c
                x[a], x[b] = rotate(hi2lo, x[a], x[b], *sc[table_base(k, N, j) + a])
    return x


def window_steps(hi2lo, B, E, off, win, ins, pairs):
    """stage_steps: ins the entering elements (E), pairs[b] the E pairs of sweep b by place in the copy
    (None: no rotation); returns the leaving ones."""
    W2, outs = 2 * B, []
    for e in range(E):
        u = off + e
        outs.append(win[u % W2])
        win[u % W2] = ins[e]
        if pairs is None:
            continue
        pos = E - 1 - e if hi2lo else e
        for b in range(B):
            s, c = pairs[b][pos]
            xl, xu = (u - 2 * b) % W2, (u - 2 * b - 1) % W2
            if hi2lo:
                win[xl], win[xu] = rotate(True, win[xl], win[xu], s, c)
            else:
                win[xu], win[xl] = rotate(False, win[xu], win[xl], s, c)
    return outs


def stage_pairs(k, N, skew, jpar, i0, kappa, B, E):
    """Pairs of a stage's chunk: per sweep of the stage and place, every chain; None past the block's
    chunks.  The copy is B * E * CH pairs from chunk kappa of the block of sweep i0."""
    assert i0 % B == 0 and B == ROWS
    beta, C = i0 // ROWS, chains(k)
    nk = skew_chunks(k, N, jpar, beta) if beta < skew_blocks(k, N, jpar) else 0
    kap = kappa * (E // LEN)
    assert kap >= 0
    if kap >= nk:
        return None
    at, n = skew_at(k, N, jpar, beta) + kap * skew_chunk(k), B * E * C
    assert at + n <= skew_at(k, N, jpar, beta) + (nk + 1) * skew_chunk(k) <= skew_len(k, N)
    copy = skew[at:at + n]
    place = lambda pos: pos // LEN * ROWS * LEN * C + pos % LEN * C
    return [[[copy[r * LEN * C + c + place(pos)] for pos in range(E)] for c in range(C)] for r in range(B)]


def streamed(k, N, M, mbase, orders, cols, hi2lo, shape, sc, skew, blk, spin, copy_all):
    """A group's columns (order -> column) through every pass of rot_kernel."""
    W, B, E, _ = shape
    C, D, st = chains(k), 2 * B // E, step(k)
    nsw, jlo = task_sweeps(k, M, mbase, blk, spin, orders)
    jpar = 0 if k == TRI else ((mbase + spin) & 1 if k == SPIN else mbase & 1)
    npass = -(-nsw // (W * B))
    for r in range(npass):
        at = npass - 1 - r if hi2lo else r
        left = nsw - at * W * B
        p0 = (jlo - jpar) // st + at * W * B
        stages = W if left >= W * B else -(-left // B)
        last = chain_len(k, N, 0) - 1
        emax = top(k, N, jpar + st * p0, 0) + 1
        if (copy_all and r == 0) or emax > last:
            emax = last
        emax = max(emax, 0)
        nchunk = emax // E + 1 if hi2lo else (emax + 1) // E + 1
        pmin = lambda i: (nchunk - 1 - i) * E if hi2lo else i * E - 1
        assert {p for i in range(nchunk) for p in range(pmin(i), pmin(i) + E)} >= set(range(emax + 1))
        for m, col in cols.items():
            js = set(order_sweeps(k, m, jpar, blk, spin))
            for c in range(C):
                def at_pos(p):
                    return col[C * p + c] if 0 <= p <= emax and C * p + c < N else 0.0
                stream = [[at_pos(p) for p in (range(pmin(i) + E - 1, pmin(i) - 1, -1) if hi2lo else range(pmin(i), pmin(i) + E))]
                          for i in range(nchunk)]
                for q in range(stages):
                    i0 = p0 + (stages - 1 - q if hi2lo else q) * B
                    win, out = [0.0] * (2 * B), []
                    for kk in range(nchunk + D):
                        pairs = stage_pairs(k, N, skew, jpar, i0, nchunk - 1 + D - kk if hi2lo else kk, B, E)
                        sel = None
                        if pairs is not None:
                            sel = []
                            for b in range(B):
                                i = i0 + B - 1 - b if hi2lo else i0 + b
                                sel.append(pairs[i - i0][c] if jpar + st * i in js else [(0.0, 1.0)] * E)
                        off = E % (2 * B) if D > 1 and kk & 1 else 0
                        got = window_steps(hi2lo, B, E, off, win, stream[kk] if kk < nchunk else [0.0] * E, sel)
                        if kk >= D:
                            out.append(got)
                    stream = out
                for i in range(nchunk):
                    for u, v in enumerate(stream[i]):
                        p = pmin(i) + (E - 1 - u if hi2lo else u)
                        if 0 <= p <= emax and C * p + c < N:
                            col[C * p + c] = v


def resident(k, N, M, mbase, orders, cols, hi2lo, sc, skew, blk, spin):
    """A group's columns in rot_resident_kernel."""
    W, B, E = 8, 8, 8
    C, D, st = chains(k), 2 * B // E, step(k)
    nsw, jlo = task_sweeps(k, M, mbase, blk, spin, orders)
    jpar = 0 if k == TRI else ((mbase + spin) & 1 if k == SPIN else mbase & 1)
    nblk, last = -(-nsw // B), chain_len(k, N, 0) - 1
    rows = (chain_len(k, N, 0) + E - 1) // E * E + E       # positions -1 .. rows - 2
    words = {}                                             # every value a block publishes, and what it has finished then
    for g in range(nblk):
        i0 = (jlo - jpar) // st + (nblk - 1 - g if hi2lo else g) * B
        emax = max(0, min(last, top(k, N, jpar + st * i0, 0) + 1))
        chi = emax // E if hi2lo else (emax + 1) // E
        K = chi + 1 + D
        assert chi < 2000
        published = [(g * 4096 + (2048 - (chi + 1) if hi2lo else 0), set())]
        done = set()
        for kk in range(K):
            cin = chi - kk if hi2lo else kk
            cout = cin + D if hi2lo else cin - D
            if kk <= chi:
                if g > 0:   # the block before has finished chunk cin, or never touches it
                    need = (g - 1) * 4096 + (2048 - cin if hi2lo else cin + 1)
                    first = next(s for w, s in words[g - 1] if w >= need)
                    assert cin in first or cin not in words[g - 1][-1][1]
            if kk >= D:
                done = done | {cout}
                published.append((g * 4096 + (4095 if kk + 1 == K else 2048 - cout if hi2lo else cout + 1), done))
        assert [w for w, _ in published] == sorted(w for w, _ in published) and published[-1][0] < (g + 1) * 4096
        words[g] = published
        for m, col in cols.items():
            js = set(order_sweeps(k, m, jpar, blk, spin))
            for c in range(C):
                arr = np.zeros(rows)
                arr[1:1 + chain_len(k, N, c)] = col[c::C]
                win = [0.0] * (2 * B)
                for kk in range(K):
                    cin = chi - kk if hi2lo else kk
                    cout = cin + D if hi2lo else cin - D
                    places = lambda ch: [ch * E + E - 1 - e for e in range(E)] if hi2lo else [ch * E - 1 + e for e in range(E)]
                    assert kk > chi or all(-1 <= p <= rows - 2 for p in places(cin))
                    assert kk < D or all(-1 <= p <= rows - 2 for p in places(cout))
                    pairs = stage_pairs(k, N, skew, jpar, i0, chi + D - kk if hi2lo else kk, B, E)
                    sel = None
                    if pairs is not None:
                        sel = []
                        for b in range(B):
                            i = i0 + B - 1 - b if hi2lo else i0 + b
                            sel.append(pairs[i - i0][c] if jpar + st * i in js else [(0.0, 1.0)] * E)
                    ins = [arr[1 + p] for p in places(cin)] if kk <= chi else [0.0] * E
                    outs = window_steps(hi2lo, B, E, E % (2 * B) if D > 1 and kk & 1 else 0, win, ins, sel)
                    if kk >= D:
                        for p, v in zip(places(cout), outs):
                            arr[1 + p] = v
                col[c::C] = arr[1:1 + chain_len(k, N, c)]


TABLE_CASES = [(k, n) for k in (SPH, TRI, DISK, RECT) for n in (1, 2, 3, 4, 8, 9, 15, 16, 17, 18, 19, 33, 64)]


@pytest.mark.parametrize("k,n", TABLE_CASES)
def test_table_blocks_fill_the_table(k, n):
    out = skew_table(k, n, packed_table(k, n))
    assert not np.isnan(out[:skew_len(k, n)]).any()
    # every sweep with a rotation has its row
    for j in range(table_cols(k, n)):
        for c in range(chains(k)):
            p = 0 if k == TRI else j & 1
            assert top(k, n, j, c) < 0 or (j - p) // step(k) // ROWS < skew_blocks(k, n, p)


def check(k, n, M, blk=0, spin=0, shapes=SHAPES):
    sc = packed_table(k, n)
    skew = skew_table(k, n, sc)
    rng = np.random.default_rng(n)
    cols = {m: rng.uniform(-1, 1, n) for m in range(last_order(k, M) + 1)}
    for hi2lo in (True, False):
        want = {}
        for m in cols:
            jpar = 0 if k == TRI else ((m + spin) & 1 if k == SPIN else m & 1)
            want[m] = sequential(k, n, cols[m], order_sweeps(k, m, jpar, blk, spin), hi2lo, sc)
        for shape in shapes + [None]:
            orders = 32 // (chains(k) * sequences(k)) if shape is None or shape[3] else task_orders(k)
            for copy_all in (False, True):
                for mbase in groups(k, M, orders):
                    mine = {m: cols[m].copy() for m in range(mbase, min(last_order(k, M), mbase + step(k) * (orders - 1)) + 1, step(k))}
                    if shape is None:
                        resident(k, n, M, mbase, orders, mine, hi2lo, sc, skew, blk, spin)
                    else:
                        streamed(k, n, M, mbase, orders, mine, hi2lo, shape, sc, skew, blk, spin, copy_all)
                    for m in mine:
                        assert np.array_equal(mine[m], want[m]), (k, n, hi2lo, shape, copy_all, m)


@pytest.mark.parametrize("k,n", [(SPH, 2), (SPH, 3), (SPH, 9), (SPH, 17), (SPH, 18), (SPH, 41), (TRI, 2), (TRI, 9), (TRI, 17), (TRI, 34),
                                 (DISK, 2), (DISK, 8), (DISK, 17), (DISK, 22), (RECT, 3), (RECT, 18), (RECT, 43)])
def test_columns_match_the_sequential_sweeps(k, n):
    check(k, n, default_M(k, n))


@pytest.mark.parametrize("n,s", [(3, 1), (9, 2), (18, 0), (18, 5), (29, 3)])
def test_spin_columns(n, s):
    check(SPIN, n, 2 * n - 1, spin=s)


@pytest.mark.parametrize("k,n", [(SPH, 74), (DISK, 37), (TRI, 40)])
def test_heads_of_the_blocked_paths(k, n):
    check(k, n, default_M(k, n), blk=32, shapes=[(4, 8, 16, True), (8, 8, 16, False)])


@pytest.mark.parametrize("k,n,M", [(SPH, 17, 9), (SPH, 9, 41), (DISK, 9, 7), (DISK, 6, 45), (TRI, 18, 18)])
def test_other_widths(k, n, M):
    check(k, n, M)


def test_several_passes():
    check(TRI, 72, 72, shapes=[(8, 8, 16, False), (4, 8, 8, False)])


# Mover: what a warp moves of one chunk
def place(k, nc, cols, c, cl):
    return c * (cols + 1) + cl if nc == sequences(k) else cl * chains(k) + c


@pytest.mark.parametrize("k,one", [(SPH, False), (SPH, True), (DISK, False), (DISK, True), (TRI, False), (RECT, False), (SPIN, False), (SPIN, True)])
@pytest.mark.parametrize("E", [8, 16])
def test_chunk_copies(k, one, E):
    C, ES, SEQ, st = chains(k), elem(k), sequences(k), step(k)
    nc = 1 if one else SEQ
    orders = 32 * nc // (C * SEQ)
    cols = orders * SEQ
    rowd = C * (cols + 1) if nc == SEQ else 33
    rpc, segs, per = E * C * ES, cols // ES, cols * E * C // 32
    rb, sp = (rpc // 32, 1) if rpc >= 32 else (1, 32 // rpc)
    paired = k in (SPH, DISK)
    ph_n = rb if rb > 1 else (2 if paired and sp == 1 else 1)
    nv, sstep = per // ph_n, 1 if rb > 1 else sp * ph_n
    assert rpc % 32 == 0 or 32 % rpc == 0
    slot_step = place(k, nc, cols, 0, sstep * ES)
    col_of = lambda s: {TRI: s, RECT: 2 * s, SPIN: 4 * s}.get(k, 4 * (s >> 1) + (s & 1))
    N = 21
    for M in ([33, 34, 40] if k in (TRI, RECT) else [1, 3, 33, 35, 65, 67]):
        mlast = last_order(k, M)
        for side in ((0, 1) if k == SPIN else (0,)):
            for mbase in list(groups(k, M, orders)) + ([mlast + 1] if k != TRI else []):
                no = 0 if mbase > mlast else min(orders, (mlast - mbase) // st + 1)
                # the group's columns, by sequence group (segment)
                if k == SPIN:
                    want_cols = {o: (2 * (mbase + 2 * o) - (0 if side else 1)) for o in range(no)}
                    want_cols = {o: c for o, c in want_cols.items() if 0 <= c < M}
                elif k in (TRI, RECT):
                    want_cols = {o: mbase + st * o for o in range(no)}
                else:
                    want_cols = {2 * o + h: 2 * (mbase + 2 * o) - 1 + h for o in range(no) for h in (0, 1)}
                for hi2lo in (True, False):
                    for pmin in ((0, 8) if hi2lo else (-1, 7)):
                        emax, seen = chain_len(k, N, 0) - 1, {}
                        for lane in range(32):
                            ls = lane // rpc if rpc < 32 else 0
                            nseg, seg0 = no * (segs // orders) - ls, 0
                            col0 = mbase if k in (TRI, RECT) else 2 * mbase - 1
                            if k == SPIN:
                                col0 = 2 * mbase - (0 if side else 1)
                                if col0 < 0:
                                    seg0 = 1 - ls
                                most = (M - 1 - col0) // 4 + 1
                                if nseg + ls > most:
                                    nseg = most - ls
                            base = (col0 + col_of(ls)) * ES * N
                            for ph in range(ph_n):
                                rr = ph * 32 + lane if rb > 1 else lane % rpc
                                seg = 0 if rb > 1 else ph * sp
                                p = pmin + rr // (ES * C)
                                row_ok = 0 <= p <= emax and C * p + rr // ES % C < N
                                at = base + col_of(seg) * ES * N + ES * C * pmin + rr
                                pos, c, part = rr // (ES * C), rr // ES % C, rr % ES
                                u = E - 1 - pos if hi2lo else pos
                                slot = u * rowd + place(k, nc, cols, c, (seg + ls) * ES + part)
                                for v in range(nv):
                                    ok = row_ok and seg0 <= seg + v * sstep < nseg
                                    d = slot + v * slot_step
                                    assert d not in seen        # every place of the slot once
                                    seen[d] = at + v * col_of(sstep) * ES * N if ok else None
                                    assert not ok or 0 <= seen[d] < ES * N * M
                        # what the lanes read: sequence h of lane's order, chain, at step e
                        for lane in range(32):
                            o = lane // C if nc == SEQ else lane // (C * SEQ)
                            c = lane % C
                            off = lane % C * (cols + 1) + lane // C * nc if nc == SEQ else lane
                            for e in range(E):
                                p = pmin + (E - 1 - e if hi2lo else e)
                                for h in range(nc):
                                    q = h if nc == SEQ else lane // C % SEQ
                                    s, part = (o, q) if k == SPIN else (o * SEQ + q, 0)
                                    there = s in want_cols and 0 <= p <= emax and C * p + c < N
                                    want = (want_cols[s] * N + C * p + c) * ES + part if there else None
                                    assert seen[e * rowd + off + h] == want, (k, one, E, M, mbase, side, hi2lo, lane, e, h)
