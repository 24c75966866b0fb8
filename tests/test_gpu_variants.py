"""GPU: the kernels behind a choice on sizes or structure, each at the sizes
where that choice can go wrong, against the CPU oracle (or plain numpy / FP64
torch where the oracle has no such function)."""
import numpy as np
import pytest

from isai_kernel_gb300 import gen

pytestmark = pytest.mark.gpu


def T(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def N(t):
    return t.detach().cpu().numpy()


def scalar_csr(rng, nb, bs, most, shuffled):
    """A scalar CSR matrix of nb*bs rows with up to `most` entries a row, some
    rows empty, some columns repeated; `shuffled` leaves every third row's
    entries in random order."""
    n = nb * bs
    rows = []
    for i in range(n):
        k = 0 if rng.random() < 0.15 else int(rng.integers(0, most + 1))
        c = rng.integers(0, n, size=k)
        if k > 2 and rng.random() < 0.5:
            c[1] = c[0]
        c = c if shuffled and i % 3 == 0 else np.sort(c)
        rows.append(c.astype(np.int32))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum([len(c) for c in rows], out=rp[1:])
    col = np.concatenate(rows) if n else np.zeros(0, np.int32)
    return rp, col, rng.uniform(-1, 1, size=col.shape[0])


# Bit for bit: the block columns are integers and every scalar position sums
# its entries in file order in both.
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("nb", [1, 3, 33])
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 7, 8])
def test_csr_to_bsr_merge(cuda, orc, bs, nb, shuffled):
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(100 * bs + nb)
    rp, col, val = scalar_csr(rng, nb, bs, 12 if nb < 33 else 70, shuffled)
    _, r, c, v = api.csr_to_bsr5(nb * bs, bs, T(rp, cuda), T(col, cuda), T(val, cuda))
    ro, co, vo = orc.csr_to_bsr(nb * bs, bs, rp, col, val)
    assert np.array_equal(N(r), ro) and np.array_equal(N(c), co)
    assert np.array_equal(N(v), vo)


@pytest.mark.parametrize("bad", [-1, 40])
def test_csr_to_bsr_column_out_of_range(cuda, bad):
    from isai_kernel_gb300 import api

    rp = np.arange(0, 81, 2, dtype=np.int32)
    col = np.tile(np.array([0, 39], np.int32), 40)
    col[50] = bad
    with pytest.raises(api.BiluError):
        api.csr_to_bsr5(40, 5, T(rp, cuda), T(col, cuda), T(np.ones(80), cuda))


# ------------------------------------------------------------------ level analysis
def pattern_of(rows):
    """rowptr, col of a block pattern given as one set of columns per row."""
    cols = [np.array(sorted(set(r) | {i}), np.int32) for i, r in enumerate(rows)]
    rp = np.zeros(len(rows) + 1, np.int32)
    np.cumsum([len(c) for c in cols], out=rp[1:])
    return rp, np.concatenate(cols)


def level_pattern(name):
    rng = np.random.default_rng(11)
    if name == "chain":  # every row waits for a row of its own warp
        return pattern_of([[i - 1, i + 1] if 0 < i < 99 else [] for i in range(100)])
    if name == "grid":  # grid lines that straddle the warps
        A = gen.laplace2d(21, bs=4)
        return A.rowptr, A.colind
    if name == "dense":  # rows of more dependencies than a warp takes at once
        return pattern_of([range(97) for _ in range(97)])
    if name == "hubs":  # hub rows among short ones, hubs waiting for hubs
        n = 333
        return pattern_of([rng.integers(0, n, size=200 if i % 31 == 5 else 5) for i in range(n)])
    if name == "diagonal":
        return pattern_of([[] for _ in range(65)])
    if name == "wide":  # levels of 700 and of 15,000 rows: one and two radix-sorted digits
        rows = [[i - 700] if 700 <= i < 1400 else [] for i in range(1400)]
        return pattern_of(rows + [[i - 15000] if i >= 16400 else [] for i in range(1400, 46400)])
    return pattern_of([rng.integers(0, 4000, size=9) for _ in range(4000)])  # "random"


@pytest.mark.parametrize("lower", [1, 0])
@pytest.mark.parametrize("name", ["chain", "grid", "dense", "hubs", "diagonal", "wide",
                                  "random"])
def test_level_analysis(cuda, name, lower):
    """The analysis record against longest paths on the host: the rows by
    (level, index), the level bounds, the level count and the largest
    dependency count."""
    from isai_kernel_gb300 import _lib, api

    rp, col = level_pattern(name)
    nb, nnzb = len(rp) - 1, len(col)
    level = np.zeros(nb, np.int64)
    deg = 0
    for i in (range(nb) if lower else range(nb - 1, -1, -1)):
        c = col[rp[i]:rp[i + 1]]
        c = c[c < i] if lower else c[c > i]
        deg = max(deg, len(c))
        level[i] = 1 + level[c].max() if len(c) else 0
    L = _lib.lib()
    info = api._ws(L.bilu_sptrsv_analysis_bytes(nb), cuda)
    ws = api._ws(L.bilu_sptrsv_analysis_ws_bytes(nb, nnzb), cuda)
    r, c = T(rp, cuda), T(col, cuda)
    api.call("bilu_sptrsv_analysis", nb, nnzb, 4, api._p(r), api._p(c), lower, api._p(info),
             api._p(ws), ws.numel(), api._s())
    words = N(info).view(np.int32)
    up = lambda k: (k + 63) // 64 * 64  # 256-byte steps in int32 words
    o1 = up(nb + 1)
    o2 = o1 + up(nb + 1)
    o3 = o2 + up(nb + 2)
    nlev = int(level.max()) + 1
    assert words[o3] == nlev and words[o3 + 1] == deg
    bounds = np.zeros(nlev + 1, np.int64)
    np.cumsum(np.bincount(level, minlength=nlev), out=bounds[1:])
    assert np.array_equal(words[o2:o2 + nlev + 1], bounds)
    want = np.lexsort((np.arange(nb), level))
    got = words[o1:o1 + nb].copy()
    for a, b in zip(bounds[:-1], bounds[1:]):
        if b - a > 16384:  # wider levels keep the order they were found in
            got[a:b].sort()
    assert np.array_equal(got, want)
    # one dependency more than the caller's block count leaves room for
    st = L.bilu_sptrsv_analysis(nb, nnzb - 1, 4, api._p(r), api._p(c), lower, api._p(info),
                                api._p(ws), ws.numel(), api._s())
    deps = int(sum(((col[rp[i]:rp[i + 1]] < i) if lower else (col[rp[i]:rp[i + 1]] > i)).sum()
                   for i in range(nb)))
    assert st == (0 if nnzb - 1 >= nb and deps <= nnzb - 1 - nb else
                  _lib_status("BILU_ERR_WORKSPACE" if nnzb - 1 >= nb else "BILU_ERR_ARG"))


def _lib_status(name):
    from isai_kernel_gb300 import _lib

    return {v: k for k, v in _lib.STATUS.items()}[name]


# ------------------------------------------------------------------ BILU(0)
def nine_point(side):
    """2D 9-point pattern: neighbours of a row are neighbours of each other."""
    at = lambda x, y: y * side + x
    return pattern_of([[at(u, v) for u in range(max(x - 1, 0), min(x + 2, side))
                        for v in range(max(y - 1, 0), min(y + 2, side))]
                       for y in range(side) for x in range(side)])


def bilu_pattern(name):
    if name == "5-point":
        A = gen.laplace2d(19, bs=4)
        return A.rowptr, A.colind
    if name == "7-point":
        A = gen.convdiff3d(7, bs=4)
        return A.rowptr, A.colind
    if name == "bipartite":  # 13 dependencies or 13 blocks right of the diagonal
        return pattern_of([range(13, 26) if i < 13 else range(13) for i in range(26)])
    if name == "one-sided":  # no U_KI for most dependencies
        rng = np.random.default_rng(3)
        return pattern_of([rng.integers(0, 90, size=2) for _ in range(90)])
    if name == "9-point":
        return nine_point(11)
    if name == "dense":
        return pattern_of([range(37) for _ in range(37)])
    if name == "diagonal":
        return pattern_of([[] for _ in range(7)])
    rng = np.random.default_rng(5)  # "hubs": rows of more than 32 dependencies
    return pattern_of([rng.integers(0, 300, size=150 if i % 37 == 9 else 4) for i in range(300)])


@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["5-point", "7-point", "bipartite", "one-sided", "9-point",
                                  "dense", "diagonal", "hubs"])
def test_bilu0_schedules(cuda, orc, name, bs):
    """Every schedule's factor: the same bits, and the oracle's to 1e-12 of
    the largest entry (diagonally dominant blocks: errors of a few ulps)."""
    from isai_kernel_gb300 import api

    rp, col = bilu_pattern(name)
    nb, nnzb = len(rp) - 1, len(col)
    rng = np.random.default_rng(bs)
    val = rng.uniform(-1, 1, size=(nnzb, bs, bs))
    rows = np.repeat(np.arange(nb), np.diff(rp))
    diag = np.nonzero(rows == col)[0]
    i = np.arange(bs)
    val[diag[:, None], i, i] = 2.0 * bs * np.diff(rp)[:, None]
    ref, _ = orc.bsrilu0(nb, bs, rp, col, val)
    out = []
    for schedule in (-1, 0, 1):
        v = T(val, cuda)
        assert api.bsrilu02_inplace(nb, nnzb, bs, T(rp, cuda), T(col, cuda), v, schedule) == -1
        out.append(N(v))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert np.max(np.abs(out[0] - ref)) <= 1e-12 * np.max(np.abs(ref))


def rule_pattern(name):
    """Patterns on either side of the lines between BILU(0)'s schedules."""
    if name == "two wide levels":  # 8192 rows a level, one dependency
        return pattern_of([[i - 8192] if i >= 8192 else [] for i in range(2 * 8192)])
    if name == "a little narrower":
        return pattern_of([[i - 6000] if i >= 6000 else [] for i in range(2 * 6000)])
    if name == "wide, six dependencies":
        return pattern_of([[(i * 7 + k * 31) % 8192 for k in range(6)] if i >= 8192 else []
                           for i in range(2 * 8192)])
    if name == "wide, a triangle":
        return pattern_of([[] if i < 8192 else [0, 1, i - 8192] if i > 16383 else [i - 8192]
                           for i in range(16385)] + [[8192, 0]])
    if name == "parallel long rows":  # one level of them: no chain to cut
        return pattern_of([range(i % 50, 2000, 50) if i >= 2000 else [] for i in range(2200)])
    A = gen.laplace2d(30, bs=4)
    rows = [set(A.colind[A.rowptr[i]:A.rowptr[i + 1]].tolist()) for i in range(A.nb)]
    n = {"one row of 33": 1, "long rows, 2%": 2, "long rows, 10%": 12}[name]
    for q in range(n):
        rows[A.nb - 1 - 5 * q] |= set(range(3 + q, 3 + q + 33 * 3, 3)) if n == 1 else \
            set(range(q, q + 45 * 3, 3))
    return pattern_of(rows)


@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["two wide levels", "a little narrower",
                                  "wide, six dependencies", "wide, a triangle",
                                  "parallel long rows", "one row of 33", "long rows, 2%",
                                  "long rows, 10%"])
def test_bilu0_rule_between_schedules(cuda, orc, name, bs):
    """As test_bilu0_schedules, on both sides of each line of the rule."""
    from isai_kernel_gb300 import api

    rp, col = rule_pattern(name)
    nb, nnzb = len(rp) - 1, len(col)
    rows = np.repeat(np.arange(nb), np.diff(rp))
    val = np.random.default_rng(bs).uniform(-1, 1, size=(nnzb, bs, bs))
    val[rows == col] += 2.0 * bs * np.diff(rp)[:, None, None] * np.eye(bs)
    ref, _ = orc.bsrilu0(nb, bs, rp, col, val)
    out = []
    for schedule in (-1, 0, 1):
        v = T(val, cuda)
        assert api.bsrilu02_inplace(nb, nnzb, bs, T(rp, cuda), T(col, cuda), v, schedule) == -1
        out.append(N(v))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert np.max(np.abs(out[0] - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["5-point", "7-point", "bipartite", "9-point", "dense", "hubs"])
def test_bilu0_block_count_of_the_dependencies(cuda, name, bs):
    """A block count that holds the diagonal and the dependencies, not the blocks
    right of the diagonal, is accepted: the same factor, and one block less is
    refused as long as the level analysis can see it."""
    from isai_kernel_gb300 import api

    rp, col = bilu_pattern(name)
    nb, nnzb = len(rp) - 1, len(col)
    rows = np.repeat(np.arange(nb), np.diff(rp))
    rng = np.random.default_rng(bs)
    val = rng.uniform(-1, 1, size=(nnzb, bs, bs))
    val[rows == col] += 2.0 * bs * np.diff(rp)[:, None, None] * np.eye(bs)
    low = nb + int((col < rows).sum())
    assert low < nnzb
    for schedule in (-1, 0, 1):
        want, got = T(val, cuda), T(val, cuda)
        assert api.bsrilu02_inplace(nb, nnzb, bs, T(rp, cuda), T(col, cuda), want, schedule) == -1
        assert api.bsrilu02_inplace(nb, low, bs, T(rp, cuda), T(col, cuda), got, schedule) == -1
        assert np.array_equal(N(want), N(got))
    with pytest.raises(api.BiluError) as e:
        api.bsrilu02_inplace(nb, low - 1, bs, T(rp, cuda), T(col, cuda), T(val, cuda))
    assert e.value.status == _lib_status("BILU_ERR_WORKSPACE")


def withheld(cuda, A, schedule, row, polls):
    """Status and factor of BILU(0) with `row` never publishing."""
    from isai_kernel_gb300 import _lib, api

    lu = T(A.val, cuda)
    r, c = T(A.rowptr, cuda), T(A.colind, cuda)
    L = _lib.lib()
    ws = api._ws(L.bilu_bsrilu0_ws_bytes(A.nb, A.nnzb), cuda)
    st = L.bilu_debug_bsrilu0_withhold(A.nb, A.nnzb, A.bs, api._p(r), api._p(c), api._p(lu),
                                       schedule, row, polls, api._p(ws), ws.numel(), api._s())
    return st, N(lu)


@pytest.mark.parametrize("name", ["7-point", "9-point", "dense", "hubs"])
def test_bilu0_withheld_row_times_out(cuda, orc, name):
    """Row flow, rows and blocks by ticket with a row that never publishes: the rows
    that wait for it give up, the others leave, and the next call is right."""
    rp, col = bilu_pattern(name)
    nb = len(rp) - 1
    rows = np.repeat(np.arange(nb), np.diff(rp))
    val = np.random.default_rng(1).uniform(-1, 1, size=(len(col), 4, 4))
    val[rows == col] += 8.0 * np.diff(rp)[:, None, None] * np.eye(4)
    A = gen.BSRMatrix(nb, 4, rp, col, val)
    ref, _ = orc.bsrilu0(nb, 4, rp, col, val)
    for schedule in (-1, 1):
        for row in (0, nb // 2):
            assert withheld(cuda, A, schedule, row, 4000)[0] == _lib_status("BILU_ERR_TIMEOUT")
        st, lu = withheld(cuda, A, schedule, -1, 1 << 20)
        assert st == 0 and np.max(np.abs(lu - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("lower", [1, 0])
@pytest.mark.parametrize("name", ["chain", "grid", "dense", "hubs"])
def test_level_analysis_withheld_row_times_out(cuda, name, lower):
    from isai_kernel_gb300 import _lib, api

    rp, col = level_pattern(name)
    nb, nnzb, L = len(rp) - 1, len(col), _lib.lib()
    info = api._ws(L.bilu_sptrsv_analysis_bytes(nb), cuda)
    ws = api._ws(L.bilu_sptrsv_analysis_ws_bytes(nb, nnzb), cuda)
    r, c = T(rp, cuda), T(col, cuda)
    for row in (nb // 3, nb // 2):
        st = L.bilu_debug_sptrsv_analysis_withhold(nb, nnzb, 4, api._p(r), api._p(c), lower, row,
                                                   4000, api._p(info), api._p(ws), ws.numel(),
                                                   api._s())
        assert st == _lib_status("BILU_ERR_TIMEOUT")
    api.call("bilu_sptrsv_analysis", nb, nnzb, 4, api._p(r), api._p(c), lower, api._p(info),
             api._p(ws), ws.numel(), api._s())


@pytest.mark.parametrize("bs", [4, 8])
def test_row_flow_waits_for_a_long_path(cuda, orc, bs):
    """A path of 3000 rows, walked by one warp, in front of 2000 rows that wait
    for its end: their waits last many times the limit, but rows keep finishing.
    With a row of the path withheld they give up."""
    n, fan = 3000, 2000
    rp, col = pattern_of([{max(i - 1, 0), i + 1} if i < n - 1 else
                          {n - 2, *range(n, n + 50)} if i < n else {n - 1}
                          for i in range(n + fan)])
    rng = np.random.default_rng(bs)
    val = rng.uniform(-1, 1, size=(len(col), bs, bs))
    val[np.repeat(np.arange(n + fan), np.diff(rp)) == col] += 8 * bs * np.eye(bs)
    A = gen.BSRMatrix(n + fan, bs, rp, col, val)
    st, lu = withheld(cuda, A, -1, -1, 4000)
    assert st == 0
    LU, _ = orc.bsrilu0(A.nb, bs, rp, col, val)
    assert np.max(np.abs(lu - LU)) <= 1e-12 * np.max(np.abs(LU))
    assert withheld(cuda, A, -1, n // 2, 4000)[0] == -4  # BILU_ERR_TIMEOUT
    assert withheld(cuda, A, -1, -1, 1 << 20)[0] == 0


def test_bilu0_zero_pivot_row(cuda):
    """The first row with a zero pivot is reported by every schedule."""
    from isai_kernel_gb300 import api

    A = gen.laplace2d(9, bs=4)
    val = A.val.copy()
    rows = np.repeat(np.arange(A.nb), np.diff(A.rowptr))
    for bad in (70, 33):
        val[rows == bad] = 0.0
    for schedule in (-1, 0, 1):
        assert api.bsrilu02_inplace(A.nb, A.nnzb, 4, T(A.rowptr, cuda), T(A.colind, cuda),
                                    T(val, cuda), schedule) == 33


# ------------------------------------------------------------------ patterns with long rows
@pytest.mark.parametrize("lower", [True, False])
def test_patterns_rows_walked_by_a_warp(cuda, orc, lower):
    """Rows just below, at and above the length from which a warp shares a
    row, several of them in one warp, against the oracle (integers)."""
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(17)
    n = 150
    length = {3: 47, 4: 48, 5: 49, 6: 110, 40: 149, 149: 120}
    rp, col = pattern_of([rng.choice(n, size=length.get(i, 3), replace=False) for i in range(n)])
    r, c = T(rp, cuda), T(col, cuda)
    mp, mi = api.build_bcsc_pattern_from_bsr_scalarILU(n, r, c, lower)
    omp, omi = orc.isai_pattern(n, rp, col, int(lower))
    assert np.array_equal(N(mp), omp) and np.array_equal(N(mi), omi)
    tr, tc = api.build_triangular_bcsr_pattern_from_A(n, r, c, lower)
    otr, otc = orc.tri_pattern(n, rp, col, int(lower))
    assert np.array_equal(N(tr), otr) and np.array_equal(N(tc), otc)
    # a long row out of order, and one without its diagonal block, are refused
    bad = col.copy()
    bad[rp[40] + 70], bad[rp[40] + 71] = col[rp[40] + 71], col[rp[40] + 70]
    with pytest.raises(api.BiluError):
        api.build_bcsc_pattern_from_bsr_scalarILU(n, r, T(bad, cuda), lower)
    val = np.ones((len(col), 4, 4))
    b = np.ones(4 * n)
    with pytest.raises(api.BiluError):
        api.sptrsv(n, 4, r, T(bad, cuda), T(val, cuda), T(b, cuda), lower)
    rows = np.repeat(np.arange(n), np.diff(rp))
    keep = ~((rows == 6) & (col == 6))
    rp2 = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows[keep], minlength=n), out=rp2[1:])
    with pytest.raises(api.BiluError):
        api.sptrsv(n, 4, T(rp2, cuda), T(col[keep], cuda), T(val[keep], cuda), T(b, cuda), lower)


@pytest.mark.parametrize("level", [1, 2])
@pytest.mark.parametrize("n", [1, 33, 2048, 2049, 5000])
def test_setup_builds_the_step_by_step_factors(cuda, n, level):
    """The setup builds both sides' patterns and pair lists together: the same
    structure as the entry points give one side at a time, and the same values
    (the same kernel on the same pair order).  Sizes around a scan tile."""
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(n)
    length = {5: 47, 6: 48, 7: 49, 20: 110}
    rp, col = pattern_of([rng.choice(n, size=min(length.get(i, 2), n), replace=False)
                          for i in range(n)])
    rows = np.repeat(np.arange(n), np.diff(rp))
    val = rng.standard_normal((len(col), 4, 4))
    i4 = np.arange(4)
    val[np.nonzero(rows == col)[0][:, None], i4, i4] = 8.0 * np.diff(rp)[:, None]
    r, c, v = T(rp, cuda), T(col, cuda), T(val, cuda)
    p = api.Preconditioner(n, 4, r, c, v, fp32=False, isai_level=level)
    lu, L, U = p.factors()
    pr, pc = (r, c) if level == 1 else api.pattern_product(n, r, c, r, c)
    for got, lower in ((L, True), (U, False)):
        mp, mi = api.build_bcsc_pattern_from_bsr_scalarILU(n, pr, pc, lower)
        tr, tc = api.build_triangular_bcsr_pattern_from_A(n, pr, pc, lower)
        assert np.array_equal(N(got[0]), N(tr)) and np.array_equal(N(got[1]), N(tc))
        pp, pl, ps, _ = api.build_pairs(n, r, c, mp, mi, lower)
        m = api.isai_compute(n, 4, lu, mp, mi, pp, pl, ps, api.build_Dinv(n, 4, r, c, lu, lower),
                             lower)
        m = api.reorder_bcsc_val_to_bcsr(api.build_map_bcsc2bcsr_host(n, mp, mi, tr, tc), m)
        assert np.array_equal(N(got[2]), N(m).reshape(-1, 4, 4))
    p.close()
    # a diagonal block that is not stored is refused
    if n > 1:
        keep = ~((rows == n - 1) & (col == n - 1))
        rp2 = np.zeros(n + 1, np.int32)
        np.cumsum(np.bincount(rows[keep], minlength=n), out=rp2[1:])
        with pytest.raises(api.BiluError):
            api.Preconditioner(n, 4, T(rp2, cuda), T(col[keep], cuda), T(val[keep], cuda),
                               isai_level=level)


# ------------------------------------------------------------------ adjoint products
def sparse_rows(name):
    """rowptr, col (no diagonal needed): hub rows and columns, empty rows."""
    rng = np.random.default_rng(23)
    n = 260
    if name == "empty":
        return np.zeros(n + 1, np.int32), np.zeros(0, np.int32)
    if name == "gaps":  # stored rows a long way apart
        rows = [[0, 3, 259] if i in (0, 1, 100, 258) else [] for i in range(n)]
    elif name == "hub column":  # column 7 in every row, columns of 63 to 66 rows
        rows = [[7] + [20 + k for k in range(4) if i < 63 + k] for i in range(n)]
    else:  # "hub row"
        rows = [rng.integers(0, n, size=200 if i == 31 else 3) for i in range(n)]
    cols = [np.unique(np.array(r, np.int32)) for r in rows]
    rp = np.zeros(n + 1, np.int32)
    np.cumsum([len(c) for c in cols], out=rp[1:])
    return rp, np.concatenate(cols).astype(np.int32)


@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["gaps", "hub column", "hub row"])
def test_transposed_product(cuda, name, bs):
    """M^T x against dense FP64: sums of up to 260 bs products of numbers in
    [-1, 1], so 1e-13 of the number of terms."""
    from isai_kernel_gb300 import api

    rp, col = sparse_rows(name)
    nb = len(rp) - 1
    rng = np.random.default_rng(bs)
    val, x = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=nb * bs)
    y = N(api.bcsr_spmv_transpose(nb, bs, T(rp, cuda), T(col, cuda), T(val, cuda), T(x, cuda)))
    D = np.zeros((nb, bs, nb, bs))
    D[np.repeat(np.arange(nb), np.diff(rp)), :, col, :] = val
    assert np.max(np.abs(y - D.reshape(nb * bs, -1).T @ x)) <= 1e-13 * 260 * bs
    bad = col.copy()
    bad[-1] = nb
    with pytest.raises(api.BiluError):
        api.bcsr_spmv_transpose(nb, bs, T(rp, cuda), T(bad, cuda), T(val, cuda), T(x, cuda))


@pytest.mark.parametrize("mb", [1, 31, 9727, 9728, 9729, 20000])
def test_transposed_pattern_hub_columns(cuda, mb):
    """Neighbouring dense columns (up to 9728 segments: a warp each) and short
    ones: the transposed pattern and blocks."""
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(mb)
    hubs = {c for c in (0, 1, 2, 3, mb // 2, mb - 2, mb - 1) if 0 <= c < mb}
    rp, col = pattern_of([hubs | {int(rng.integers(0, mb))} if i < 500 else {(7 * i) % mb}
                          for i in range(mb)])
    val = rng.uniform(-1, 1, size=(len(col), 4, 4))
    tr, tc, tv = api.bsr_transpose(mb, 4, T(rp, cuda), T(col, cuda), T(val, cuda))
    rows = np.repeat(np.arange(mb), np.diff(rp))
    order = np.lexsort((rows, col))
    want = np.zeros(mb + 1, np.int64)
    np.cumsum(np.bincount(col, minlength=mb), out=want[1:])
    assert np.array_equal(N(tr), want) and np.array_equal(N(tc), rows[order])
    assert np.array_equal(N(tv), val[order].transpose(0, 2, 1))


@pytest.mark.parametrize("scale", [1.0, -1.0, 2.5])
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("name", ["empty", "gaps", "hub column", "hub row"])
def test_masked_outer_runs(cuda, name, bs, scale):
    """Bit for bit: (scale u) v is one rounding (two for a general scale, in
    the same order), adding to G one more."""
    from isai_kernel_gb300 import api

    rp, col = sparse_rows(name)
    nb = len(rp) - 1
    rng = np.random.default_rng(bs)
    u, v = rng.uniform(-1, 1, size=nb * bs), rng.uniform(-1, 1, size=nb * bs)
    G0 = rng.uniform(-1, 1, size=(len(col), bs, bs))
    rows = np.repeat(np.arange(nb), np.diff(rp))
    ref = (scale * u.reshape(nb, bs)[rows])[:, :, None] * v.reshape(nb, bs)[col][:, None, :]
    args = (nb, bs, T(rp, cuda), T(col, cuda), T(u, cuda), T(v, cuda), scale)
    assert np.array_equal(N(api.masked_outer(*args)), ref)
    added = N(api.masked_outer(*args, G=T(G0, cuda)))
    assert np.max(np.abs(added - (G0 + ref)), initial=0.0) <= 2.0 ** -52 * 3  # fused or not


# ------------------------------------------------------------------ uneven rows
def uneven_pattern(name):
    """Row lengths around the splits: (nb, longest) per name."""
    rng = np.random.default_rng(29)
    n = {"one hub": 70, "hubs": 1500, "all long": 66, "big": 9000}[name]
    length = rng.integers(0, 5, size=n)
    if name == "one hub":
        length[33] = 70
    elif name == "all long":
        length[:] = 66
    else:
        length[rng.integers(0, n, size=n // 60)] = rng.integers(40, 100, size=n // 60)
        length[[0, n // 2, n - 1]] = min(n, 1400)
    cols = [np.sort(rng.choice(n, size=k, replace=False)) for k in length]
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(length, out=rp[1:])
    return rp, np.concatenate(cols).astype(np.int32)


@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["one hub", "hubs", "all long", "big"])
def test_uneven_rows_product(cuda, orc, name, bs):
    """Products over rows of 0 to 1400 blocks (empty rows among them).  FP64:
    a sum of N products of numbers in [-1, 1] is within N 2^-53 (N of them) of
    any other order.  FP32: against the same bound at 2^-24; the same call
    twice gives the same bits."""
    import torch

    from isai_kernel_gb300 import api

    rp, col = uneven_pattern(name)
    nb = len(rp) - 1
    rng = np.random.default_rng(bs)
    val, x = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=nb * bs)
    terms = np.repeat(np.diff(rp) * bs, bs).astype(float)
    ref = orc.bcsr_spmv(nb, bs, rp, col, val, x)
    r, c, v, xd = T(rp, cuda), T(col, cuda), T(val, cuda), T(x, cuda)
    y = api.bcsr_spmv(nb, bs, r, c, v, xd)
    assert torch.equal(y, api.bcsr_spmv(nb, bs, r, c, v, xd))
    assert np.all(np.abs(N(y) - ref) <= terms * terms * 2.0 ** -53)
    v32 = v.float()
    ref32 = orc.bcsr_spmv(nb, bs, rp, col, N(v32).astype(np.float64), N(xd.float()).astype(np.float64))
    y32 = api.bcsr_spmv(nb, bs, r, c, v32, xd.float())
    assert torch.equal(y32, api.bcsr_spmv(nb, bs, r, c, v32, xd.float()))
    assert np.all(np.abs(N(y32) - ref32) <= terms * terms * 2.0 ** -24)


# ------------------------------------------------------------------ several right-hand sides
@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("mb, hubs, ln", [(80, 1, 65), (608, 3, 65), (609, 40, 66), (700, 3, 64),
                                          (5000, 30, 250), (9000, 8, 300), (300, 300, 100),
                                          (12000, 12000, 70), (5000, 5000, 33)])
def test_products_of_few_long_rows(cuda, bs, mb, hubs, ln):
    """Neighbouring rows of `ln` blocks among rows of two, and patterns of one row
    length: the products of every combination of types, N terms of numbers in
    [-1, 1] each within N^2 2^-53 (FP32 values: 2^-24) of the sum in 64 bits."""
    import torch

    from isai_kernel_gb300 import api

    rng = np.random.default_rng(mb + bs + ln)
    n = np.full(mb, 2)
    n[mb - hubs:] = ln
    rp = np.zeros(mb + 1, np.int32)
    np.cumsum(n, out=rp[1:])
    rows = np.repeat(np.arange(mb), n)
    col = rng.integers(0, mb, size=len(rows)).astype(np.int32)
    val, x = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=mb * bs)
    r, c, v, xd = T(rp, cuda), T(col, cuda), T(val, cuda), T(x, cuda)
    bound = 2 * ((n * bs).astype(float) ** 2)[:, None]

    def product(a, b):
        ref = np.zeros((mb, bs))
        np.add.at(ref, rows, np.einsum("pij,pj->pi", a, b.reshape(mb, bs)[col]))
        return ref

    y = N(api.bcsr_spmv(mb, bs, r, c, v, xd)).reshape(mb, bs)
    assert np.all(np.abs(y - product(val, x)) <= bound * 2.0 ** -53)
    v32 = v.float()
    ref = product(N(v32).astype(np.float64), x.astype(np.float32).astype(np.float64))
    for xt in (torch.float32, torch.float64):
        for yt in (torch.float32, torch.float64):
            out = torch.full((mb * bs,), float("nan"), dtype=yt, device=cuda)
            y = N(api.bcsr_spmv(mb, bs, r, c, v32, xd.to(xt), out)).reshape(mb, bs)
            # (an FP64 x is rounded where it is read)
            assert np.all(np.abs(y - ref) <= bound * 2.0 ** -24)


@pytest.mark.parametrize("k", [1, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("bs", [4, 5, 8])
def test_spmm_splits(cuda, orc, bs, k):
    """Every lane split at its edges, over rows of 0 to 70 blocks, against the
    column-by-column product: N products of numbers in [-1, 1] are within
    N 2^-53 (2^-24 for FP32-stored values) of any order, N of them.  A
    right-hand side of zeros, infinities and subnormals converts as IEEE says."""
    import torch

    from isai_kernel_gb300 import api

    rp, col = uneven_pattern("one hub")
    nb = len(rp) - 1
    rng = np.random.default_rng(100 * bs + k)
    val, X = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=(nb * bs, k))
    terms = (np.repeat(np.diff(rp) * bs, bs).astype(float) ** 2)[:, None]
    r, c, v = T(rp, cuda), T(col, cuda), T(val, cuda)
    D = np.zeros((nb, bs, nb, bs))
    rows = np.repeat(np.arange(nb), np.diff(rp))
    D[rows, :, col, :] = val
    Y = N(api.bcsr_spmm(nb, bs, r, c, v, T(X, cuda)))
    assert np.all(np.abs(Y - D.reshape(nb * bs, -1) @ X) <= terms * 2.0 ** -53 * 2)
    v32 = v.float()
    D[rows, :, col, :] = N(v32)
    Y32 = N(api.bcsr_spmm(nb, bs, r, c, v32, T(X, cuda)))
    ref = D.reshape(nb * bs, -1) @ X.astype(np.float32).astype(np.float64)
    assert np.all(np.abs(Y32 - ref) <= terms * 2.0 ** -24 * 2)
    # values that start off a 16-byte boundary
    odd = torch.empty(v32.numel() + 1, dtype=torch.float32, device=cuda)[1:].view_as(v32)
    odd.copy_(v32)
    assert np.array_equal(N(api.bcsr_spmm(nb, bs, r, c, odd, T(X, cuda))), Y32)
    # one identity block per row: Y is X rounded to FP32
    n = nb * bs
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, -1e-45, 1e39, 3.4028235677973366e38,
                        1.1754943508222875e-38, 1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24, -1e-310])
    Xs = np.resize(special, (n, 1)).repeat(k, axis=1)
    eye = np.zeros((nb, 1, 1)) + np.eye(bs)
    # (0 * inf: keep one special value per block row)
    Xs[np.arange(n) % bs != 0] = 0.0
    got = N(api.bcsr_spmm(nb, bs, T(np.arange(nb + 1, dtype=np.int32), cuda),
                          T(np.arange(nb, dtype=np.int32), cuda), T(eye, cuda).float(),
                          T(Xs, cuda)))[::bs]
    with np.errstate(over="ignore"):
        want = Xs[::bs].astype(np.float32).astype(np.float64)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("k", [1, 33])
@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("mb, ncol, repeated", [(3, 200, False), (64, 65, False), (65, 300, False),
                                                (16, 16, True)])
def test_spmm_few_rows_of_many_blocks(cuda, bs, k, mb, ncol, repeated):
    """Slices with more block columns than block rows, and rows that hold a
    column several times: every row of Y is written, by the sum of its blocks
    (bounds as in test_spmm_splits)."""
    import torch

    from isai_kernel_gb300 import api

    rng = np.random.default_rng(1000 * mb + 10 * bs + k)
    cols = [np.sort(rng.integers(0, ncol, size=90)) if repeated else np.arange(ncol)
            for _ in range(mb)]
    rp = np.zeros(mb + 1, np.int32)
    np.cumsum([len(c) for c in cols], out=rp[1:])
    col = np.concatenate(cols).astype(np.int32)
    val, X = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=(ncol * bs, k))
    rows = np.repeat(np.arange(mb), np.diff(rp))
    r, c, x = T(rp, cuda), T(col, cuda), T(X, cuda)
    bound = 2 * (np.repeat(np.diff(rp) * bs, bs).astype(float) ** 2)[:, None]
    for dtype, eps in ((torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)):
        v = T(val, cuda).to(dtype)
        D = np.zeros((mb, bs, ncol, bs))
        np.add.at(D, (rows, slice(None), col, slice(None)), N(v).astype(np.float64))
        Xr = X if dtype == torch.float64 else X.astype(np.float32).astype(np.float64)
        Y = torch.full((mb * bs, k), float("nan"), dtype=torch.float64, device=cuda)
        api.call("bilu_bcsr_spmm" if dtype == torch.float64 else "bilu_bcsr_spmm_f32", mb, bs, k,
                 api._p(r), api._p(c), api._p(v), api._p(x), api._p(Y), api._s())
        assert np.all(np.abs(N(Y) - D.reshape(mb * bs, -1) @ Xr) <= bound * eps)


@pytest.mark.parametrize("k", [1, 6, 33])
@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("mb, hubs, ln", [(65, 65, 65), (608, 9, 64), (608, 9, 65), (609, 9, 65),
                                          (1217, 1217, 67), (1300, 1300, 131), (5000, 20, 300)])
def test_spmm_hub_rows(cuda, bs, k, mb, hubs, ln):
    """Neighbouring rows of `ln` blocks among rows of two: as ordinary rows (64
    blocks; rows all alike) and each by a CTA, on matrices around the sizes where
    a CTA looks through one, two and more rows at a time (bounds as in
    test_spmm_splits)."""
    import torch

    from isai_kernel_gb300 import api

    rng = np.random.default_rng(mb + 10 * bs + k + ln)
    n = np.full(mb, 2)
    n[mb - hubs:] = ln
    rp = np.zeros(mb + 1, np.int32)
    np.cumsum(n, out=rp[1:])
    rows = np.repeat(np.arange(mb), n)
    col = rng.integers(0, mb, size=len(rows)).astype(np.int32)
    val, X = rng.uniform(-1, 1, size=(len(col), bs, bs)), rng.uniform(-1, 1, size=(mb * bs, k))
    r, c = T(rp, cuda), T(col, cuda)
    bound = 2 * ((n * bs).astype(float) ** 2)[:, None, None]
    for dtype, eps in ((torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)):
        v = T(val, cuda).to(dtype)
        Xr = X if dtype == torch.float64 else X.astype(np.float32).astype(np.float64)
        ref = np.zeros((mb, bs, k))
        np.add.at(ref, rows, np.einsum("pij,pjk->pik", N(v).astype(np.float64),
                                       Xr.reshape(mb, bs, k)[col]))
        Y = N(api.bcsr_spmm(mb, bs, r, c, v, T(X, cuda))).reshape(mb, bs, k)
        assert np.all(np.abs(Y - ref) <= bound * eps)


# ------------------------------------------------------------------ rows of mixed lengths
@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("n", [1, 6, 31, 1000])
def test_fp64_product_mixed_rows(cuda, n, bs):
    """The FP64 product and its transpose with rows of 0 to 9 blocks side by
    side in a warp, the last warp partly filled, against numpy: at most 72
    products a sum, so 72 eps of the sum of their magnitudes."""
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(n)
    cols = [np.sort(rng.choice(n, size=min(n, int(rng.integers(0, 10))), replace=False))
            for _ in range(n)]
    cols[0] = np.arange(min(n, 3))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum([len(c) for c in cols], out=rp[1:])
    col = np.concatenate(cols).astype(np.int32)
    val, x = rng.standard_normal((len(col), bs, bs)), rng.standard_normal((n, bs))
    rows = np.repeat(np.arange(n), np.diff(rp))
    for transpose in (False, True):
        ref, mag = np.zeros((n, bs)), np.zeros((n, bs))
        to, at = (col, rows) if transpose else (rows, col)
        v = val.transpose(0, 2, 1) if transpose else val
        np.add.at(ref, to, np.einsum("pij,pj->pi", v, x[at]))
        np.add.at(mag, to, np.einsum("pij,pj->pi", np.abs(v), np.abs(x[at])))
        f = api.bcsr_spmv_transpose if transpose else api.bcsr_spmv
        got = N(f(n, bs, T(rp, cuda), T(col, cuda), T(val, cuda), T(x.ravel(), cuda)))
        most = max(int(np.bincount(to, minlength=n).max()) * bs, 72)
        assert np.all(np.abs(got.reshape(n, bs) - ref) <= 2 * most * 1.2e-16 * mag + 1e-300)


# ------------------------------------------------------------------ products one after another
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("bs", [4, 5, 8])
@pytest.mark.parametrize("name", ["gaps", "hub row", "grid"])
def test_apply_starts_before_the_first_product_ends(cuda, name, bs, fp32):
    """The second product of the apply is started while the first one drains:
    it has to give the bits of two separate products, with rows without blocks,
    when the matrices, b and the buffers change right before the call, on a side
    stream, and replayed from a graph."""
    import torch

    from isai_kernel_gb300 import api

    if name == "grid":
        A = gen.convdiff3d(23, bs=4)
        rp, col, n = A.rowptr, A.colind, A.nb
    else:
        rp, col = sparse_rows(name)
        n = len(rp) - 1
    dt = torch.float32 if fp32 else torch.float64
    r, c = T(rp, cuda), T(col, cuda)
    g = torch.Generator(device=cuda).manual_seed(5)
    rand = lambda *s: torch.randn(*s, dtype=torch.float64, device=cuda, generator=g)
    vl, vu, b = rand(len(col), bs, bs).to(dt), rand(len(col), bs, bs).to(dt), rand(n * bs)
    prec = api.BILU_FP32 if fp32 else api.BILU_FP64

    def both():
        got = api.isai_apply(n, bs, (r, c, vl), (r, c, vu), b, prec)
        y = api.bcsr_spmv(n, bs, r, c, vl, b.to(dt))
        x = torch.empty_like(b)
        return got, api.bcsr_spmv(n, bs, r, c, vu, y, x)

    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(8):
                vl.mul_(-0.5)
                vu.add_(vl)
                b.neg_()
                got, ref = both()
                assert torch.equal(got, ref)
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = api.isai_apply(n, bs, (r, c, vl), (r, c, vu), b, prec)
    for _ in range(3):
        vu.mul_(-0.25)
        b.add_(1.0)
        graph.replay()
        assert torch.equal(got, both()[1])


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("bs", [4, 5, 8])
def test_hub_kernels_keep_the_stream_order(cuda, bs, fp32):
    """The hub rows' kernels start beside the other rows' one: what is written right
    before a product is read by both, what follows sees both, on the current and a
    side stream and replayed from a graph; the bits are those of a product on its
    own."""
    import torch

    from isai_kernel_gb300 import api

    mb, k = 7000, 9
    n = np.full(mb, 3)
    n[1000:1012] = 200
    rp = np.zeros(mb + 1, np.int32)
    np.cumsum(n, out=rp[1:])
    g = torch.Generator(device=cuda).manual_seed(bs)
    rand = lambda *s: torch.randn(*s, dtype=torch.float64, device=cuda, generator=g)
    col = np.random.default_rng(bs).integers(0, mb, size=rp[-1]).astype(np.int32)
    dt = torch.float32 if fp32 else torch.float64
    r, c, v = T(rp, cuda), T(col, cuda), rand(len(col), bs, bs).to(dt)
    X, x = rand(mb * bs, k), rand(mb * bs).to(dt)

    def chain():
        Y = api.bcsr_spmm(mb, bs, r, c, v, X)
        y = api.bcsr_spmv(mb, bs, r, c, v, x)
        # each result goes straight into the next product
        return Y, api.bcsr_spmm(mb, bs, r, c, v, Y), y, api.bcsr_spmv(mb, bs, r, c, v, y)

    def apart():
        out = []
        for f, a in ((api.bcsr_spmm, X), (api.bcsr_spmv, x)):
            for _ in range(2):
                torch.cuda.synchronize()
                a = f(mb, bs, r, c, v, a)
                torch.cuda.synchronize()
                out.append(a)
        return out

    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(8):
                v.mul_(-0.5)
                X.add_(0.25)
                x.neg_()
                got = chain()
                assert all(torch.equal(a, b) for a, b in zip(got, apart()))
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain()
    for _ in range(3):
        v.mul_(-1.5)
        X.neg_()
        x.add_(1.0)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, apart()))


# ------------------------------------------------------------------ orthogonalisation
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("per_thread", [0, 2, 4, 6, 7])
def test_mgs_step_forms(cuda, fp32, per_thread):
    """n one element below, at and above what fills 2, 4 and 6 vectors a thread
    of two 512-thread CTAs per SM (where the kernel's form changes), against
    the same Gram-Schmidt in FP64: v_{j+1} within 1e-12 (FP32 2e-5) of its
    largest element.  (h_i carries the rounding of a sum of |v_i| |w|: some
    50 eps sqrt(n), that is 50 eps of an element of w after h_i v_i.)"""
    import torch

    from isai_kernel_gb300 import _lib, api

    L = _lib.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    full = sms * 1024 * (4 if fp32 else 2) * max(per_thread, 1)
    dt, tol = (torch.float32, 2e-5) if fp32 else (torch.float64, 1e-12)
    j = 2
    for n in ((1, 7, 513) if per_thread == 0 else (full - 1, full, full + 5)):
        gen_ = torch.Generator(device=cuda).manual_seed(n)
        j = min(2, n - 1)
        B = torch.randn(n, j + 1, dtype=torch.float64, device=cuda, generator=gen_)
        Q = torch.linalg.qr(B)[0].T.contiguous()
        ldv = (n + 31) // 32 * 32
        V = torch.zeros(j + 1, ldv, dtype=dt, device=cuda)
        V[:, :n] = Q.to(dt)
        w = torch.zeros(ldv, dtype=dt, device=cuda)
        w[:n] = torch.randn(n, dtype=torch.float64, device=cuda, generator=gen_).to(dt)
        wr, Vr = w[:n].double().clone(), V[:, :n].double()  # the kernel uses w up
        h = torch.empty(j + 2, dtype=torch.float64, device=cuda)
        vn = torch.zeros_like(w)
        ws = torch.empty(L.bilu_debug_mgs_step_ws_bytes(), dtype=torch.uint8, device=cuda)
        assert L.bilu_debug_mgs_step(n, fp32, api._p(V), ldv, j, api._p(w), api._p(h),
                                     api._p(vn), api._p(ws), ws.numel(), api._s()) == 0
        for i in range(j + 1):
            hi = Vr[i] @ wr
            assert abs(hi - h[i]) <= tol * n ** 0.5
            wr = wr - hi * Vr[i]
        if n == 1:  # nothing is left but rounding
            continue
        ref = wr / wr.norm()
        assert (vn[:n].double() - ref).abs().max() <= tol * ref.abs().max()
        assert torch.all(vn[n:] == 0)


def step_vectors(cuda, fp32, n, j):
    """V (rows of ldv elements), w and the workspace of a Gram-Schmidt step."""
    import torch

    from isai_kernel_gb300 import _lib

    g = torch.Generator(device=cuda).manual_seed(n)
    dt = torch.float32 if fp32 else torch.float64
    ldv = (n + 31) // 32 * 32
    V = torch.zeros(j + 1, ldv, dtype=dt, device=cuda)
    V[:, :n] = torch.linalg.qr(
        torch.randn(n, j + 1, dtype=torch.float64, device=cuda, generator=g))[0].T.to(dt)
    w = torch.zeros(ldv, dtype=dt, device=cuda)
    w[:n] = torch.randn(n, dtype=torch.float64, device=cuda, generator=g).to(dt)
    ws = torch.empty(_lib.lib().bilu_debug_mgs_step_ws_bytes(), dtype=torch.uint8, device=cuda)
    return V, w, ws


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("n", [513, 300001, 1500002, 2500003, 4000001])
def test_mgs_step_leaves_the_orthogonalised_vector(cuda, fp32, n):
    """Every form of the step (up to 2, 4 and 6 vectors a thread, and more) leaves
    w - sum h_i v_i in w: v_{j+1} is that over the square root of h_{j+1}, one
    rounded product per element (root, quotient and product: 4 eps)."""
    import torch

    from isai_kernel_gb300 import _lib, api

    j = 2
    V, w, ws = step_vectors(cuda, fp32, n, j)
    h = torch.empty(j + 2, dtype=torch.float64, device=cuda)
    vn = torch.zeros_like(w)
    assert _lib.lib().bilu_debug_mgs_step(n, fp32, api._p(V), V.shape[1], j, api._p(w), api._p(h),
                                          api._p(vn), api._p(ws), ws.numel(), api._s()) == 0
    eps = torch.finfo(w.dtype).eps
    want = w[:n].double() / h[j + 1].sqrt()
    assert torch.all((vn[:n].double() - want).abs() <= 4 * eps * want.abs())
    assert abs(h[j + 1] - (w[:n].double() ** 2).sum()) <= eps * n ** 0.5 * h[j + 1]


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("n", [513, 300001, 1500002])
def test_mgs_step_forms_give_the_same_bits(cuda, fp32, n):
    """The streaming and the resident form: h, ||w||^2, v_{j+1} and w."""
    import torch

    from isai_kernel_gb300 import _lib, api

    j, out = 3, []
    for streaming in (1, 0):
        V, w, ws = step_vectors(cuda, fp32, n, j)
        h = torch.empty(j + 2, dtype=torch.float64, device=cuda)
        vn = torch.zeros_like(w)
        assert _lib.lib().bilu_debug_mgs_step_ex(
            n, fp32, api._p(V), V.shape[1], j, api._p(w), api._p(h), api._p(vn), streaming, -1,
            1 << 20, api._p(ws), ws.numel(), api._s()) == 0
        out.append((h, vn, w))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("streaming", [0, 1])
@pytest.mark.parametrize("cta", [0, 1, 200])
def test_mgs_step_withheld_sum_times_out(cuda, fp32, streaming, cta):
    """A CTA that never stores its sums: every wait gives up, the call says so,
    and the next one on the same workspace is right."""
    import torch

    from isai_kernel_gb300 import _lib, api

    n, j, L = 300001, 2, _lib.lib()
    V, w, ws = step_vectors(cuda, fp32, n, j)
    h = torch.empty(j + 2, dtype=torch.float64, device=cuda)
    vn = torch.zeros_like(w)
    st = L.bilu_debug_mgs_step_ex(n, fp32, api._p(V), V.shape[1], j, api._p(w.clone()), api._p(h),
                                  api._p(vn), streaming, cta, 2000, api._p(ws), ws.numel(),
                                  api._s())
    assert st == _lib_status("BILU_ERR_TIMEOUT")
    assert L.bilu_debug_mgs_step(n, fp32, api._p(V), V.shape[1], j, api._p(w), api._p(h),
                                 api._p(vn), api._p(ws), ws.numel(), api._s()) == 0
    eps = torch.finfo(w.dtype).eps
    assert torch.all((V[:, :n].double() @ vn[:n].double()).abs() <= 50 * eps * n ** 0.5)


# ------------------------------------------------------------------ conversion
@pytest.mark.parametrize("shift_in, shift_out", [(0, 0), (1, 0), (0, 1), (2, 4)])
def test_values_to_fp32(cuda, shift_in, shift_out):
    """bilu_convert_f64_to_f32 on sizes and starts with and without whole
    16-byte groups, bit for bit the rounding of the type conversion (zeros,
    subnormals, overflow, infinities and NaN included)."""
    import torch

    from isai_kernel_gb300 import api

    g = torch.Generator(device=cuda).manual_seed(1)
    special = torch.tensor([0.0, -0.0, 1e-310, 1e-46, 1.4e-45, -3e-39, 3.5e38, -1e300, float("inf"),
                            float("-inf"), float("nan"), 1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24],
                           dtype=torch.float64, device=cuda)
    for n in (1, 3, 4, 5, 1021, 300000):
        src = torch.randn(n + shift_in, dtype=torch.float64, device=cuda, generator=g)
        k = min(n, len(special))
        src[shift_in:shift_in + k] = special[:k]
        out = torch.full((n + shift_out + 3,), 7.0, dtype=torch.float32, device=cuda)
        api.call("bilu_convert_f64_to_f32", n, src.data_ptr() + 8 * shift_in,
                 out.data_ptr() + 4 * shift_out, api._s())
        ref = src[shift_in:].float()
        got = out[shift_out:shift_out + n]
        same = (got.view(torch.int32) == ref.view(torch.int32)) | (got.isnan() & ref.isnan())
        assert bool(same.all())
        assert bool((out[:shift_out] == 7).all()) and bool((out[shift_out + n:] == 7).all())
