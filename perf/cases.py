"""The measured cases: what a user of the block-ILU(0) + ISAI engine has it do.

Each case is one call (or the few calls that belong together) through the
package's public functions, on inputs that are made on the GPU from a seed:

* ``apply``     x = M_U (M_L b), the preconditioner apply of a Krylov step
* ``spmm``      Y = A X, several right-hand sides at once
* ``convert``   scalar CSR to BSR, the first step from a Matrix Market file
* ``setup``     the whole preconditioner setup from a BSR matrix: BILU(0),
                ISAI patterns and pair lists, the ISAI factors
* ``trisolve``  y = L^-1 b, x = U^-1 y on a packed factor (the exact apply)
* ``adjoint``   forward and backward of the differentiable ISAI apply or of
                the differentiable exact solve
* ``solve``     preconditioned (F)GMRES on a handle that is already set up

The systems are those of ``isai_kernel_gb300.gen`` (2D 5-point Laplacian with
coupled unknowns, 3D upwinded convection-diffusion, power-law block matrix),
rebuilt with torch so that a large one takes milliseconds.  A pattern depends
on the case's sizes alone, values and right-hand sides on the seed.
"""
from __future__ import annotations

import functools

import torch

from isai_kernel_gb300 import api, autograd as ag

DEV = "cuda"
F64, F32, I32 = torch.float64, torch.float32, torch.int32
PREC = {"fp64": api.BILU_FP64, "fp32": api.BILU_FP32, "ilu": api.BILU_ILU,
        "ilu_fp32": api.BILU_ILU_FP32, "nested": api.BILU_NESTED}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one apply of the 64 x 64 configuration: the smallest call, where a
        # launch's latency is most of the time
        dict(name="apply 64x64", op="apply", grid="64x64", bs=4, prec="fp64"),
        # an ordinary apply at the block size of the prototype, ragged sides
        dict(name="apply bs5", op="apply", grid="47x43x41", bs=5, prec="fp64"),
        # the mixed-precision apply of the 128^3 headline system
        dict(name="apply 128^3 fp32", op="apply", grid="128x128x128", bs=4, prec="fp32"),
        # the apply on the 500,000-unknown power-law configuration: rows of a
        # few to two thousand 8x8 blocks
        dict(name="apply powerlaw", op="apply", powerlaw=62500, bs=8, prec="fp64"),
        # 32 right-hand sides on the largest grid of the batch configuration,
        # FP32-stored values
        dict(name="spmm fp32", op="spmm", grid="512x512", bs=4, prec="fp32", k=32),
        # a scalar CSR matrix with partly filled 5x5 blocks to BSR
        dict(name="csr to bsr", op="convert", grid="50x50x50", bs=5, fill=0.8),
        # setup of the nested solver on a mid-sized 3D system
        dict(name="setup 64^3", op="setup", grid="64x64x64", bs=4, mode="nested", level=1),
        # setup on an irregular pattern (narrow levels, hub rows)
        dict(name="setup powerlaw", op="setup", powerlaw=20011, bs=8, mode="fp64", level=1),
        # both triangular solves of the exact preconditioner, one-shot form
        dict(name="trisolve 64^3", op="trisolve", grid="64x64x64", bs=4),
        # a training step through the apply: gradients of b and both factors
        dict(name="adjoint isai", op="adjoint", kind="isai", grid="40x40x40", bs=5),
        # a training step through the exact solve
        dict(name="adjoint ilu", op="adjoint", kind="ilu", grid="256x256", bs=4),
        # the headline call on a mid-sized system: nested GMRES to 1e-10
        dict(name="solve nested", op="solve", grid="64x64x64", bs=4, prec="nested"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_pattern(rng, lo, hi, grids=False):
    """A pattern of about lo..hi block rows, ragged sides."""
    nb = _log(rng, lo, hi)
    t = rng.randrange(1 if grids else 0, 5)
    if t == 0:
        return dict(powerlaw=max(64, min(nb, 62500)))
    if t <= 2:
        x = max(8, int(nb ** 0.5 * rng.uniform(0.6, 1.5)))
        return dict(grid="%dx%d" % (x, max(8, nb // x)))
    x = max(6, int(nb ** (1 / 3) * rng.uniform(0.7, 1.3)))
    y = max(6, int(nb ** (1 / 3) * rng.uniform(0.7, 1.3)))
    return dict(grid="%dx%dx%d" % (x, y, max(6, nb // (x * y))))


def draw(rng):
    op = rng.choice(["apply", "apply", "spmm", "convert", "setup", "trisolve", "adjoint", "solve"])
    bs = rng.choice([4, 5, 8])
    if op == "apply":
        return dict(op=op, **_draw_pattern(rng, 1000, 1000000 if bs == 4 else 300000), bs=bs,
                    prec=rng.choice(["fp64", "fp32"]))
    if op == "spmm":
        return dict(op=op, **_draw_pattern(rng, 1000, 200000 if bs == 4 else 80000), bs=bs,
                    prec=rng.choice(["fp64", "fp32"]), k=rng.choice([1, 2, 7, 16, 32, 33, 64]))
    if op == "convert":
        # files of assembled grids: a hub row of thousands of scalar entries
        # takes seconds
        return dict(op=op, **_draw_pattern(rng, 1000, 100000 if bs < 8 else 40000, grids=True),
                    bs=bs, fill=rng.choice([1.0, 0.8, 0.4]))
    if op == "setup":
        level = rng.choice([1, 1, 2])
        p = _draw_pattern(rng, 500, 200000 if level == 1 else 30000)
        if "powerlaw" in p:
            p, level = dict(powerlaw=min(p["powerlaw"], 20000)), 1
        return dict(op=op, **p, bs=bs, mode=rng.choice(["fp64", "fp32", "nested"]), level=level)
    if op == "trisolve":
        return dict(op=op, **_draw_pattern(rng, 500, 200000 if bs < 8 else 60000), bs=bs)
    if op == "adjoint":
        return dict(op=op, kind=rng.choice(["isai", "ilu"]),
                    **_draw_pattern(rng, 500, 100000 if bs < 8 else 40000), bs=bs)
    # convection-diffusion only: GMRES(30) stagnates on the larger Laplacians
    # with random couplings whatever the preconditioner
    s = [max(8, _log(rng, 8, 64)) for _ in range(3)]
    return dict(op=op, grid="%dx%dx%d" % tuple(s), bs=bs if s[0] * s[1] * s[2] < 60000 else 4,
                prec=rng.choice(["nested", "nested", "fp64", "fp32", "ilu", "ilu_fp32"]))


# ------------------------------------------------------------------ patterns
class Pattern:
    """rowptr, col (int32), row of every block (int64) and, for the grids,
    each block's stencil coefficient."""

    def __init__(self, rows, cols, nb, coef=None):
        self.nb = nb
        self.row, self.col, self.coef = rows, cols, coef
        self.rowptr = torch.zeros(nb + 1, dtype=torch.int64, device=rows.device)
        self.rowptr[1:] = torch.bincount(rows, minlength=nb).cumsum(0)
        self.nnzb = int(cols.numel())

    def csr(self):
        return self.rowptr.to(I32), self.col.to(I32)

    def part(self, keep):
        return Pattern(self.row[keep], self.col[keep], self.nb,
                       None if self.coef is None else self.coef[keep])


def _grid(dims):
    nb = 1
    for d in dims:
        nb *= d
    node = torch.arange(nb, device=DEV)
    x, y = node % dims[0], node // dims[0] % dims[1]
    s2 = dims[0] * dims[1]
    every = torch.ones(nb, dtype=torch.bool, device=DEV)
    if len(dims) == 2:
        legs = [(-dims[0], y > 0, -1.0), (-1, x > 0, -1.0), (0, every, 4.0),
                (1, x < dims[0] - 1, -1.0), (dims[0], y < dims[1] - 1, -1.0)]
    else:
        z = node // s2
        # upwinded, cell Peclet 10 along x, 5 along y, 2.5 along z
        legs = [(-s2, z > 0, -3.5), (-dims[0], y > 0, -6.0), (-1, x > 0, -11.0),
                (0, every, 23.5), (1, x < dims[0] - 1, -1.0),
                (dims[0], y < dims[1] - 1, -1.0), (s2, z < dims[2] - 1, -1.0)]
    on = torch.stack([m for _, m, _ in legs], 1)
    cols = torch.stack([node + o for o, _, _ in legs], 1)[on]
    coef = torch.tensor([c for _, _, c in legs], dtype=F64, device=DEV).expand(nb, -1)[on]
    rows = node[:, None].expand(-1, len(legs))[on]
    return Pattern(rows, cols, nb, coef)


def _powerlaw(nb):
    """Off-diagonal blocks per row ~ k^-2.1 up to 2000, mean 12, uniform columns."""
    g = torch.Generator(device=DEV).manual_seed(nb)
    k = torch.arange(1, 2001, dtype=F64, device=DEV)
    p = k ** -2.1
    p /= p.sum()
    raw = torch.multinomial(p, nb, replacement=True, generator=g) + 1
    cnt = (raw * (12.0 / float((k * p).sum()))).round().clamp(1, min(2000, nb - 1)).long()
    rows = torch.repeat_interleave(torch.arange(nb, device=DEV), cnt)
    c = torch.randint(0, nb - 1, (rows.numel(),), device=DEV, generator=g)
    c = c + (c >= rows)
    every = torch.arange(nb, device=DEV)
    key = torch.unique(torch.cat([rows * nb + c, every * (nb + 1)]))
    return Pattern(key // nb, key % nb, nb)


@functools.lru_cache(maxsize=2)
def _pattern_of(grid, powerlaw):
    return _powerlaw(powerlaw) if powerlaw else _grid([int(s) for s in grid.split("x")])


def _pattern(case):
    return _pattern_of(case.get("grid", ""), int(case.get("powerlaw", 0)))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(shape, g, scale=1.0, dtype=F64):
    return (torch.rand(shape, dtype=dtype, device=DEV, generator=g) * 2 - 1) * scale


def _matrix(P, bs, g):
    """Block values of the system on pattern P."""
    val = _uniform((P.nnzb, bs, bs), g)
    i = torch.arange(bs, device=DEV)
    if P.coef is not None:
        val *= 0.1 if float(P.coef.max()) == 4.0 else 0.05
        val[:, i, i] = P.coef[:, None].expand(-1, bs)
        return val
    d = P.row == P.col
    total = torch.segment_reduce(val.abs().sum(2), "sum", lengths=P.rowptr[1:] - P.rowptr[:-1])
    dv = val[d]
    dv[:, i, i] = 1.2 * (total - dv[:, i, i].abs())
    val[d] = dv
    return val


def _packed_factor(P, bs, g):
    """A packed L\\U on pattern P of the size a BILU(0) of the system has:
    the lower part scaled by the pivots, the upper part as it is."""
    val = _matrix(P, bs, g)
    d = P.row == P.col
    i = torch.arange(bs, device=DEV)
    piv = torch.empty(P.nb, bs, dtype=F64, device=DEV)
    piv[P.row[d]] = val[d][:, i, i]
    low = P.row > P.col
    val[low] = val[low] / piv[P.col[low]][:, None, :]
    dv = val[d]
    val[d] = torch.where(torch.ones(bs, bs, device=DEV).tril(-1) > 0, dv / piv[:, None, :], dv)
    return val


def _isai_factors(P, bs, g):
    """(pattern, values) of M_L and M_U of the size the ISAI of the system
    has: first-order inverses on the triangles of P."""
    lu = _packed_factor(P, bs, g)
    i = torch.arange(bs, device=DEV)
    d = P.row == P.col
    piv = torch.empty(P.nb, bs, dtype=F64, device=DEV)
    piv[P.row[d]] = lu[d][:, i, i]
    out = []
    for lower in (True, False):
        keep = P.row >= P.col if lower else P.row <= P.col
        T, v = P.part(keep), -lu[keep]
        if not lower:
            v = v / (piv[T.row][:, :, None] * piv[T.col][:, None, :])
        td = T.row == T.col
        dv = v[td].tril(-1) if lower else v[td].triu(1)
        dv[:, i, i] = torch.ones_like(piv) if lower else 1.0 / piv
        v[td] = dv
        out.append((T, v))
    return out


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    P, bs, op, g = _pattern(case), case["bs"], case["op"], _gen(seed)
    n = P.nb * bs
    st = dict(op=op, nb=P.nb, bs=bs)
    if op == "apply":
        (L, lv), (U, uv) = _isai_factors(P, bs, g)
        dt = F64 if case["prec"] == "fp64" else F32
        st.update(L=(*L.csr(), lv.to(dt)), U=(*U.csr(), uv.to(dt)), b=_uniform(n, g),
                  prec=PREC[case["prec"]])
    elif op == "spmm":
        dt = F64 if case["prec"] == "fp64" else F32
        st.update(A=(*P.csr(), _matrix(P, bs, g).to(dt)), X=_uniform((n, case["k"]), g))
    elif op == "convert":
        st.update(n=n, csr=_scalar_csr(P, bs, case["fill"], _matrix(P, bs, g)))
    elif op == "setup":
        st.update(A=(*P.csr(), _matrix(P, bs, g)), level=case["level"],
                  fp32=case["mode"] == "fp32", nested=case["mode"] == "nested")
    elif op == "trisolve":
        st.update(LU=(*P.csr(), _packed_factor(P, bs, g)), b=_uniform(n, g))
    elif op == "adjoint":
        b, w = _uniform(n, g).requires_grad_(), _uniform(n, g)
        st.update(kind=case["kind"], b=b, w=w)
        if case["kind"] == "isai":
            (L, lv), (U, uv) = _isai_factors(P, bs, g)
            st.update(L=L.csr(), U=U.csr(), lv=lv.requires_grad_(), uv=uv.requires_grad_())
        else:
            st.update(pat=P.csr(), lu=_packed_factor(P, bs, g).requires_grad_())
    elif op == "solve":
        row, col = P.csr()
        prec = case["prec"]
        st.update(prec=PREC[prec], b=_uniform(n, g),
                  handle=api.Preconditioner(P.nb, bs, row, col, _matrix(P, bs, g),
                                            fp32=prec == "fp32", ilu=prec == "ilu",
                                            ilu_fp32=prec == "ilu_fp32", nested=prec == "nested"))
    return st


def _scalar_csr(P, bs, fill, val):
    """The scalar CSR of a BSR matrix of which a share `fill` of the
    off-diagonal scalar entries is stored (the same ones for every seed)."""
    n = P.nb * bs
    r = torch.arange(bs, device=DEV)
    start = P.rowptr[P.row]
    length = (P.rowptr[P.row + 1] - start) * bs
    place = torch.arange(P.nnzb, device=DEV) - start
    # position of entry (p, r, c) in the scalar CSR of all entries
    pos = (start * bs * bs)[:, None, None] + length[:, None, None] * r[None, :, None] + \
        (place * bs)[:, None, None] + r[None, None, :]
    rows = (P.row * bs)[:, None, None] + r[None, :, None] + 0 * r[None, None, :]
    cols = (P.col * bs)[:, None, None] + r[None, None, :] + 0 * r[None, :, None]
    order = torch.empty(P.nnzb * bs * bs, dtype=torch.int64, device=DEV)
    order[pos.reshape(-1)] = torch.arange(order.numel(), device=DEV)
    rows, cols, v = (t.reshape(-1)[order] for t in (rows, cols, val))
    if fill < 1.0:
        keep = torch.rand(rows.numel(), device=DEV, generator=_gen(1)) < fill
        keep |= rows == cols
        rows, cols, v = rows[keep], cols[keep], v[keep]
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return rp.to(I32), cols.to(I32), v.contiguous()


# ------------------------------------------------------------------ run
def run(st):
    op, nb, bs = st["op"], st["nb"], st["bs"]
    if op == "apply":
        return api.isai_apply(nb, bs, st["L"], st["U"], st["b"], st["prec"])
    if op == "spmm":
        return api.bcsr_spmm(nb, bs, *st["A"], st["X"])
    if op == "convert":
        _, row, col, val = api.csr_to_bsr5(st["n"], bs, *st["csr"])
        return dict(row=row, col=col, val=val)
    if op == "setup":
        p = api.Preconditioner(nb, bs, *st["A"], fp32=st["fp32"], nested=st["nested"],
                               isai_level=st["level"])
        lu, L, U = p.factors()
        p.close()
        return dict(lu=lu, L=L, U=U)
    if op == "trisolve":
        y = api.sptrsv(nb, bs, *st["LU"], st["b"], lower=True)
        return dict(y=y, x=api.sptrsv(nb, bs, *st["LU"], y, lower=False))
    if op == "adjoint":
        if st["kind"] == "isai":
            x = ag.isai_apply(st["b"], st["lv"], st["uv"], st["L"], st["U"], nb, bs)
            gb, gl, gu = torch.autograd.grad(x, [st["b"], st["lv"], st["uv"]], st["w"])
            return dict(x=x.detach(), gb=gb, gl=gl, gu=gu)
        x = ag.ilu_solve(st["b"], st["lu"], *st["pat"], nb, bs)
        gb, glu = torch.autograd.grad(x, [st["b"], st["lu"]], st["w"])
        return dict(x=x.detach(), gb=gb, glu=glu)
    x, _ = st["handle"].solve(st["b"], prec=st["prec"], restart=30, tol=1e-10, maxit=1200)
    return x


# ------------------------------------------------------------------ work
def work(case):
    """Every input read once, every output written once."""
    P, bs, op = _pattern(case), case["bs"], case["op"]
    nb, nnz, n, b2 = P.nb, P.nnzb, P.nb * case["bs"], case["bs"] ** 2
    tri = nnz + nb  # blocks of M_L and M_U together
    ptr = 4 * (nb + 1)
    if op == "apply":
        v = 8 if case["prec"] == "fp64" else 4
        return dict(bytes=tri * (b2 * v + 4) + 2 * ptr + 16 * n, flops=2 * tri * b2)
    if op == "spmm":
        v, k = 8 if case["prec"] == "fp64" else 4, case["k"]
        return dict(bytes=nnz * (b2 * v + 4) + ptr + 16 * n * k, flops=2 * nnz * b2 * k)
    if op == "convert":
        entries = nnz * b2 * case["fill"]
        return dict(bytes=entries * 12 + 4 * (n + 1) + nnz * (8 * b2 + 4) + ptr, flops=0)
    if op == "setup":
        extra = dict(fp64=0, fp32=4 * tri * b2, nested=4 * (tri + nnz) * b2)[case["mode"]]
        # one division by a pivot block per lower block, one update each, one
        # product per ISAI entry off the diagonal
        return dict(bytes=nnz * (16 * b2 + 4) + tri * (8 * b2 + 4) + 3 * ptr + extra,
                    flops=2 * b2 * bs * (1.5 * (nnz - nb) + 2 * nnz))
    if op == "trisolve":
        return dict(bytes=nnz * (8 * b2 + 4) + ptr + 24 * n, flops=2 * nnz * b2)
    if op == "adjoint":
        if case["kind"] == "isai":
            return dict(bytes=tri * (16 * b2 + 4) + 2 * ptr + 32 * n, flops=6 * tri * b2)
        return dict(bytes=nnz * (16 * b2 + 4) + ptr + 32 * n, flops=6 * nnz * b2)
    # the operator and both factors at least once, b, x
    v = 4 if case["prec"] in ("fp32", "nested", "ilu_fp32") else 8
    m = nnz if case["prec"].startswith("ilu") else tri
    return dict(bytes=(nnz + m) * (v * b2 + 4) + 3 * ptr + 16 * n, flops=2 * (nnz + m) * b2)


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """run()'s outputs in 64 bits, by plain torch."""
    op, bs = case["op"], case["bs"]
    P = _pattern(case)
    n, nb = P.nb * bs, P.nb
    if op == "solve" and n > 12000:
        return None  # a dense solve of this size takes too long
    if op == "setup" and (nb > 300000 or ("powerlaw" in case and nb > 25000)):
        return None
    if op in ("trisolve", "adjoint") and case.get("kind") != "isai" and "powerlaw" in case \
            and nb > 40000:
        return None
    if op == "solve":
        g = _gen(seed)
        b = _uniform(n, g)
        val = _matrix(P, bs, g)
        D = torch.zeros(nb, bs, nb, bs, dtype=F64, device=DEV)
        D[P.row, :, P.col, :] = val
        return torch.linalg.solve(D.view(n, n), b)
    if op == "setup":
        A = _matrix(P, bs, _gen(seed))
        lu = _bilu0(P, A)
        M = P if case["level"] == 1 else _square(P)
        out = dict(lu=lu)
        for name, lower in (("L", True), ("U", False)):
            T = M.part(M.row >= M.col if lower else M.row <= M.col)
            out[name] = (*T.csr(), _isai(P, lu, T, lower))
        return out
    st = prepare(case, seed)
    if op == "apply":
        y = _product(st["L"], st["b"], nb, bs)
        return _product(st["U"], y, nb, bs)
    if op == "spmm":
        return _product(st["A"], st["X"], nb, bs)
    if op == "convert":
        rp, ci, v = st["csr"]
        r = torch.repeat_interleave(torch.arange(n, device=DEV), (rp[1:] - rp[:-1]).long())
        c = ci.long()
        key = (r // bs) * nb + c // bs
        uniq = torch.unique(key)
        out = torch.zeros(uniq.numel(), bs, bs, dtype=F64, device=DEV)
        out[torch.searchsorted(uniq, key), r % bs, c % bs] = v
        Q = Pattern(uniq // nb, uniq % nb, nb)
        row, col = Q.csr()
        return dict(row=row, col=col, val=out)
    if op == "trisolve":
        y = _tri(P, st["LU"][2], st["b"], True, False)
        return dict(y=y, x=_tri(P, st["LU"][2], y, False, False))
    b, w = st["b"].detach(), st["w"]
    if case["kind"] == "isai":
        L, U = (*st["L"], st["lv"].detach()), (*st["U"], st["uv"].detach())
        y = _product(L, b, nb, bs)
        gy = _product(U, w, nb, bs, True)
        return dict(x=_product(U, y, nb, bs), gb=_product(L, gy, nb, bs, True),
                    gl=_outer(L, gy, b, nb, bs), gu=_outer(U, w, y, nb, bs))
    lu = st["lu"].detach()
    y = _tri(P, lu, b, True, False)
    x = _tri(P, lu, y, False, False)
    lam = _tri(P, lu, w, False, True)
    mu = _tri(P, lu, lam, True, True)
    A = (*P.csr(), lu)
    low = (P.row > P.col)[:, None, None] | ((P.row == P.col)[:, None, None] &
                                            (torch.ones(bs, bs, device=DEV).tril(-1) > 0))
    return dict(x=x, gb=mu,
                glu=torch.where(low, -_outer(A, mu, y, nb, bs), -_outer(A, lam, x, nb, bs)))


def _rows_of(A, nb):
    return torch.repeat_interleave(torch.arange(nb, device=DEV), (A[0][1:] - A[0][:-1]).long())


def _product(A, x, nb, bs, transpose=False):
    """A x (or A^T x) for vectors or several columns, in chunks of blocks."""
    rows, cols, val = _rows_of(A, nb), A[1].long(), A[2]
    if transpose:
        rows, cols = cols, rows
    X = x.view(nb, bs, -1)
    Y = torch.zeros_like(X)
    step = max(1, (1 << 26) // (bs * max(bs, X.shape[2])))
    for s in range(0, rows.numel(), step):
        v = val[s:s + step].to(F64)
        Y.index_add_(0, rows[s:s + step],
                     torch.bmm(v.mT if transpose else v, X[cols[s:s + step]]))
    return Y.view(x.shape)


def _outer(A, u, v, nb, bs):
    rows, cols = _rows_of(A, nb), A[1].long()
    return u.view(nb, bs)[rows][:, :, None] * v.view(nb, bs)[cols][:, None, :]


def _levels(rows, deps, nb):
    """Dependency level of every row (row depends on dep)."""
    lv = torch.zeros(nb, dtype=torch.int64, device=DEV)
    while True:
        new = torch.zeros_like(lv).scatter_reduce_(0, rows, lv[deps] + 1, "amax")
        if torch.equal(new, lv):
            return lv
        lv = new


def _level_rows(lv):
    order = torch.argsort(lv, stable=True)
    return torch.split(order, torch.bincount(lv).tolist())


def _expand(start, count):
    """(which, position): for every i the positions start[i] .. start[i]+count[i]-1."""
    which = torch.repeat_interleave(torch.arange(start.numel(), device=DEV), count)
    first = torch.cumsum(count, 0) - count
    return which, start[which] + torch.arange(which.numel(), device=DEV) - first[which]


def _tri(P, lu, b, lower, transpose):
    """x of L x = b (unit lower) or U x = b on the packed factor, or of the
    transposed system, level by level."""
    nb, bs = P.nb, lu.shape[1]
    rows, cols, val = P.row, P.col, lu
    if transpose:
        rows, cols, val = cols, rows, lu.mT
    keep = (P.row > P.col) if lower else (P.row < P.col)
    order = torch.argsort(rows[keep], stable=True)
    r, c, v = rows[keep][order], cols[keep][order], val[keep][order]
    start = torch.searchsorted(r, torch.arange(nb + 1, device=DEV))
    d = lu[P.row == P.col]
    d = d.tril(-1) + torch.eye(bs, dtype=F64, device=DEV) if lower else d.triu()
    d = d.mT if transpose else d
    upper = lower == transpose
    x, B = torch.zeros(nb, bs, dtype=F64, device=DEV), b.view(nb, bs)
    for R in _level_rows(_levels(r, c, nb)):
        which, at = _expand(start[R], start[R + 1] - start[R])
        rhs = B[R].clone()
        rhs.index_add_(0, which, torch.bmm(v[at], x[c[at]][:, :, None])[:, :, 0], alpha=-1)
        x[R] = torch.linalg.solve_triangular(d[R], rhs[:, :, None], upper=upper)[:, :, 0]
    return x.view(-1)


def _bilu0(P, A):
    """Block ILU(0) without pivoting, level by level, a row's dependencies in
    ascending order."""
    nb, bs = P.nb, A.shape[1]
    v = A.clone()
    key = P.row * nb + P.col
    diag = torch.nonzero(P.row == P.col)[:, 0]
    low = P.row > P.col
    rp = P.rowptr
    eye = torch.eye(bs, dtype=F64, device=DEV)
    for R in _level_rows(_levels(P.row[low], P.col[low], nb)):
        ndep = diag[R] - rp[R]
        for q in range(int(ndep.max())):
            act = R[ndep > q]
            p = rp[act] + q
            K = P.col[p]
            uk = v[diag[K]].triu()
            # L_IK U_KK = A_IK
            lik = torch.linalg.solve_triangular(uk.mT, v[p].mT, upper=False).mT
            v[p] = lik
            which, pos = _expand(diag[K] + 1, rp[K + 1] - diag[K] - 1)
            want = act[which] * nb + P.col[pos]
            at = torch.searchsorted(key, want).clamp(max=key.numel() - 1)
            hit = key[at] == want
            v[at[hit]] -= torch.bmm(lik[which[hit]], v[pos[hit]])
        D = v[diag[R]]
        for k in range(bs):
            D[:, k + 1:, k] /= D[:, k, k, None]
            D[:, k + 1:, k + 1:] -= D[:, k + 1:, k, None] * D[:, k, None, k + 1:]
        v[diag[R]] = D
        which, pos = _expand(diag[R] + 1, rp[R + 1] - diag[R] - 1)
        if pos.numel():
            v[pos] = torch.linalg.solve_triangular(D[which].tril(-1) + eye, v[pos], upper=False,
                                                   unitriangular=True)
    return v


def _square(P):
    """The pattern of A^2."""
    which, pos = _expand(P.rowptr[P.col], P.rowptr[P.col + 1] - P.rowptr[P.col])
    key = torch.unique(P.row[which] * P.nb + P.col[pos])
    return Pattern(key // P.nb, key % P.nb, P.nb)


def _isai(P, lu, T, lower):
    """The approximate inverse of the factor's triangle on pattern T: for
    every column j, (triangle restricted to the column's rows) Y = e_j."""
    nb, bs = P.nb, lu.shape[1]
    key = P.row * nb + P.col
    d = lu[P.row == P.col]
    eye = torch.eye(bs, dtype=F64, device=DEV)
    d = d.tril(-1) + eye if lower else d.triu()
    # blocks of T by column, rows in the order of the substitution
    by = torch.argsort(T.col * nb + (T.row if lower else nb - 1 - T.row))
    rows, cols = T.row[by], T.col[by]
    start = torch.searchsorted(cols, torch.arange(nb + 1, device=DEV))
    length = start[1:] - start[:-1]
    Y = torch.zeros(T.nnzb, bs, bs, dtype=F64, device=DEV)
    for i in range(int(length.max())):
        j = torch.nonzero(length > i)[:, 0]
        t = rows[start[j] + i]
        rhs = torch.where((t == j)[:, None, None], eye, torch.zeros_like(eye))
        for p in range(i):
            want = t * nb + rows[start[j] + p]
            at = torch.searchsorted(key, want).clamp(max=key.numel() - 1)
            hit = torch.nonzero(key[at] == want)[:, 0]
            rhs[hit] -= torch.bmm(lu[at[hit]], Y[start[j[hit]] + p])
        Y[start[j] + i] = torch.linalg.solve_triangular(d[t], rhs, upper=not lower)
    out = torch.empty_like(Y)
    out[by] = Y
    return out
