"""The workloads that the speed of this framework is measured on.

Every case is one pass through the public interface (Handle.setup, result_into,
apply, adjoint_device) on matrices that are made on the GPU from a seed:

  grid2d     2-D 5-point diffusion, coefficient 1 in x and `cy` in y, every face
             multiplied by a random factor in [0.8, 1.2]
  convdiff   3-D 7-point convection-diffusion, log-uniform coefficients, upwind
  ragged     random nonsymmetric, 4..32 off-diagonals in a column, diagonal 1.5
             times the column's absolute off-diagonal sum
  block27    27-point stencil with 3 unknowns per node, 3 x 3 blocks

with the start patterns a user picks: the diagonal, the pattern of A, or the
pattern of A^2 without the entries below 1e-3 of their column's largest.  The
structures belong to the case; the seed gives the values, as in a program that
keeps its patterns and gets new coefficients.
"""
import math

import torch

import mspai_b200 as mb

DEV = "cuda"

# family, grid edge or column count, start pattern, what is called, and options
_LISTED = [
    # the smallest call: one 64 x 64 Poisson-like grid in FP64, P = pattern(A);
    # an application that sets up a coarse level or many small systems
    dict(name="grid64_fp64", family="grid2d", size=64, cy=1.0, pattern="A", call="setup", prec="fp64", rows=0, ns=0, rho=1.0, keep=False),
    # SPAI with pattern updates from the diagonal, the classic adaptive use
    dict(name="convdiff48_adaptive", family="convdiff", size=48, cy=0.0, pattern="diag", call="setup", prec="mixed", rows=0, ns=5, rho=1.0, keep=False),
    # a denser fixed pattern on the same kind of problem: pattern(A^2), about 25
    # entries per column, an odd grid
    dict(name="convdiff41_square", family="convdiff", size=41, cy=0.0, pattern="A2", call="setup", prec="mixed", rows=0, ns=0, rho=1.0, keep=False),
    # the benchmark configuration: a million ragged columns of 10 to 300 entries
    dict(name="ragged1m", family="ragged", size=1_000_000, cy=0.0, pattern="A2", call="setup", prec="mixed", rows=0, ns=0, rho=1.0, keep=False),
    # the same kind of columns for a user who asks for FP64 throughout
    dict(name="ragged20k_fp64", family="ragged", size=20_011, cy=0.0, pattern="A2", call="setup", prec="fp64", rows=0, ns=0, rho=1.0, keep=False),
    # time stepping: two setups with new values of the same structure, from the
    # factors that the handle keeps
    dict(name="ragged60k_resetup", family="ragged", size=60_000, cy=0.0, pattern="A2", call="resetup", prec="mixed", rows=0, ns=0, rho=1.0, keep=True),
    # the backward pass of M as a function of A (gradient of M given, factors kept)
    dict(name="ragged12k_backward", family="ragged", size=12_000, cy=0.0, pattern="A2", call="backward", prec="mixed", rows=0, ns=0, rho=1.0, keep=True),
    # MSPAI probing on a large anisotropic grid: forward ...
    dict(name="aniso1024_probing", family="grid2d", size=1024, cy=1e-3, pattern="A", call="setup", prec="mixed", rows=2, ns=0, rho=10.0, keep=False),
    # ... and the gradient of ||C M - B||_F^2 with respect to C and B
    dict(name="aniso1024_adjoint", family="grid2d", size=1024, cy=1e-3, pattern="A", call="adjoint", prec="mixed", rows=2, ns=0, rho=10.0, keep=False),
    # block SPAI from the block diagonal, block updates allowed, a probing row
    dict(name="block40", family="block27", size=40, cy=0.0, pattern="diag", call="setup", prec="mixed", rows=1, ns=3, rho=10.0, keep=False),
    # block SPAI on the block pattern of A: 27 blocks a block column
    dict(name="block20_pattern", family="block27", size=20, cy=0.0, pattern="A", call="setup", prec="mixed", rows=0, ns=0, rho=1.0, keep=False),
    # the preconditioner's application, once per iteration of a Krylov solver
    dict(name="ragged200k_apply", family="ragged", size=200_000, cy=0.0, pattern="A2", call="apply", prec="mixed", rows=0, ns=0, rho=1.0, keep=False),
]


def listed():
    return [dict(c) for c in _LISTED]


def draw(rng):
    """One more case: a workload as above, its size anywhere in its range."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(family="", size=0, cy=0.0, pattern="A", call="setup",
             prec=rng.choice(["mixed", "mixed", "fp64"]), rows=0, ns=0, rho=1.0, keep=False)
    kind = rng.choice(["grid", "adaptive", "square", "ragged", "ragged", "resetup", "backward",
                       "probing", "probing_adjoint", "block", "block", "block_adjoint",
                       "apply"])
    if kind == "grid":
        c.update(family="grid2d", size=size(16, 1024), cy=rng.choice([1.0, 1e-2]))
    elif kind == "adaptive":
        c.update(family="convdiff", size=size(9, 48), pattern="diag", ns=rng.choice([2, 3, 5]))
    elif kind == "square":
        c.update(family="convdiff", size=size(9, 60), pattern="A2")
    elif kind == "ragged":
        c.update(family="ragged", size=size(2000, 400_000), pattern="A2")
        if c["prec"] == "fp64":
            c["size"] = min(c["size"], 40_000)
    elif kind == "resetup":
        c.update(family="ragged", size=size(2000, 60_000), pattern="A2", call="resetup",
                 prec="mixed", keep=True)
    elif kind == "backward":
        c.update(family="ragged", size=size(1500, 12_000), pattern="A2", call="backward",
                 keep=True)
    elif kind in ("probing", "probing_adjoint"):
        c.update(family="grid2d", size=size(33, 1024), cy=rng.choice([1.0, 1e-3]),
                 rows=rng.choice([1, 2]), rho=rng.choice([1.0, 10.0, 100.0]),
                 call="adjoint" if kind.endswith("adjoint") else "setup")
    elif kind in ("block", "block_adjoint"):
        if kind == "block" and rng.random() < 0.5:
            c.update(family="block27", size=size(5, 20))
        else:
            c.update(family="block27", size=size(6, 40), pattern="diag", rows=rng.choice([0, 1]),
                     ns=3, rho=10.0, call="adjoint" if kind.endswith("adjoint") else "setup")
    else:
        c.update(family="ragged", size=size(2000, 200_000), pattern="A2", call="apply",
                 prec="mixed")
    return c


# ------------------------------------------------------------------ matrices
class Csc:
    """Column pointers, sorted rows and values (None: a pattern) on the GPU."""

    def __init__(self, nrows, ncols, ptr, idx, val):
        self.nrows, self.ncols, self.ptr, self.idx, self.val = nrows, ncols, ptr, idx, val

    @property
    def nnz(self):
        return self.idx.numel()

    def cols(self):
        return torch.repeat_interleave(torch.arange(self.ncols, device=self.idx.device),
                                       self.ptr[1:] - self.ptr[:-1])

    def device_csc(self, pattern=False):
        return mb.DeviceCSC(self.nrows, self.ncols, self.ptr, self.idx,
                            None if pattern else self.val)


def _pointers(sorted_cols, ncols):
    ptr = torch.zeros(ncols + 1, dtype=torch.int64, device=sorted_cols.device)
    ptr[1:] = torch.cumsum(torch.bincount(sorted_cols, minlength=ncols), 0)
    return ptr


def _from_coo(nrows, ncols, rows, cols, vals):
    key, order = torch.sort(cols * nrows + rows)
    c = torch.div(key, nrows, rounding_mode="floor")
    return Csc(nrows, ncols, _pointers(c, ncols), (key - c * nrows).to(torch.int32),
               vals[order].contiguous())


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _grid2d(nx, cy, g):
    n = nx * nx
    idx = torch.arange(n, device=DEV)
    x, y = idx % nx, torch.div(idx, nx, rounding_mode="floor")
    diag = torch.full((n,), 2.0 + 2.0 * cy, dtype=torch.float64, device=DEV)
    rows, cols, vals = [], [], []
    for pos, step, coef in ((x, 1, 1.0), (y, nx, cy)):
        face = coef * (0.8 + 0.4 * torch.rand(n, generator=g, dtype=torch.float64, device=DEV))
        a = idx[pos + 1 < nx]
        w = face[a]
        diag[a] += w - coef
        diag[a + step] += w - coef
        rows += [a, a + step]
        cols += [a + step, a]
        vals += [-w, -w]
    return _from_coo(n, n, torch.cat(rows + [idx]), torch.cat(cols + [idx]),
                     torch.cat(vals + [diag]))


def _convdiff(N, base, g):
    n, h = N ** 3, 1.0 / (N + 1)
    u = torch.rand(n, generator=base, dtype=torch.float64, device=DEV)
    kappa = torch.exp(math.log(1e-2) * u)
    if g is not None:
        kappa *= torch.exp(0.1 * torch.randn(n, generator=g, dtype=torch.float64, device=DEV))
    idx = torch.arange(n, device=DEV)
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    rows, cols, vals = [], [], []
    for d, v in enumerate((20.0, 10.0, 5.0)):
        step = N ** d
        c = torch.div(idx, step, rounding_mode="floor") % N
        for sgn in (-1, 1):
            inside = (c + sgn >= 0) & (c + sgn < N)
            nb = (idx + sgn * step).clamp(0, n - 1)
            kf = torch.where(inside, 2.0 * kappa * kappa[nb] / (kappa + kappa[nb]), kappa)
            diag += kf
            rows.append(idx[inside])
            cols.append(nb[inside])
            vals.append((-kf - (h * v if sgn < 0 else 0.0))[inside])
        diag += h * v
    return _from_coo(n, n, torch.cat(rows + [idx]), torch.cat(cols + [idx]),
                     torch.cat(vals + [diag]))


def _ragged(n, base, g):
    cnt = torch.randint(4, 33, (n,), generator=base, device=DEV)
    cols = torch.repeat_interleave(torch.arange(n, device=DEV), cnt)
    r = torch.randint(0, n - 1, cols.shape, generator=base, device=DEV)
    key = torch.unique(cols * n + r + (r >= cols))  # a row drawn twice counts once
    cols = torch.div(key, n, rounding_mode="floor")
    rows = key - cols * n
    f64 = dict(dtype=torch.float64, device=DEV)
    vals = torch.randn(key.numel(), generator=base, **f64)
    if g is not None:
        vals *= 1.0 + 0.1 * torch.randn(key.numel(), generator=g, **f64)
    diag = torch.segment_reduce(vals.abs(), "sum", offsets=_pointers(cols, n))
    idx = torch.arange(n, device=DEV)
    return _from_coo(n, n, torch.cat([rows, idx]), torch.cat([cols, idx]),
                     torch.cat([vals, 1.5 * diag]))


def _block27(N, g):
    nn = N ** 3
    idx = torch.arange(nn, device=DEV)
    x, y = idx % N, torch.div(idx, N, rounding_mode="floor") % N
    z = torch.div(idx, N * N, rounding_mode="floor")
    Q = torch.randn(nn, 3, 3, generator=g, dtype=torch.float64, device=DEV)
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    brow, bcol, blocks = [idx], [idx], [Q @ Q.transpose(1, 2) + 3.0 * eye]
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if dx == dy == dz == 0:
                    continue
                ok = ((x + dx >= 0) & (x + dx < N) & (y + dy >= 0) & (y + dy < N)
                      & (z + dz >= 0) & (z + dz < N))
                src = idx[ok]
                brow.append(src + dx + dy * N + dz * N * N)
                bcol.append(src)
                blocks.append(torch.randn(src.numel(), 3, 3, generator=g, dtype=torch.float64,
                                          device=DEV) / -26.0)
    brow, bcol, blocks = torch.cat(brow), torch.cat(bcol), torch.cat(blocks)
    t = torch.arange(3, device=DEV)
    ii = (3 * brow[:, None, None] + t[None, :, None]).expand(-1, 3, 3)
    jj = (3 * bcol[:, None, None] + t[None, None, :]).expand(-1, 3, 3)
    P = _from_coo(nn, nn, brow, bcol, torch.ones(brow.numel(), device=DEV))
    return (_from_coo(3 * nn, 3 * nn, ii.reshape(-1), jj.reshape(-1), blocks.reshape(-1)), P)


def _square_pattern(A, drop=1e-3):
    """pattern(A^2) without the entries below `drop` of their column's largest."""
    n = A.ncols
    alen = A.ptr[1:] - A.ptr[:-1]
    work = torch.cumsum(alen[A.idx.long()], 0)  # products up to each entry of A
    ptrs, rows = [], []
    chunk = max(1, int(n * 6e7 / max(1, int(work[-1]))))
    for c0 in range(0, n, chunk):
        c1 = min(n, c0 + chunk)
        e0, e1 = int(A.ptr[c0]), int(A.ptr[c1])
        mid = A.idx[e0:e1].long()
        col = torch.repeat_interleave(torch.arange(c1 - c0, device=DEV), alen[c0:c1])
        src, at = _expand(A, mid)
        key, order = torch.sort(col[at] * n + A.idx[src], stable=True)
        key, count = torch.unique_consecutive(key, return_counts=True)
        val = torch.segment_reduce((A.val[src] * A.val[e0:e1][at])[order], "sum", lengths=count)
        val.abs_()
        col = torch.div(key, n, rounding_mode="floor")
        top = torch.zeros(c1 - c0, dtype=torch.float64, device=DEV)
        top.scatter_reduce_(0, col, val, "amax")
        keep = val >= drop * top[col]
        ptrs.append(torch.bincount(col[keep], minlength=c1 - c0))
        rows.append((key - col * n)[keep].to(torch.int32))
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.cat(ptrs), 0)
    return Csc(n, n, ptr, torch.cat(rows), None)


def _expand(M, cols):
    """Entry numbers of M's columns `cols`, one column after the other, and for
    each the place in `cols` that it belongs to."""
    lens = (M.ptr[1:] - M.ptr[:-1])[cols]
    at = torch.repeat_interleave(torch.arange(cols.numel(), device=cols.device), lens)
    first = torch.cumsum(lens, 0) - lens
    return M.ptr[cols][at] + torch.arange(at.numel(), device=cols.device) - first[at], at


def _with_rows(A, E, rho, explicit):
    """C = [A; rho E^T A] (explicit: values given by E, else E^T A) for p rows."""
    n, p = A.ncols, E.shape[1]
    col = A.cols()
    if explicit:
        extra = E
    else:
        extra = torch.stack([torch.segment_reduce(A.val * E[A.idx.long(), q], "sum",
                                                  offsets=A.ptr) for q in range(p)], 1)
    jr = torch.arange(n, device=DEV)
    rows = [A.idx.long()] + [torch.full((n,), n + q, device=DEV) for q in range(p)]
    cols = [col] + [jr] * p
    vals = [A.val] + [rho * extra[:, q] for q in range(p)]
    return _from_coo(n + p, n, torch.cat(rows), torch.cat(cols), torch.cat(vals))


def _problem(case, seed):
    """(C, B or None, P, block size, generator) of the case."""
    g, size, pattern = _gen(seed), case["size"], case["pattern"]
    bs, P = 1, None
    if case["family"] == "grid2d":
        A = _grid2d(size, case["cy"], g)
    elif case["family"] == "block27":
        A, P = _block27(size, g)
        bs = 3
    else:
        make = _convdiff if case["family"] == "convdiff" else _ragged
        if pattern == "A2":
            P = _square_pattern(make(size, _gen(size), None))
        A = make(size, _gen(size), g)
    n = A.ncols
    if pattern == "diag":
        n //= bs
        P = Csc(n, n, torch.arange(n + 1, device=DEV),
                torch.arange(n, dtype=torch.int32, device=DEV), None)
        n *= bs
    elif P is None:
        P = Csc(n, n, A.ptr, A.idx, None)
    C, B = A, None
    if case["rows"]:
        E = torch.ones(n, case["rows"], dtype=torch.float64, device=DEV)
        E[1::2, 1:] = -1.0  # the second probing vector alternates
        C = _with_rows(A, E, case["rho"], False)
        j = torch.arange(n, device=DEV)
        I = Csc(n, n, torch.arange(n + 1, device=DEV), j.to(torch.int32),
                torch.ones(n, dtype=torch.float64, device=DEV))
        B = _with_rows(I, E, case["rho"], True)
    return C, B, P, bs, g


def _options(case, bs):
    adaptive = case["ns"] > 0
    return mb.Options(ep=0.4, ns=case["ns"], mn=3 if bs > 1 else 5, bs=bs, prec=case["prec"],
                      rho=case["rho"], probing=1 if case["rows"] and not adaptive else 0,
                      keep_factors=case["keep"])


def _step_values(C, g, count):
    """`count` later value sets of C: every entry changed by about 1e-4."""
    return [C.val * (1.0 + 1e-4 * torch.randn(C.nnz, generator=g, dtype=torch.float64,
                                              device=DEV)) for _ in range(count)]


def prepare(case, seed):
    C, B, P, bs, g = _problem(case, seed)
    s = dict(call=case["call"], handle=mb.Handle(0), C=C.device_csc(),
             B=None if B is None else B.device_csc(), P=P.device_csc(pattern=True),
             options=_options(case, bs), fixed=case["ns"] == 0 and bs == 1)
    f64 = dict(dtype=torch.float64, device=DEV)
    h, call = s["handle"], case["call"]
    most = _most(case, P, bs)
    s["values"] = torch.zeros(most, **f64)
    if not s["fixed"]:  # M's pattern is its own: room for all that it can hold
        s["ptr"] = torch.zeros(C.ncols + 1, dtype=torch.int64, device=DEV)
        s["idx"] = torch.zeros(most, dtype=torch.int32, device=DEV)
    if call == "resetup":
        s["steps"] = [mb.DeviceCSC(C.nrows, C.ncols, C.ptr, C.idx, v)
                      for v in _step_values(C, g, 2)]
        s["again"] = mb.Options(ns=0, prec=case["prec"], keep_factors=True, reuse_factors=6)
    if call == "backward":
        s["gbar"] = torch.randn(P.nnz, generator=g, **f64)
    if call in ("adjoint", "backward"):
        s["dC"] = torch.empty(C.nnz, **f64)
        s["dB"] = None if B is None else torch.empty(B.nnz, **f64)
    if call == "apply":
        s["x"] = torch.randn(C.ncols, generator=g, **f64)
    torch.cuda.synchronize()  # the handle works on a stream of its own
    if call != "setup":
        h.setup(s["C"], s["P"], B=s["B"], options=s["options"])
    return s


def _most(case, P, bs):
    """Entries that M can have: the start pattern and what the updates can add."""
    return (P.nnz + P.ncols * case["ns"] * (3 if bs > 1 else 5)) * bs * bs


def _result(s):
    h = s["handle"]
    if s["fixed"]:  # M has P's pattern: only its values are new
        h.result_into(values=s["values"], device=True)
        return s["values"]
    h.result_into(colptr=s["ptr"], rowidx=s["idx"], values=s["values"], device=True)
    return s["ptr"], s["idx"], s["values"]


def run(s):
    h, call = s["handle"], s["call"]
    if call == "setup":
        h.setup(s["C"], s["P"], B=s["B"], options=s["options"])
        return _result(s)
    if call == "resetup":
        for C in s["steps"]:
            h.setup(C, s["P"], B=s["B"], options=s["again"])
        return _result(s)
    if call == "apply":
        return h.apply(s["x"])
    if call == "adjoint":
        loss = h.adjoint_device(s["C"], s["dC"], B=s["B"], dB=s["dB"])
    else:
        loss = h.adjoint_device(s["C"], s["dC"], gbar=s["gbar"], residual_weight=0.0)
    return dict(dC=s["dC"], dB=s["dB"], loss=loss)


# ---------------------------------------------------------------- cost of a pass
def _sizes(case):
    """Columns n, entries per column of C, |J| and the shared rows' entries per
    column problem (means, from the generators' distributions)."""
    s = case["size"]
    if case["family"] == "grid2d":
        n, c = s * s, 5.0
    elif case["family"] == "convdiff":
        n, c = s ** 3, 7.0
    elif case["family"] == "ragged":
        n, c = s, 19.0
    else:
        n, c = 3 * s ** 3, 81.0
    c += case["rows"]
    if case["pattern"] == "diag":
        j = 3.0 if case["family"] == "block27" else 4.0  # about what the updates end with
    elif case["pattern"] == "A":
        j = c - case["rows"]
    else:
        j = 134.0 if case["family"] == "ragged" else 22.0
    return n, c, j


def work(case):
    """Inputs read once and outputs written once; one least-squares solution of
    every column by the normal equations of its |J| unknowns (block columns
    share theirs)."""
    n, c, j = _sizes(case)
    bs = 3 if case["family"] == "block27" else 1
    nnz_c, nnz_p, nnz_m = n * c, n * j / bs ** 2, n * j
    tgt = 12.0 * n * (1 + case["rows"]) if case["rows"] else 0.0
    read = 12.0 * nnz_c + 8.0 * n + 4.0 * nnz_p + tgt
    solve = n / bs * (j ** 3 / 3.0) + n * (2.0 * j * j + 4.0 * c * j)
    call = case["call"]
    if call == "setup":
        out = 8.0 * nnz_m if case["ns"] == 0 and bs == 1 else 12.0 * nnz_m + 8.0 * n
        return dict(bytes=read + out, flops=solve)
    if call == "resetup":
        return dict(bytes=2 * (read + 8.0 * nnz_m), flops=2 * n * (2.0 * j * j + 4.0 * c * j))
    if call == "apply":
        return dict(bytes=12.0 * nnz_m + 16.0 * n, flops=2.0 * nnz_m)
    grads = 8.0 * nnz_c + (8.0 * n * (1 + case["rows"]) if case["rows"] else 0.0)
    flops = n * 6.0 * c * j + (2.0 * n * j * j if call == "backward" else 0.0)
    return dict(bytes=read + 12.0 * nnz_m + (8.0 * nnz_m if call == "backward" else 0.0) + grads,
                flops=flops)


# ------------------------------------------------------------ values in 64 bits
def _solve(C, ks, owner, cols, target, nrhs=1, gbar=None):
    """Least-squares problems ks[i] with the columns cols[owner == i] of C (owner
    ascending) and the target entries target = (owner, row, value, rhs): yields
    for chunks of problems the solutions, residuals and multipliers."""
    K = ks.numel()
    nj = torch.bincount(owner, minlength=K)
    start = torch.cumsum(nj, 0) - nj
    clen = C.ptr[1:] - C.ptr[:-1]
    ne = torch.zeros(K, dtype=torch.int64, device=DEV).index_add_(0, owner, clen[cols])
    order = torch.argsort(ne)
    ne_s, nj_s = ne[order].tolist(), torch.cummax(nj[order], 0).values.tolist()
    t_own, t_row, t_val, t_rhs = target
    i0 = 0
    while i0 < K:
        i1 = i0 + 1
        total = ne_s[i0]
        while (i1 < K and (i1 + 1 - i0) * ne_s[i1] * nj_s[i1] < 2e8
               and total + ne_s[i1] < 4e7):
            total += ne_s[i1]
            i1 += 1
        sel = torch.sort(order[i0:i1]).values
        k = sel.numel()
        loc = torch.full((K,), -1, dtype=torch.int64, device=DEV)
        loc[sel] = torch.arange(k, device=DEV)
        pairs = torch.nonzero(loc[owner] >= 0).squeeze(1)
        po, pc = loc[owner[pairs]], cols[pairs]
        pj = pairs - start[owner[pairs]]
        src, at = _expand(C, pc)
        eo, ej = po[at], pj[at]
        rows, inv = torch.unique(eo * C.nrows + C.idx[src], return_inverse=True)
        ro = torch.div(rows, C.nrows, rounding_mode="floor")
        mk = torch.bincount(ro, minlength=k)
        m, n = int(mk.max()), int(nj[sel].max())
        local = torch.arange(rows.numel(), device=DEV) - (torch.cumsum(mk, 0) - mk)[ro]
        A = torch.zeros(k, m, n, dtype=torch.float64, device=DEV)
        A[eo, local[inv], ej] = C.val[src]
        b = torch.zeros(k, m, nrhs, dtype=torch.float64, device=DEV)
        tl = loc[t_own]
        key = tl * C.nrows + t_row
        pos = torch.searchsorted(rows, key).clamp(max=rows.numel() - 1)
        hit = (tl >= 0) & (rows[pos] == key)
        b[tl[hit], local[pos[hit]], t_rhs[hit]] = t_val[hit]
        G = A.transpose(1, 2) @ A
        pad = torch.arange(n, device=DEV)[None, :] >= nj[sel][:, None]
        G += torch.diag_embed(pad.to(torch.float64))
        L = torch.linalg.cholesky(G)
        x = torch.zeros(k, n, nrhs, dtype=torch.float64, device=DEV)
        r = b
        for _ in range(3):
            x = x + torch.cholesky_solve(A.transpose(1, 2) @ r, L)
            r = b - A @ x
        lam = q = None
        if gbar is not None:
            gb = torch.zeros(k, n, 1, dtype=torch.float64, device=DEV)
            gb[po, pj, 0] = gbar[pairs]
            lam = torch.zeros_like(gb)
            for _ in range(3):
                lam = lam + torch.cholesky_solve(gb - A.transpose(1, 2) @ (A @ lam), L)
            q = A @ lam
        yield dict(sel=sel, pairs=pairs, po=po, pj=pj, src=src, eo=eo, ej=ej, er=local[inv],
                   rows=rows, ro=ro, local=local, x=x, r=r, lam=lam, q=q, t=torch.nonzero(
                       tl >= 0).squeeze(1), hit=hit, pos=pos, tl=tl)
        i0 = i1


def _target(C, B, n, bs):
    if B is None:
        k = torch.arange(n, device=DEV)
        own = torch.div(k, bs, rounding_mode="floor")
        return own, k, torch.ones(n, dtype=torch.float64, device=DEV), k - bs * own
    col = B.cols()
    own = torch.div(col, bs, rounding_mode="floor")
    return own, B.idx.long(), B.val, col - bs * own


def _scalar_columns(P, bs):
    """(problem, scalar column of C) pairs of the pattern, problem by problem."""
    own, j = P.cols(), P.idx.long()
    if bs > 1:
        own = own[:, None].expand(-1, bs).reshape(-1)
        j = (bs * j[:, None] + torch.arange(bs, device=DEV)).reshape(-1)
    return own, j


def _adaptive(C, ep, mn, ns):
    """Pattern updates from the diagonal (candidates from the rows of I and k,
    at most mn of the smallest rho not above their mean)."""
    n = C.ncols
    byrow = _from_coo(n, n, C.cols(), C.idx.long(), C.val)  # column k: C's row k
    allk = torch.arange(n, device=DEV)
    pairs = allk * n + allk
    active = torch.ones(n, dtype=torch.bool, device=DEV)
    norm2 = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, C.cols(), C.val ** 2)
    values = torch.zeros(0, dtype=torch.float64, device=DEV)
    for step in range(ns + 1):
        own = torch.div(pairs, n, rounding_mode="floor")
        col = pairs - own * n
        values = torch.zeros(pairs.numel(), dtype=torch.float64, device=DEV)
        new = [pairs]
        grown = torch.zeros(n, dtype=torch.bool, device=DEV)
        for s in _solve(C, allk, own, col, _target(C, None, n, 1)):
            values[s["pairs"]] = s["x"][s["po"], s["pj"], 0]
            res = s["r"].square().sum((1, 2)).sqrt()
            go = active[s["sel"]] & (res > ep)
            if step == ns or not bool(go.any()):
                continue
            r = s["r"][s["ro"], s["local"], 0]
            rk = s["sel"][s["ro"]]
            rr = s["rows"] - s["ro"] * n
            rowkey = rk * n + rr  # ascending: sel is
            m = go[s["ro"]]
            L = torch.unique(torch.cat([rowkey[m], s["sel"][go] * (n + 1)]))
            lk = torch.div(L, n, rounding_mode="floor")
            src, at = _expand(byrow, L - lk * n)
            cand = torch.unique(lk[at] * n + byrow.idx[src])
            p = torch.searchsorted(pairs, cand).clamp(max=pairs.numel() - 1)
            cand = cand[pairs[p] != cand]
            if cand.numel() == 0:
                continue
            ck = torch.div(cand, n, rounding_mode="floor")
            cj = cand - ck * n
            src, at = _expand(C, cj)
            key = ck[at] * n + C.idx[src]
            p = torch.searchsorted(rowkey, key).clamp(max=rowkey.numel() - 1)
            num = torch.zeros(cand.numel(), dtype=torch.float64, device=DEV)
            num.index_add_(0, at, torch.where(rowkey[p] == key, r[p] * C.val[src], 0.0))
            full = torch.zeros(n, dtype=torch.float64, device=DEV)
            full[s["sel"]] = res
            rho = (full[ck] ** 2 - num ** 2 / norm2[cj]).clamp(min=0).sqrt()
            cnt = torch.bincount(ck, minlength=n)
            mean = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, ck, rho) / cnt
            order = torch.argsort(rho, stable=True)
            order = order[torch.argsort(ck[order], stable=True)]
            rank = torch.arange(cand.numel(), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[ck]
            take = (rank < mn) & (rho[order] <= mean[ck])
            new.append(cand[order][take])
            grown[ck[take]] = True
        if len(new) == 1:
            break
        active = grown
        pairs = torch.sort(torch.cat(new)).values
    own = torch.div(pairs, n, rounding_mode="floor")
    return _pointers(own, n), (pairs - own * n).to(torch.int32), values


def exact(case, seed):
    n, c, j = _sizes(case)
    if n / (3 if case["family"] == "block27" else 1) * c * j > 6e8:
        return None  # too long
    C, B, P, bs, g = _problem(case, seed)
    call, n = case["call"], C.ncols
    most = _most(case, P, bs)
    if case["ns"] > 0 and bs == 1:
        return _padded(most, *_adaptive(C, 0.4, 5, case["ns"]))
    if call == "resetup":
        C.val = _step_values(C, g, 2)[1]
    gbar = None
    f64 = dict(dtype=torch.float64, device=DEV)
    if call == "backward":
        gbar = torch.randn(P.nnz, generator=g, **f64)
    own, cols = _scalar_columns(P, bs)
    target = _target(C, B, n, bs)
    X = torch.zeros(cols.numel(), bs, **f64)
    grads = call in ("adjoint", "backward")
    w = 1.0 if call == "adjoint" else 0.0
    dC = torch.zeros(C.nnz, **f64) if grads else None
    dB = torch.zeros(B.nnz, **f64) if grads and B is not None else None
    loss = torch.zeros((), **f64)
    for s in _solve(C, torch.arange(P.ncols, device=DEV), own, cols, target, bs, gbar):
        x, r = s["x"], s["r"]
        X[s["pairs"]] = x[s["po"], s["pj"]]
        if case["ns"] > 0 and float(r.square().sum((1, 2)).max().sqrt()) > 0.4 * math.sqrt(bs):
            return None  # a block column that updates its pattern
        if not grads:
            continue
        e, er, ej = s["eo"], s["er"], s["ej"]
        gv = -2.0 * w * (r[e, er] * x[e, ej]).sum(1)
        if gbar is not None:
            gv += r[e, er, 0] * s["lam"][e, ej, 0] - s["q"][e, er, 0] * x[e, ej, 0]
            loss += (gbar[s["pairs"]] * x[s["po"], s["pj"], 0]).sum()
        dC.index_add_(0, s["src"], gv)
        t = s["t"]
        hit, lk, lr = s["hit"][t], s["tl"][t], s["local"][s["pos"][t]]
        rt = torch.where(hit, r[lk, lr, target[3][t]], target[2][t])
        loss += w * (r.square().sum() + target[2][t][~hit].square().sum())
        if dB is not None:
            dB[t] = 2.0 * w * rt
    if grads:
        return dict(dC=dC, dB=dB, loss=float(loss))
    if call == "apply":
        x = torch.randn(n, generator=g, **f64)
        return torch.zeros(n, **f64).index_add_(0, cols, X[:, 0] * x[own])
    if bs == 1:
        return X[:, 0].contiguous()
    # scalar column bs k + c of M: the rows of problem k, its c-th solution
    col = bs * own[:, None] + torch.arange(bs, device=DEV)
    M = _from_coo(n, n, cols[:, None].expand(-1, bs).reshape(-1), col.reshape(-1), X.reshape(-1))
    return _padded(most, M.ptr, M.idx, M.val)


def _padded(most, ptr, idx, val):
    """As _result lays them out: zeros after M's entries."""
    i = torch.zeros(most, dtype=torch.int32, device=DEV)
    v = torch.zeros(most, dtype=torch.float64, device=DEV)
    i[:idx.numel()], v[:val.numel()] = idx, val
    return ptr, i, v
