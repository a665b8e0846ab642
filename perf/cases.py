"""Measured cases of the merged two-site DMRG inner loop, through the Python call surface.

Every case is one call that a sweep, a gradient or a parameter scan makes at a bond in
the middle of a half-filled chain, on synthetic operands with the block structure, the
sizes and the value distributions of the library's own workloads:

* ``hubbard``: a chain of ``norb`` sites, MPO bond dimension 6 (configurations C1, C3, C4);
* ``qc``: ``norb`` orbitals under the complementary-operator MPO, whose middle bond has
  4 m^2 + 2 m (m - 1) + 2 m^2 + 2 + 8 m operators for m = norb / 2 (862 at norb = 20,
  configuration C2).

The sectors of a bond are (N, 2Sz) pairs with dimensions that fall off as a Gaussian in
N and 2Sz around half filling (a converged C2 bond has a spread of 1.3 in N and 1.7 in
2Sz), rounded: ragged, from 1 to about M/7.  Operators hold an identity, a block
Hamiltonian of magnitude 10 and operators whose magnitudes spread over 10^-3 .. 10^0.5
as the MPO coefficients do; wavefunction rows and columns decay over four decades
(an eigenproblem starts from a guess on the low configurations).

``exact`` computes the same results with torch in 64 bits from the definitions.
"""
import functools
import math

import numpy as np
import torch

SITE = [(0, 0), (1, 1), (1, -1), (2, 0)]


# --------------------------------------------------------------------------------------
# block structures
# --------------------------------------------------------------------------------------
def _neg(qs):
    return [(-a, -b) for a, b in qs]


def _bond(sites, M):
    """Sectors and dimensions of a bond with `sites` half-filled sites on one side."""
    cells = []
    for n in range(max(0, sites - 5), min(2 * sites, sites + 5) + 1):
        for s in range(-6, 7):
            up, dn = (n + s) // 2, (n - s) // 2
            if (n + s) % 2 or not (0 <= up <= sites and 0 <= dn <= sites):
                continue
            w = math.exp(-0.5 * ((n - sites) / 1.3) ** 2 - 0.5 * (s / 1.7) ** 2)
            cells.append(((n, s), w, math.comb(sites, up) * math.comb(sites, dn)))
    tot = sum(c[1] for c in cells)
    q, d = [], []
    for (qq, w, most) in cells:
        dim = min(most, int(M * w / tot + 0.5))
        if dim > 0:
            q.append(qq)
            d.append(dim)
    return q, d


def _merge(qa, da, qb, db):
    """Merged sectors of an index pair in order of first appearance, with the place
    (merged sector, offset) of every pair."""
    where, q, d, place = {}, [], [], {}
    for i, (x, dx) in enumerate(zip(qa, da)):
        for j, (y, dy) in enumerate(zip(qb, db)):
            s = (x[0] + y[0], x[1] + y[1])
            if s not in where:
                where[s] = len(q)
                q.append(s)
                d.append(0)
            k = where[s]
            place[i, j] = (k, d[k])
            d[k] += dx * dy
    return q, d, place


def _mpo_bond(model, norb):
    """Quantum numbers of the middle MPO bond: identity, block Hamiltonian, the rest."""
    if model == "hubbard":
        return [(0, 0), (0, 0), (1, 1), (1, -1), (-1, -1), (-1, 1)]
    m = norb // 2
    q = [(0, 0)] * (2 * m * m + 2)
    for x in ((0, 2), (0, -2), (2, 0), (-2, 0)):
        q += [x] * (m * m)
    for x in ((2, 2), (2, -2), (-2, 2), (-2, -2)):
        q += [x] * (m * (m - 1) // 2)
    for x in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
        q += [x] * (2 * m)
    return q


class Layout:
    """The stored blocks of a block-sparse array: every block that the total quantum number
    allows, packed by ascending row-major tag, each dense row-major."""

    def __init__(self, q, qshape, dshape):
        self.q, self.qshape, self.dshape = tuple(q), [list(x) for x in qshape], [list(x) for x in dshape]
        n = [len(x) for x in qshape]
        grid = np.indices(n, dtype=np.int32).reshape(len(n), -1)
        tot = [np.zeros(grid.shape[1], dtype=np.int32) for _ in range(2)]
        size = np.ones(grid.shape[1], dtype=np.int64)
        for i in range(len(n)):
            for c in range(2):
                tot[c] += np.array([x[c] for x in qshape[i]], dtype=np.int32)[grid[i]]
            size *= np.array(dshape[i], dtype=np.int64)[grid[i]]
        ok = np.flatnonzero((tot[0] == q[0]) & (tot[1] == q[1]) & (size > 0))
        self.index = grid[:, ok].T.copy()
        self.size = size[ok]
        self.off = np.concatenate([[0], np.cumsum(self.size)])
        self.nnz = int(self.off[-1])

    @functools.cached_property
    def slot(self):
        return {tuple(x): i for i, x in enumerate(self.index.tolist())}

    def block(self, data, b):
        dims = [self.dshape[i][k] for i, k in enumerate(self.index[b])]
        return data[int(self.off[b]):int(self.off[b + 1])].view(dims)


@functools.lru_cache(maxsize=8)
def _structure(model, norb, M):
    ls = (norb - 2) // 2
    rs = norb - 2 - ls
    ql, dl = _bond(ls, M)
    qr, dr = _bond(rs, M)
    one = [1] * 4
    A = _merge(ql, dl, SITE, one)
    B = _merge(SITE, one, qr, dr)
    total = (norb, norb % 2)
    w = _mpo_bond(model, norb)
    return {"ql": ql, "dl": dl, "qr": qr, "dr": dr, "A": A, "B": B, "w": w, "total": total,
            "L": Layout((0, 0), [A[0], w, _neg(A[0])], [A[1], [1] * len(w), A[1]]),
            "R": Layout((0, 0), [B[0], _neg(w), _neg(B[0])], [B[1], [1] * len(w), B[1]]),
            "psi": Layout(total, [A[0], B[0]], [A[1], B[1]])}


def _kept(d, M):
    """Dimensions that a truncation of merged sectors to M states keeps."""
    return [min(x, max(0, int(M * x / sum(d) + 0.5))) for x in d]


@functools.lru_cache(maxsize=8)
def _site(model, norb, M, forward):
    """Environment and site MPO of the merged operator (forward: left, backward: right)."""
    s = _structure(model, norb, M)
    w = s["w"]
    inner = _mpo_bond(model, max(2, norb - 2))  # the bond on the environment's side
    q, d = (s["ql"], s["dl"]) if forward else (s["qr"], s["dr"])
    # W[w, s, t, v] with q_w + q_s - q_t - q_v = 0; forward contracts w, backward v
    left, right = (inner, w) if forward else (w, inner)
    env = Layout((0, 0), [q, _neg(left) if forward else right, _neg(q)], [d, [1] * len(inner), d])
    rng = np.random.default_rng(len(w) * 7919 + len(inner))
    by_q = {}
    for v, x in enumerate(right):
        by_q.setdefault(x, []).append(v)
    hops = [(a, b, (SITE[a][0] - SITE[b][0], SITE[a][1] - SITE[b][1])) for a in range(4) for b in range(4)]
    tags, seen = [], {}
    for i, x in enumerate(left):
        same = by_q.get(x, [])
        if same:  # the operator passed through
            v = same[seen.get(x, 0) % len(same)]
            seen[x] = seen.get(x, 0) + 1
            tags += [((i * 4 + a) * 4 + a) * len(right) + v for a in range(4)]
        picks = 8 if model == "hubbard" else 36
        open_ = [(a, b, vs) for a, b, h in hops for vs in [by_q.get((x[0] + h[0], x[1] + h[1]))] if vs]
        for _ in range(picks if open_ else 0):
            a, b, vs = open_[rng.integers(len(open_))]
            tags.append(((i * 4 + a) * 4 + b) * len(right) + vs[rng.integers(len(vs))])
    tags = sorted(set(tags))
    return {"env": env, "qshape": [left, SITE, _neg(SITE), _neg(right)], "tags": tags,
            "merged": s["A"] if forward else s["B"], "nright": len(right)}


# --------------------------------------------------------------------------------------
# values
# --------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _per_block(lay, scale):
    """One value per block spread over its elements."""
    return torch.repeat_interleave(torch.as_tensor(scale, dtype=torch.float64, device="cuda"),
                                   torch.as_tensor(lay.size, device="cuda"))


def _operator(lay, g, identity, hamiltonian, hermitian=False):
    """Operator blocks [i, w, j]; `identity` and `hamiltonian` are the w of those two."""
    nw = len(lay.qshape[1])
    mag = 10.0 ** (torch.rand(nw, generator=g, device="cuda", dtype=torch.float64) * 3.5 - 3.0)
    mag[hamiltonian] = 10.0
    x = torch.randn(lay.nnz, generator=g, device="cuda", dtype=torch.float64)
    x *= _per_block(lay, mag[torch.as_tensor(lay.index[:, 1], device="cuda", dtype=torch.long)])
    for b in np.flatnonzero(lay.index[:, 1] == identity):
        blk = lay.block(x, b)[:, 0, :]
        blk.copy_(torch.eye(blk.shape[0], device="cuda", dtype=torch.float64))
    if hermitian:
        _make_hermitian(lay, x, identity, hamiltonian)
    return x


def _make_hermitian(lay, x, identity, hamiltonian):
    """w with opposite quantum numbers become adjoint pairs and w of zero quantum number
    symmetric; couplings shrink to a few percent and the block Hamiltonian to ascending
    levels, so that the lowest state is separated as a ground state is."""
    q = lay.qshape[1]
    partner, free = {}, {}
    for w, a in enumerate(q):
        if a == (0, 0):
            partner[w] = w
            continue
        other = free.get((-a[0], -a[1]))
        if other:
            partner[w] = other.pop(0)
            partner[partner[w]] = w
        else:
            free.setdefault(a, []).append(w)
    x *= _per_block(lay, np.where(lay.index[:, 1] == identity, 1.0, 0.02))
    for b, (i, w, j) in enumerate(lay.index.tolist()):
        p = partner.get(w)
        if w == identity:
            continue
        c = None if p is None else lay.slot.get((j, p, i))
        blk = lay.block(x, b)[:, 0, :]
        if c is None:
            blk.zero_()
        elif c == b:
            blk.copy_(0.5 * (blk + blk.T).clone())
            if w == hamiltonian:
                level = 0.3 * i + 2.0 * torch.arange(blk.shape[0], device="cuda", dtype=torch.float64).sqrt()
                blk.mul_(0.2).add_(torch.diag(level))
        elif c > b:
            lay.block(x, c)[:, 0, :].copy_(blk.T)


def _wavefunction(lay, g):
    x = torch.randn(lay.nnz, generator=g, device="cuda", dtype=torch.float64)
    rows = [10.0 ** (-4.0 * torch.rand(d, generator=g, device="cuda", dtype=torch.float64)) for d in lay.dshape[0]]
    cols = [10.0 ** (-4.0 * torch.rand(d, generator=g, device="cuda", dtype=torch.float64)) for d in lay.dshape[1]]
    for b, (i, j) in enumerate(lay.index.tolist()):
        lay.block(x, b).mul_(rows[i][:, None]).mul_(cols[j][None, :])
    return x / x.norm()


def _schmidt_wavefunction(lay, g):
    """A wavefunction whose singular values fall over six decades in every block, the same
    ones for every seed, so that a truncation keeps the same sectors and dimensions."""
    x = torch.empty(lay.nnz, device="cuda", dtype=torch.float64)
    rng = np.random.default_rng(lay.nnz)
    for b in range(len(lay.size)):
        blk = lay.block(x, b)
        k = min(blk.shape)
        u, v = (torch.linalg.qr(torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64))[0]
                for n in blk.shape)
        sv = 10.0 ** (-6.0 * (np.arange(k) + rng.random()) / k)
        blk.copy_(u * torch.as_tensor(sv, device="cuda") @ v.T)
    return x / x.norm()


def _isometry(s, forward, M, g):
    """The left (right) singular vectors of a truncation: Layout and values."""
    q, d, _ = s["A"] if forward else s["B"]
    k = _kept(d, M)
    keep = [i for i, x in enumerate(k) if x > 0]
    new_q, new_d = [q[i] for i in keep], [k[i] for i in keep]
    if forward:
        lay = Layout((0, 0), [q, _neg(new_q)], [d, new_d])
    else:
        lay = Layout((0, 0), [_neg(new_q), q], [new_d, d])
    x = torch.empty(lay.nnz, device="cuda", dtype=torch.float64)
    for b in range(len(lay.size)):
        blk = lay.block(x, b)
        m, n = blk.shape
        u = torch.linalg.qr(torch.randn(max(m, n), min(m, n), generator=g, device="cuda", dtype=torch.float64))[0]
        blk.copy_(u if m >= n else u.T)
    return lay, x


def _mpo_values(site, seed):
    rng = np.random.default_rng(seed)
    n = len(site["tags"])
    v = 10.0 ** rng.uniform(-3.0, 0.5, n) * rng.choice([-1.0, 1.0], n)
    v[rng.random(n) < 0.2] = 1.0
    return v


def _inputs(case, seed):
    """Everything a case computes from: {name: (Layout, values)}, and the site MPOs."""
    g = _gen(seed)
    model, norb, M, fw = case["model"], case["norb"], case["M"], case.get("forward", True)
    op = case["op"]
    s = _structure(model, norb, M)
    out = {}
    if op in ("sigma", "diagonal", "diagonalize"):
        herm = op == "diagonalize"
        out["L"] = (s["L"], _operator(s["L"], g, 0, 1, herm))
        out["R"] = (s["R"], _operator(s["R"], g, 1, 0, herm))
    if op in ("sigma", "gradient"):
        out["psi"] = (s["psi"], _wavefunction(s["psi"], g))
    if op == "canonicalize":
        out["psi"] = (s["psi"], _schmidt_wavefunction(s["psi"], g))
    if op == "renormalize":
        lay = s["L" if fw else "R"]
        out["O"] = (lay, _operator(lay, g, 0 if fw else 1, 1 if fw else 0))
        out["U"] = _isometry(s, fw, M, g)
    if op == "diagonalize":  # a bond's guess: most weight on the low configurations
        diag = _exact_diagonal(s, out["L"][1], out["R"][1])
        x = 1.0 + 0.3 * torch.randn(s["psi"].nnz, generator=g, device="cuda", dtype=torch.float64)
        x /= (1.0 + diag - diag.min()) ** 3
        out["psi"] = (s["psi"], x / x.norm())
    for side in (True, False):
        if op == "gradient" or (op == "merged_operator" and side == fw):
            site = _site(model, norb, M, side)
            out["env%d" % side] = (site["env"], _operator(site["env"], g, 0 if side else 1, 1 if side else 0))
            out["mpo%d" % side] = (site, _mpo_values(site, int(seed) * 2 + side))
    return out


# --------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------
def _case(name, op, model, norb, M, **more):
    return dict(name=name, op=op, model=model, norb=norb, M=M, **more)


def listed():
    return [
        # the smallest H_eff*psi of a user's run (C1: Hubbard, M = 64): launches and latency
        _case("sigma fp64 hubbard small", "sigma", "hubbard", 12, 64, precision="fp64"),
        # a long chain at M = 512 (C4's bond), FP64
        _case("sigma fp64 hubbard", "sigma", "hubbard", 32, 512, precision="fp64"),
        # the FP64 product that the FP64 sweep and every accepted split energy of C2 take
        _case("sigma fp64 qc", "sigma", "qc", 20, 512, precision="fp64"),
        # a chain of the scan (C3) swept by itself in split precision
        _case("sigma split hubbard", "sigma", "hubbard", 24, 256, precision="split"),
        # the Davidson product of C2 in split precision
        _case("sigma split qc", "sigma", "qc", 20, 512, precision="split"),
        # renormalisation at the end of a C2 bond step, forward; and backward at odd sizes
        _case("renormalize qc forward", "renormalize", "qc", 20, 512, forward=True),
        _case("renormalize qc backward", "renormalize", "qc", 13, 203, forward=False),
        # the merged operator and the preconditioner's diagonal at the start of a bond step
        _case("merged operator qc", "merged_operator", "qc", 20, 512, forward=False),
        _case("diagonal qc", "diagonal", "qc", 16, 256),
        # a bond's whole eigenproblem in FP64
        _case("diagonalize hubbard", "diagonalize", "hubbard", 16, 128, tol=1e-10),
        # one bond of the energy gradient (C4)
        _case("gradient hubbard", "gradient", "hubbard", 32, 512),
        # the truncation of a C2 bond
        _case("canonicalize qc", "canonicalize", "qc", 20, 512, forward=True),
    ]


def draw(rng):
    op = rng.choice(["sigma", "sigma", "sigma", "renormalize", "renormalize", "merged_operator", "diagonal",
                     "diagonalize", "gradient", "canonicalize"])
    model = "hubbard" if op in ("diagonalize", "gradient") else rng.choice(["hubbard", "qc", "qc"])
    norb = rng.randint(12, 32) if model == "hubbard" else rng.randint(8, 20)
    M = int(round(math.exp(rng.uniform(math.log(32), math.log(160 if op == "diagonalize" else 512)))))
    c = dict(op=op, model=model, norb=norb, M=M)
    if op == "sigma":
        c["precision"] = rng.choice(["fp64", "fp64", "split"])
    elif op in ("renormalize", "merged_operator", "canonicalize"):
        c["forward"] = rng.random() < 0.5
    elif op == "diagonalize":
        c["tol"] = 1e-10
    return c


# one stream for every context, as one program has
@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


class _Array:
    """A library tensor's device data for torch; keeps the tensor alive."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": (t.nnz,), "typestr": "<f8", "data": (t.device_ptr(), False),
                                         "version": 2}


def _view(t):
    return torch.as_tensor(_Array(t), device="cuda")


def prepare(case, seed):
    from mpsxx_gb300 import core

    ctx = core.Context(0, _stream().cuda_stream)
    core.set_precision(ctx, core.SPLIT_TF32 if case.get("precision") == "split" else core.FP64)
    st = {"case": case, "ctx": ctx}
    for name, (lay, x) in _inputs(case, seed).items():
        if name.startswith("mpo"):
            t = core.Tensor.create(ctx, (0, 0), lay["qshape"], [[1] * len(q) for q in lay["qshape"]], lay["tags"])
            t.upload(x)
        else:
            t = core.Tensor.create(ctx, lay.q, lay.qshape, lay.dshape)
            _view(t).copy_(x)
        st[name] = t
    if "psi" in st:
        st["out"] = st["psi"].like()
        st["out_data"], st["psi_data"] = _view(st["out"]), _view(st["psi"])
    if case["op"] in ("diagonal", "diagonalize"):
        s = _structure(case["model"], case["norb"], case["M"])["psi"]
        st["diag"] = core.Tensor.create(ctx, s.q, s.qshape, s.dshape)
        st["diag_data"] = _view(st["diag"])
        if case["op"] == "diagonalize":
            torch.cuda.synchronize()
            core.compute_diagonal_elements(ctx, st["L"], st["R"], st["diag"])
    torch.cuda.synchronize()
    return st


def run(st):
    from mpsxx_gb300 import core

    case, ctx = st["case"], st["ctx"]
    op = case["op"]
    with torch.cuda.stream(_stream()):
        if op == "sigma":
            st["out_data"].zero_()
            core.compute_sigma_vector(ctx, st["L"], st["R"], st["psi"], st["out"])
            return st["out_data"]
        if op == "diagonal":
            st["diag_data"].zero_()
            core.compute_diagonal_elements(ctx, st["L"], st["R"], st["diag"])
            return st["diag_data"]
        if op == "diagonalize":
            st["out_data"].copy_(st["psi_data"])
            e, _ = core.diagonalize(ctx, st["L"], st["R"], st["diag"], st["out"], case["tol"])
            return {"energy": e, "wavefunction": st["out_data"]}
        if op == "renormalize":
            return _view(core.renormalize(ctx, case["forward"], st["O"], st["U"], st["U"]))
        if op == "merged_operator":
            side = case["forward"]
            return _view(core.compute_merged_operator(ctx, side, st["mpo%d" % side], st["env%d" % side]))
        if op == "gradient":
            gl, gr = core.mpo_gradient(ctx, st["mpo1"], st["mpo0"], st["env1"], st["env0"], st["psi"])
            return {"left": gl, "right": gr}
        lm, rm = core.canonicalize(ctx, case["forward"], st["psi"], case["M"])
        return {"left": _view(lm), "right": _view(rm)}


# --------------------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------------------
def _sigma_flops(s):
    da, db = np.array(s["A"][1], dtype=float), np.array(s["B"][1], dtype=float)
    place = {tuple(x): 1 for x in s["psi"].index.tolist()}
    col = {i: j for i, j in place}          # A sector -> its B sector
    row = {j: i for i, j in place}
    f = 0.0
    for i, _, j in s["L"].index.tolist():   # L[A,w,A'] psi[A',B']
        if j in col:
            f += 2 * da[i] * da[j] * db[col[j]]
    for i, _, j in s["R"].index.tolist():   # (L psi)[A,(w,B')] R[B,(w,B')]
        if i in row and j in row:
            f += 2 * da[row[i]] * db[i] * db[j]
    return f


def _renorm_flops(lay, d, k):
    f = 0.0
    for i, _, j in lay.index.tolist():
        if k[i]:
            f += 2.0 * k[i] * d[i] * d[j]
            if k[j]:
                f += 2.0 * k[i] * d[j] * k[j]
    return f


def work(case):
    s = _structure(case["model"], case["norb"], case["M"])
    op, fw = case["op"], case.get("forward", True)
    L, R, psi = s["L"], s["R"], s["psi"]
    if op in ("sigma", "diagonalize"):
        times = 12 if op == "diagonalize" else 1  # a Davidson run takes about a dozen products
        return {"bytes": times * 8 * (L.nnz + R.nnz + 2 * psi.nnz), "flops": times * float(_sigma_flops(s))}
    if op == "diagonal":
        tied = sum(x.dshape[0][i] for x in (L, R) for i, _, j in x.index.tolist() if i == j)
        f = sum(2.0 * p * int(np.sum((L.index[:, 0] == i) & (L.index[:, 2] == i)))
                for (i, _), p in zip(psi.index.tolist(), psi.size.tolist()))
        return {"bytes": 8 * (tied + psi.nnz), "flops": f}
    if op == "canonicalize":
        f = sum(14.0 * x * min(psi.dshape[0][i], psi.dshape[1][j]) for (i, j), x in zip(psi.index, psi.size.tolist()))
        return {"bytes": 24 * psi.nnz, "flops": f}
    if op == "renormalize":
        lay, (_, d, _) = (L, s["A"]) if fw else (R, s["B"])
        k = _kept(d, case["M"])
        out = sum(k[i] * k[j] for i, _, j in lay.index.tolist())
        return {"bytes": 8 * (lay.nnz + sum(a * b for a, b in zip(d, k)) + out), "flops": _renorm_flops(lay, d, k)}
    sides = (True, False) if op == "gradient" else (fw,)
    b = f = 0.0
    for side in sides:
        site = _site(case["model"], case["norb"], case["M"], side)
        axis = 0 if side else 3
        nr = site["nright"]
        per = np.bincount([t // (16 * nr) if axis == 0 else t % nr for t in site["tags"]],
                          minlength=len(site["env"].qshape[1]))
        f += 2.0 * float(np.sum(per[site["env"].index[:, 1]] * site["env"].size))
        b += 8 * site["env"].nnz
        if op == "merged_operator":
            b += 8 * (L if side else R).nnz
    if op == "gradient":
        d = s["A"][1]
        b += 8 * psi.nnz
        # the adjoint of each merged operator: two contractions with psi
        f += 2 * _sigma_flops(s)
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------------------------
# the same results by definition, in 64 bits
# --------------------------------------------------------------------------------------
def _groups(lay):
    """Blocks of an operator by outer sectors: (i, j) -> ([w], [block])."""
    g = {}
    for b, (i, w, j) in enumerate(lay.index.tolist()):
        g.setdefault((i, j), []).append((w, b))
    return g


def _stack(lay, x, blocks, di, dj):
    """Blocks of equal shape as one [n, di, dj] array."""
    off = torch.as_tensor(lay.off[blocks], device="cuda")
    return x[off[:, None] + torch.arange(di * dj, device="cuda")[None, :]].view(len(blocks), di, dj)


def _exact_sigma(s, L, R, psi):
    """sum_w L_w psi R_w^T, block by block."""
    lay = s["psi"]
    col = {i: (j, b) for b, (i, j) in enumerate(lay.index.tolist())}
    da, db = s["A"][1], s["B"][1]
    gr = _groups(s["R"])
    out = torch.zeros_like(psi)
    for (i, i2), lw in _groups(s["L"]).items():
        if i not in col or i2 not in col:
            continue
        (j, b), (j2, b2) = col[i], col[i2]
        rb = dict(gr.get((j, j2), []))
        pair = [(x, rb[w]) for w, x in lw if w in rb]
        if not pair:
            continue
        lx = _stack(s["L"], L, [x for x, _ in pair], da[i], da[i2])
        rx = _stack(s["R"], R, [y for _, y in pair], db[j], db[j2])
        t = torch.matmul(lx, lay.block(psi, b2))                                   # [w, dA, dB']
        lay.block(out, b).add_(t.permute(1, 0, 2).reshape(da[i], -1) @ rx.permute(0, 2, 1).reshape(-1, db[j]))
    return out


def _exact_merged(site, forward, env, coef, out_lay):
    """The merged operator in out_lay's blocks."""
    place, dims = site["merged"][2], out_lay.dshape[0]
    lay, nr = site["env"], site["nright"]
    ent = {}
    for t, c in zip(site["tags"], coef):
        w, sx, tx, v = t // (16 * nr), (t // (4 * nr)) % 4, (t // nr) % 4, t % nr
        con, out = (w, v) if forward else (v, w)
        ent.setdefault((sx, tx), []).append((con, out, float(c)))
    nout = len(out_lay.qshape[1])
    C = {}
    for k, e in ent.items():
        m = torch.zeros(nout, len(lay.qshape[1]), device="cuda", dtype=torch.float64)
        m[[x[1] for x in e], [x[0] for x in e]] = torch.tensor([x[2] for x in e], device="cuda", dtype=torch.float64)
        C[k] = m
    res = torch.zeros(out_lay.nnz, device="cuda", dtype=torch.float64)
    groups = _groups(out_lay)
    for (a, x), ws in _groups(lay).items():
        da, dx = lay.dshape[0][a], lay.dshape[2][x]
        E = _stack(lay, env, [b for _, b in ws], da, dx).reshape(len(ws), -1)
        wi = [w for w, _ in ws]
        for (sx, tx), m in C.items():
            A, ro = place[(a, sx) if forward else (sx, a)]
            A2, co = place[(x, tx) if forward else (tx, x)]
            dst = groups.get((A, A2))
            if not dst:
                continue
            rows = [u for u, _ in dst]
            v = (m[rows][:, wi] @ E).view(len(rows), da, dx)
            off = torch.as_tensor(out_lay.off[[b for _, b in dst]], device="cuda")
            at = (off[:, None, None] + (ro + torch.arange(da, device="cuda"))[None, :, None] * dims[A2]
                  + co + torch.arange(dx, device="cuda")[None, None, :])
            res[at] += v
    return res


def _merged_layout(site, forward):
    """Blocks of the merged operator: the places that some entry of the MPO reaches."""
    q, d, place = site["merged"]
    nr = site["nright"]
    other = site["qshape"][3 if forward else 0]
    lay = Layout((0, 0), [q, other, _neg(q)], [d, [1] * len(other), d])
    reach = set()
    by_con = {}
    for t in site["tags"]:
        w, sx, tx, v = t // (16 * nr), (t // (4 * nr)) % 4, (t // nr) % 4, t % nr
        con, out = (w, v) if forward else (v, w)
        by_con.setdefault(con, []).append((sx, tx, out))
    for a, c, x in site["env"].index.tolist():
        for sx, tx, out in by_con.get(c, []):
            A = place[(a, sx) if forward else (sx, a)][0]
            A2 = place[(x, tx) if forward else (tx, x)][0]
            reach.add((A, out, A2))
    keep = np.array([tuple(i) in reach for i in lay.index.tolist()], dtype=bool)
    lay.index, lay.size = lay.index[keep], lay.size[keep]
    lay.off = np.concatenate([[0], np.cumsum(lay.size)])
    lay.nnz = int(lay.off[-1])
    return lay


def _exact_gradient(s, sites, inp):
    psi = inp["psi"][1]
    lay = s["psi"]
    col = {i: (j, b) for b, (i, j) in enumerate(lay.index.tolist())}
    row = {j: (i, b) for b, (i, j) in enumerate(lay.index.tolist())}
    out = []
    for side in (True, False):  # the site whose coefficients are differentiated
        other = not side
        olay = _merged_layout(sites[other], other)
        O = _exact_merged(sites[other], other, inp["env%d" % other][1], inp["mpo%d" % other][1], olay)
        # Y[A,w,A'] = psi[A,B] O[B,w,B'] psi[A',B'] (left site), its mirror image (right site)
        Y = {}
        d = olay.dshape[0]
        for (x, y), ws in _groups(olay).items():
            pick = row if side else col
            if x not in pick or y not in pick:
                continue
            (i, bi), (j, bj) = pick[x], pick[y]
            O3 = _stack(olay, O, [b for _, b in ws], d[x], d[y])
            pi, pj = lay.block(psi, bi), lay.block(psi, bj)
            if not side:
                pi, pj = pi.T, pj.T
            Y[i, j] = ({w: n for n, (w, _) in enumerate(ws)}, pi @ O3 @ pj.T)
        site = sites[side]
        env_lay, env = inp["env%d" % side]
        place, nr = site["merged"][2], site["nright"]
        E = {}
        for (a, x), ws in _groups(env_lay).items():
            E[a, x] = ({w: n for n, (w, _) in enumerate(ws)},
                       _stack(env_lay, env, [b for _, b in ws], env_lay.dshape[0][a], env_lay.dshape[2][x]))
        acc = torch.zeros(len(site["tags"]), device="cuda", dtype=torch.float64)
        for (a, x), (wn, e3) in E.items():
            da, dx = e3.shape[1:]
            for sx in range(4):
                for tx in range(4):
                    A, ro = place[(a, sx) if side else (sx, a)]
                    A2, co = place[(x, tx) if side else (tx, x)]
                    if (A, A2) not in Y:
                        continue
                    un, y3 = Y[A, A2]
                    sub = y3[:, ro:ro + da, co:co + dx].reshape(y3.shape[0], -1)
                    dots = e3.reshape(e3.shape[0], -1) @ sub.T
                    idx, p, r = [], [], []
                    for n, t in enumerate(site["tags"]):
                        if (t // (4 * nr)) % 4 != sx or (t // nr) % 4 != tx:
                            continue
                        con, o = (t // (16 * nr), t % nr) if side else (t % nr, t // (16 * nr))
                        if con in wn and o in un:
                            idx.append(n)
                            p.append(wn[con])
                            r.append(un[o])
                    if idx:
                        acc[idx] += dots[p, r]
        out.append(acc)
    return {"left": out[0], "right": out[1]}


def _exact_ground_state(s, L, R, psi):
    """Lowest eigenvalue by a Davidson iteration without restarts."""
    diag = _exact_diagonal(s, L, R)
    v = psi / psi.norm()
    V, S = v[:, None], _exact_sigma(s, L, R, v)[:, None]
    for _ in range(120):
        h = V.T @ S
        e, c = torch.linalg.eigh(0.5 * (h + h.T))
        x, r = V @ c[:, 0], S @ c[:, 0] - e[0] * (V @ c[:, 0])
        if r.norm() < 1e-12 * max(1.0, abs(float(e[0]))):
            break
        den = e[0] - diag
        t = r / torch.where(den.abs() < 1e-8, torch.full_like(den, 1e-8), den)
        for _ in range(3):
            t = t / t.norm()
            t = t - V @ (V.T @ t)
        t = t / t.norm()
        V = torch.cat([V, t[:, None]], 1)
        S = torch.cat([S, _exact_sigma(s, L, R, t)[:, None]], 1)
    return float(e[0])


def _exact_diagonal(s, L, R):
    lay = s["psi"]
    gl, gr = _groups(s["L"]), _groups(s["R"])
    out = torch.zeros(lay.nnz, device="cuda", dtype=torch.float64)
    da, db = s["A"][1], s["B"][1]
    for b, (i, j) in enumerate(lay.index.tolist()):
        rb = dict(gr.get((j, j), []))
        pair = [(x, rb[w]) for w, x in gl.get((i, i), []) if w in rb]
        if pair:
            dl = _stack(s["L"], L, [x for x, _ in pair], da[i], da[i]).diagonal(dim1=1, dim2=2)
            dr = _stack(s["R"], R, [y for _, y in pair], db[j], db[j]).diagonal(dim1=1, dim2=2)
            lay.block(out, b).copy_(dl.T @ dr)
    return out


def exact(case, seed):
    op, fw = case["op"], case.get("forward", True)
    if op == "canonicalize":
        return None  # singular vectors have no value of their own (signs)
    s = _structure(case["model"], case["norb"], case["M"])
    inp = _inputs(case, seed)
    if op == "sigma":
        return _exact_sigma(s, inp["L"][1], inp["R"][1], inp["psi"][1])
    if op == "diagonal":
        return _exact_diagonal(s, inp["L"][1], inp["R"][1])
    if op == "diagonalize":
        # (the eigenvector's sign is free)
        return {"energy": _exact_ground_state(s, inp["L"][1], inp["R"][1], inp["psi"][1]), "wavefunction": None}
    if op == "renormalize":
        lay, x = inp["O"]
        ul, u = inp["U"]
        at = {int(k[0 if fw else 1]): (int(k[1 if fw else 0]), b) for b, k in enumerate(ul.index)}
        q, d = (_neg(ul.qshape[1]), ul.dshape[1]) if fw else (_neg(ul.qshape[0]), ul.dshape[0])
        out_lay = Layout((0, 0), [q, lay.qshape[1], _neg(q)], [d, lay.dshape[1], d])
        out = torch.zeros(out_lay.nnz, device="cuda", dtype=torch.float64)
        og = _groups(out_lay)
        for (i, j), ws in _groups(lay).items():
            if i not in at or j not in at:
                continue
            (a, bi), (c, bj) = at[i], at[j]
            ui, uj = ul.block(u, bi), ul.block(u, bj)
            if not fw:
                ui, uj = ui.T, uj.T
            r = ui.T @ _stack(lay, x, [b for _, b in ws], lay.dshape[0][i], lay.dshape[2][j]) @ uj
            off = torch.as_tensor(out_lay.off[[b for _, b in og[a, c]]], device="cuda")
            out[off[:, None] + torch.arange(r[0].numel(), device="cuda")[None, :]] = r.reshape(r.shape[0], -1)
        return out
    sites = {x: _site(case["model"], case["norb"], case["M"], x) for x in (True, False)}
    if op == "merged_operator":
        lay = _merged_layout(sites[fw], fw)
        return _exact_merged(sites[fw], fw, inp["env%d" % fw][1], inp["mpo%d" % fw][1], lay)
    return _exact_gradient(s, sites, inp)
