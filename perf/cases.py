"""The work that users of this library have it do, as cases that a timing program can run.

A case is one of four kinds:

* ``stack``     one ``Kernel.call`` on a stack of equal block triples on the device, the drop-in
                for the reference's ``Kernel<T>::call``;
* ``contract``  one block-sparse contraction (or ``steps`` of them, the later ones added into the
                same C with beta = 1) through ``contract``, planning included;
* ``plan``      one execute of a plan that the program keeps, for patterns that stay;
* ``serve``     a burst of requests through a running ``Server``, waited for.

The block-sparse families are the repository's four workloads (c0 .. c3: see
``shtensor_b200/workloads.py``) at their own sizes and at fractions of them.  A case fixes the
sparsity pattern; the seed draws the values.  Patterns, values and the 64-bit results are made
here, so they do not depend on the library.
"""
import math

import numpy as np
import torch

import shtensor_b200 as sht

MODES = {"plain": sht.Mode.PLAIN_FP64, "batched": sht.Mode.BATCHED_FP64, "split": sht.Mode.SPLIT}
EXPR = {"c0": "ijl, lk -> ijk", "c1": "iaP, jbP -> ijab", "c2": "iaP, jbP -> ijab", "c3": "abcd, cdij -> abij"}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's own block-kernel test: a short stack of small blocks, one call of launch latency
        _stack("stack_f64_short", "ikl, ljk -> ij", "8,8,8", "8,8,8", 64, "f64"),
        # the same blocks as a long stack, as a block-sparse driver collects them: memory-bound
        _stack("stack_f64_long", "ikl, ljk -> ij", "8,8,8", "8,8,8", 10000, "f64"),
        # Kernel<float> on ragged c0 blocks (odd extents, three free modes)
        _stack("stack_f32_ragged", "ijl, lk -> ijk", "13,9,11", "11,15", 5000, "f32"),
        # c1's block products, the largest blocks the stack kernel meets
        _stack("stack_f64_blocks", "iaP, jbP -> ijab", "13,32,64", "9,25,64", 64, "f64"),
        # a small contraction into a new C in the default mode: matching, growth of C's pattern, launches
        _contract("c0_plain_new", "c0", "plain", scale=1.0, occupancy=0.3, new=True),
        # the same size in the batched form, two products added up in one C (beta = 0, then 1)
        _contract("c0_batched_sum", "c0", "batched", scale=1.0, occupancy=0.3, steps=2),
        # the benchmark's contraction at full size in each of the three forms
        _contract("c1_plain", "c1", "plain", scale=1.0, occupancy=0.15),
        _contract("c1_batched", "c1", "batched", scale=1.0, occupancy=0.15),
        _contract("c1_split", "c1", "split", scale=1.0, occupancy=0.15),
        # order 4 x order 4 with few, large blocks and norm screening
        _contract("c3_split_screened", "c3", "split", scale=0.125),
        # the same patterns contracted again and again: a kept plan, only its execute
        _plan("c3_batched_plan", "c3", "batched", scale=0.125),
        # a burst of mixed requests at a server in the split form
        {"name": "serve_split_burst", "kind": "serve", "mode": "split", "requests": 12, "scale": 0.5, "pattern": 1},
    ]


def _stack(name, expr, sa, sb, ops, dtype):
    return {"name": name, "kind": "stack", "expr": expr, "sa": sa, "sb": sb, "ops": ops, "dtype": dtype}


def _contract(name, family, mode, scale, occupancy=0.15, steps=1, new=False, pattern=1):
    return {"name": name, "kind": "contract", "family": family, "mode": mode, "scale": scale, "occupancy": occupancy,
            "steps": steps, "new": new, "pattern": pattern}


def _plan(name, family, mode, scale, occupancy=0.15, pattern=1):
    return {"name": name, "kind": "plan", "family": family, "mode": mode, "scale": scale, "occupancy": occupancy,
            "pattern": pattern}


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["stack", "stack", "contract", "contract", "contract", "plan", "serve"])
    if kind == "stack":
        expr = rng.choice(["ik, kj -> ij", "ikl, ljk -> ij", "kil, ljk -> ji", "ikl, lkmj -> mij", "ijl, lk -> ijk",
                           "iaP, jbP -> ijab", "abcd, cdij -> abij"])
        left, right = (s.strip() for s in expr.split("->")[0].split(","))
        top = {4: 12, 3: 16, 2: 64}[max(len(left), len(right))]
        ext = {c: rng.randint(2, top) for c in left + right}
        if expr == "iaP, jbP -> ijab":
            ext |= {"a": rng.randint(5, 32), "b": rng.randint(5, 32), "P": rng.randint(8, 64)}
        elems = sum(math.prod(ext[c] for c in s) for s in (left, right, expr.split("->")[1].strip()))
        ops = max(1, int(min(_log(rng, 1, 20000), 3e7 / elems, 2e10 / _stack_flops(left, right, ext))))
        return {"kind": "stack", "expr": expr, "sa": ",".join(str(ext[c]) for c in left),
                "sb": ",".join(str(ext[c]) for c in right), "ops": ops, "dtype": rng.choice(["f64", "f64", "f32"])}
    if kind == "serve":
        return {"kind": "serve", "mode": rng.choice(["batched", "split"]), "requests": rng.randint(3, 14),
                "scale": round(_log(rng, 0.2, 0.5), 3), "pattern": rng.randint(2, 10 ** 6)}
    family, mode = rng.choice(["c0", "c1", "c2", "c3"]), rng.choice(["plain", "batched", "split"])
    if family == "c3":
        # fewer blocks in the plain form, which takes longer for them than the largest listed case
        scale = _log(rng, 0.05, 0.08 if mode == "plain" else 0.12)
    else:
        scale = _log(rng, 0.2, 0.9)
    case = {"kind": kind, "family": family, "mode": mode, "scale": round(scale, 3),
            "occupancy": round(rng.uniform(0.05, 0.15 if family != "c0" else 0.4), 3), "pattern": rng.randint(2, 10 ** 6)}
    if kind == "contract":
        # two products at full size would cost more than the largest listed case
        small = family == "c0" or (family != "c3" and scale < 0.7)
        case |= {"steps": rng.choice([1, 2]) if small else 1, "new": rng.random() < 0.3}
    return case


# ------------------------------------------------------------------ patterns
class Blocks:
    """The pattern of one block-sparse tensor in the library's layout: ids ascending, blocks packed."""

    def __init__(self, sizes, keep, factor=None):
        self.sizes = [list(map(int, s)) for s in sizes]
        nblk = [len(s) for s in self.sizes]
        ids = np.arange(math.prod(nblk), dtype=np.int64)
        stride = np.concatenate([[1], np.cumprod(nblk)[:-1]]).astype(np.int64)
        coords = np.stack([(ids // stride[d]) % nblk[d] for d in range(len(nblk))], axis=1)
        mask = keep(coords)
        self.ids, self.coords, self.stride = ids[mask], coords[mask], stride
        self.dims = np.stack([np.asarray(s, np.int64)[self.coords[:, d]] for d, s in enumerate(self.sizes)], axis=1)
        self.elems = self.dims.prod(axis=1) if len(self.ids) else np.zeros(0, np.int64)
        self.offsets = np.concatenate([[0], np.cumsum(self.elems)]).astype(np.int64)
        self.nnz = int(self.offsets[-1])
        self.factor = np.ones(len(self.ids)) if factor is None else factor(self.coords)

    def lists(self):
        return [self.coords[:, d].astype(np.int32) for d in range(self.coords.shape[1])]

    def values(self, gen, uniform):
        """Values on the GPU: uniform in [-1, 1] or normal, times the block's factor."""
        v = torch.empty(self.nnz, dtype=torch.float64, device="cuda")
        v = v.uniform_(-1.0, 1.0, generator=gen) if uniform else v.normal_(generator=gen)
        if np.any(self.factor != 1.0):
            f = torch.from_numpy(self.factor).cuda()
            v *= torch.repeat_interleave(f, torch.from_numpy(self.elems).cuda())
        return v


def _extent(rng, extent, choices):
    sizes = []
    while sum(sizes) < extent:
        sizes.append(int(rng.choice(choices)))
    return sizes


def _family(family, scale, occupancy, pattern):
    """(A, B, block sizes of C, screening threshold) of one contraction of a family."""
    rng = np.random.default_rng(pattern)
    some = lambda c: rng.random(len(c)) < occupancy  # noqa: E731
    if family == "c0":
        i, j, l, k = (list(rng.integers(5, 16, max(2, round(20 * scale)))) for _ in range(4))
        return Blocks([i, j, l], some), Blocks([l, k], some), [i, j, k], 0.0
    if family in ("c1", "c2"):
        i, j = (_extent(rng, 64 * scale, [5, 9, 13]) for _ in range(2))
        a, b = (_extent(rng, 512 * scale, [13, 25, 32]) for _ in range(2))
        P = _extent(rng, 2048 * scale, [32, 48, 64])
        if family == "c2":
            fa = fb = lambda c: 10.0 ** rng.uniform(-6.0, 2.0, len(c))  # noqa: E731
        else:
            def decay(nx):
                return lambda c: np.exp(-np.abs(c[:, 1] - np.rint(c[:, 2] * (nx - 1) / max(len(P) - 1, 1))) / 4.0)
            fa, fb = decay(len(a)), decay(len(b))
        return Blocks([i, a, P], some, fa), Blocks([j, b, P], some, fb), [i, j, a, b], 0.0
    a, b, c, d = (_extent(rng, 768 * scale, np.arange(24, 49)) for _ in range(4))
    i, j = (_extent(rng, max(96 * scale, 8), np.arange(8, 17)) for _ in range(2))
    spread = lambda x: x.max(axis=1) - x.min(axis=1)  # noqa: E731
    delta = lambda x: np.abs(x[:, 0] - x[:, 1]) + np.abs(x[:, 2] - x[:, 3])  # noqa: E731
    V = Blocks([a, b, c, d], lambda x: np.exp(-0.5 * spread(x)) >= 0.1, lambda x: np.exp(-0.5 * spread(x)))
    T = Blocks([c, d, i, j], lambda x: np.exp(-0.5 * delta(x)) >= 1e-10, lambda x: np.exp(-0.5 * delta(x)))
    return V, T, [a, b, i, j], 1e-10


def _letters(expr):
    left, out = expr.split("->")
    x, y = left.split(",")
    return x.strip(), y.strip(), out.strip()


def _pairs(expr, A, B, eps, na, nb):
    """Storage positions of the block pairs that meet, and the C block coordinates of each."""
    x, y, out = _letters(expr)
    con = [c for c in x if c in y]
    key = lambda T, s: [tuple(r) for r in T.coords[:, [s.index(c) for c in con]].tolist()]  # noqa: E731
    of_b = {}
    for n, k in enumerate(key(B, y)):
        of_b.setdefault(k, []).append(n)
    ia, ib = [], []
    for n, k in enumerate(key(A, x)):
        m = of_b.get(k, [])
        ia += [n] * len(m)
        ib += m
    ia, ib = np.asarray(ia, np.int64), np.asarray(ib, np.int64)
    if eps > 0:
        kept = na[ia] * nb[ib] >= eps
        ia, ib = ia[kept], ib[kept]
    c = np.stack([A.coords[ia, x.index(q)] if q in x else B.coords[ib, y.index(q)] for q in out], axis=1)
    return ia, ib, c


def _work_of(family, scale, occupancy, pattern):
    expr = EXPR[family]
    A, B, sizes, eps = _family(family, scale, occupancy, pattern)
    norm = lambda T: T.factor * np.sqrt(T.elems)  # noqa: E731  expected block norms
    ia, ib, c = _pairs(expr, A, B, eps, norm(A), norm(B))
    x, y, out = _letters(expr)
    ext = np.ones(len(ia))
    for q in set(x + y):
        ext = ext * (A.dims[ia, x.index(q)] if q in x else B.dims[ib, y.index(q)])
    u = np.unique(c, axis=0)
    nnz_c = sum(int(math.prod(sizes[d][r[d]] for d in range(len(sizes)))) for r in u.tolist())
    return {"bytes": 8.0 * (A.nnz + B.nnz + nnz_c), "flops": 2.0 * float(ext.sum()), "nnz_c": nnz_c}


def _requests(case):
    """The requests of a serving burst: families in turn, extents and occupancies as a mixed load has them."""
    rng = np.random.default_rng(case["pattern"])
    got = []
    for n in range(case["requests"]):
        family = ("c0", "c1", "c2", "c3")[n % 4]
        u = float(rng.uniform(0.5, 1.0)) * case["scale"]
        got.append((family, 0.125 * u if family == "c3" else u, float(rng.uniform(0.05, 0.3)), int(rng.integers(1, 1 << 30))))
    return got


def _stack_flops(left, right, ext):
    return 2.0 * math.prod(ext[c] for c in set(left + right))


def work(case):
    if case["kind"] == "stack":
        x, y, out = _letters(case["expr"])
        ext = dict(zip(x, map(int, case["sa"].split(",")))) | dict(zip(y, map(int, case["sb"].split(","))))
        elems = sum(math.prod(ext[c] for c in s) for s in (x, y, out))
        return {"bytes": float(case["ops"] * elems * (8 if case["dtype"] == "f64" else 4)),
                "flops": case["ops"] * _stack_flops(x, y, ext)}
    if case["kind"] == "serve":
        each = [_work_of(*r) for r in _requests(case)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    w = _work_of(case["family"], case["scale"], case["occupancy"], case["pattern"])
    steps = case.get("steps", 1)
    # a later product reads C as well as writing it, and takes operands of its own
    return {"bytes": steps * w["bytes"] + (steps - 1) * 8.0 * w["nnz_c"], "flops": steps * w["flops"]}


# ------------------------------------------------------------------ states
class _Memory:
    """A tensor's device data for torch (kept alive by the torch tensor made from it)."""

    def __init__(self, tensor):
        self.tensor, self.ptr = tensor, tensor.device_ptr()
        self.__cuda_array_interface__ = {"shape": (tensor.nnz,), "typestr": "<f8", "data": (self.ptr, False), "version": 3,
                                         "strides": None}


def _data(tensor):
    return torch.as_tensor(_Memory(tensor), device="cuda")


class State:
    """What a program holds before the call, besides its context and its server."""

    def __init__(self, case):
        self.case, self.seen = case, {}

    def view(self, tensor):
        """torch's view of C, made again only when C has moved."""
        old = self.seen.get(id(tensor))
        if old is None or old[0] != (tensor.device_ptr(), tensor.nnz):
            old = self.seen[id(tensor)] = ((tensor.device_ptr(), tensor.nnz), _data(tensor))
        return old[1]


_MADE = {}


def _context():
    """The program's context: one device pool for all its tensors, plans and scratch."""
    if "ctx" not in _MADE:
        _MADE["ctx"] = sht.Context(60 << 30)
    return _MADE["ctx"]


def _server(mode):
    """The program's server of a form, with a context of its own (a server's context is its own to plan in)."""
    if mode not in _MADE:
        ctx = sht.Context(24 << 30)
        _MADE[mode] = (ctx, sht.Server(ctx, mode=MODES[mode]))
    return _MADE[mode]


def _resident(ctx, blocks, values):
    t = sht.Tensor(ctx, blocks.sizes).reserve(blocks.lists())
    if blocks.nnz:
        _data(t).copy_(values)
    return t


def _empty(ctx, sizes):
    return sht.Tensor(ctx, sizes).reserve([[] for _ in sizes])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))


def _operands(case, seed):
    """[(A, values, B, values)] of the steps; every step has the pattern and values of its own."""
    gen = _generator(seed)
    got = []
    for _ in range(case.get("steps", 1)):
        A, B, sizes, eps = _family(case["family"], case["scale"], case["occupancy"], case["pattern"])
        uni = case["family"] == "c0"
        got.append((A, A.values(gen, uni), B, B.values(gen, uni)))
    return got, sizes, eps


def _stack_inputs(case, seed):
    x, y, out = _letters(case["expr"])
    sa, sb = (list(map(int, case[s].split(","))) for s in ("sa", "sb"))
    ext = dict(zip(x, sa)) | dict(zip(y, sb))
    sc = [ext[c] for c in out]
    gen = _generator(seed)
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    a, b = (torch.empty(case["ops"] * math.prod(s), dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=gen)
            for s in (sa, sb))
    return a, b, sa, sb, sc, dt


def prepare(case, seed):
    s = State(case)
    if case["kind"] == "stack":
        a, b, sa, sb, sc, dt = _stack_inputs(case, seed)
        s.kernel = sht.Kernel(_context(), case["expr"], sa, sb, sc, 1.0, 0.0, sht.KernelType.XMM,
                              np.float64 if case["dtype"] == "f64" else np.float32)
        s.a, s.b, s.c = a, b, torch.zeros(case["ops"] * math.prod(sc), dtype=dt, device="cuda")
        return s
    if case["kind"] == "serve":
        gen = _generator(seed)
        ctx, s.server = _server(case["mode"])
        s.requests = []
        for r in _requests(case):
            A, B, sizes, eps = _family(*r)
            a, b = A.values(gen, r[0] == "c0"), B.values(gen, r[0] == "c0")
            s.requests.append((EXPR[r[0]], _resident(ctx, A, a), _resident(ctx, B, b), _empty(ctx, sizes), eps))
        return s
    ops, s.sizes, s.eps = _operands(case, seed)
    s.ctx, s.expr, s.mode = _context(), EXPR[case["family"]], MODES[case["mode"]]
    s.steps = [(_resident(s.ctx, A, a), _resident(s.ctx, B, b)) for A, a, B, b in ops]
    s.c = _empty(s.ctx, s.sizes)
    if case["kind"] == "plan":
        s.plan = sht.Plan(s.ctx, s.expr, s.steps[0][0], s.steps[0][1], s.c, s.eps, mode=s.mode)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "stack":
        return s.kernel.call(s.a, s.b, s.c, s.case["ops"])
    if kind == "plan":
        s.plan.execute(1.0, 0.0)
        return s.view(s.c)
    if kind == "serve":
        ids = [s.server.submit(e, 1.0, A, B, 0.0, C, eps) for e, A, B, C, eps in s.requests]
        for i in ids:
            s.server.wait(i)
        return [s.view(r[3]) for r in s.requests]
    c = _empty(s.ctx, s.sizes) if s.case["new"] else s.c
    beta, pairs = 0.0, []
    for A, B in s.steps:
        pairs.append(sht.contract(s.ctx, s.expr, 1.0, A, B, beta, c, s.eps, mode=s.mode)["npairs"])
        beta = 1.0
    return {"c": _data(c) if s.case["new"] else s.view(c), "pairs": pairs}


# ------------------------------------------------------------------ the values in 64 bits
def _matrix(block, dims, letters, order):
    """A column-major block as the matrix whose index order is `order`'s first letters, then its others."""
    t = block.view([int(d) for d in dims[::-1]])
    back = letters[::-1]
    return t.permute([back.index(c) for c in order])


def _contracted(expr, sizes, eps, ops):
    """The C data (blocks ascending by id, packed) of the sum of the products, and the pairs of each."""
    x, y, out = _letters(expr)
    con = [c for c in x if c in y]
    fa, fb = [c for c in x if c not in y], [c for c in y if c not in x]
    stride = np.concatenate([[1], np.cumprod([len(s) for s in sizes])[:-1]]).astype(np.int64)
    acc, where = {}, {}
    for A, a, B, b in ops:
        def norms(T, v):
            return np.array([float(v[T.offsets[n]:T.offsets[n + 1]].norm()) for n in range(len(T.ids))]) if eps > 0 else None
        ia, ib, c = _pairs(expr, A, B, eps, norms(A, a), norms(B, b))
        used = lambda T, v, n, s, order, rows: _matrix(  # noqa: E731
            v[T.offsets[n]:T.offsets[n + 1]], T.dims[n], s, order).reshape(rows, -1)
        ma = {n: used(A, a, n, x, fa + con, math.prod(A.dims[n, x.index(q)] for q in fa)) for n in set(ia.tolist())}
        mb = {n: used(B, b, n, y, con + fb, math.prod(B.dims[n, y.index(q)] for q in con)) for n in set(ib.tolist())}
        for p, q, r, i in zip(ia.tolist(), ib.tolist(), c.tolist(), (c @ stride).tolist()):
            if i in acc:
                acc[i].addmm_(ma[p], mb[q])
            else:
                acc[i], where[i] = ma[p] @ mb[q], r
        del ma, mb
    parts = []
    for i in sorted(acc):
        d = {q: sizes[n][where[i][n]] for n, q in enumerate(out)}
        t = acc.pop(i).view([d[q] for q in fa + fb])
        parts.append(t.permute([(fa + fb).index(q) for q in out[::-1]]).reshape(-1))
    return torch.cat(parts) if parts else torch.zeros(0, dtype=torch.float64, device="cuda")


def exact(case, seed):
    if case["kind"] == "stack":
        a, b, sa, sb, sc, _ = _stack_inputs(case, seed)
        x, y, out = _letters(case["expr"])
        n = case["ops"]
        # column-major blocks: torch sees the modes in reverse; '.' stands for the stack
        sub = "Z%s,Z%s->Z%s" % (x[::-1], y[::-1], out[::-1])
        return torch.einsum(sub, a.double().view([n] + sa[::-1]), b.double().view([n] + sb[::-1])).reshape(-1)
    if case["kind"] == "serve":
        gen = _generator(seed)
        got = []
        for r in _requests(case):
            A, B, sizes, eps = _family(*r)
            a, b = A.values(gen, r[0] == "c0"), B.values(gen, r[0] == "c0")
            got.append(_contracted(EXPR[r[0]], sizes, eps, [(A, a, B, b)]))
        return got
    ops, sizes, eps = _operands(case, seed)
    c = _contracted(EXPR[case["family"]], sizes, eps, ops)
    return c if case["kind"] == "plan" else {"c": c, "pairs": None}
