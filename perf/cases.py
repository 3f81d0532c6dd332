"""Performance cases of the block-tensor path: what a coupled-cluster program
asks of it, through the public operations of libtensor_b200.core.

    ladder  r(i,j,a,b) = 1/2 sum_cd t(i,j,c,d) V(a,b,c,d)   btod_contract2
    ring    r(i,j,a,b) (+)= sum_kc t(i,k,a,c) W(k,b,c,j)    btod_contract2
    fock    r(i,j,a,c) = sum_d t(i,j,a,d) f(d,c)            btod_contract2
    copy    B = P V                                         btod_copy
    add     r = X - P(ij)X - 1/2 P(ab)X + 1/2 P(ij)P(ab)X   btod_add
    symm    r = X - P(ij)X                                  btod_symmetrize
    dot     <V, P V'>                                       btod_dotprod
    ccd     one amplitude iteration, replayed as a graph

Occupied and virtual dimensions hold the blocks named by `occ` and `vir` once
per spin; with `irreps` block b of a spin carries point-group label b.  A case
is those lists, the operation, its arithmetic (`mode`, `slices`) and options.
exact() gives each result from dense FP64 torch algebra.
"""
import math
from itertools import product

import numpy as np
import torch

from libtensor_b200 import core
from libtensor_b200._capi import check, lib
from libtensor_b200.spec import BTSpec, spin_forbidden

MODES = {"fp64": core.MODE_PLAIN_FP64, "modular": core.MODE_OZAKI_CRT, "bf16": core.MODE_OZAKI_BF16,
         "fp8": core.MODE_OZAKI_FP8, "int8": core.MODE_OZAKI_INT8}
D2H_OCC, D2H_VIR = "6,2,3,1,5,2,3,1", "40,12,18,8,36,10,16,8"
T_SCALE, V_SCALE = 0.05, 1.0


def listed():
    return [
        # the smallest call: a molecule of a few atoms, where launches count
        dict(name="ladder-10-40-fp64", op="ladder", occ="5", vir="16,4", mode="fp64", slices=0),
        # the drop-in FP64 arithmetic at full size
        dict(name="ladder-40-240-fp64", op="ladder", occ="20", vir="48,40,32", mode="fp64", slices=0),
        # blocks as they fall out of a basis: odd extents, no alignment
        dict(name="ladder-26-130-fp64", op="ladder", occ="7,6", vir="29,23,13", mode="fp64", slices=0),
        # the headline: effective FP64 from INT8 products, full size
        dict(name="ladder-40-240-modular", op="ladder", occ="20", vir="64,56", mode="modular", slices=13),
        # the same arithmetic in an ordinary calculation, odd blocks
        dict(name="ladder-20-90-modular", op="ladder", occ="10", vir="25,20", mode="modular", slices=13),
        # reduced-precision iterations far from convergence
        dict(name="ladder-40-240-bf16x4", op="ladder", occ="20", vir="64,56", mode="bf16", slices=4),
        dict(name="ladder-30-150-fp8x8", op="ladder", occ="15", vir="40,35", mode="fp8", slices=8),
        # point-group symmetry: thousands of small blocks, added to a residual
        dict(name="ring-46-296-fp64", op="ring", occ=D2H_OCC, vir=D2H_VIR, irreps=True, mode="fp64", slices=0,
             add=True),
        dict(name="ring-46-296-modular", op="ring", occ=D2H_OCC, vir=D2H_VIR, irreps=True, mode="modular",
             slices=13),
        # antisymmetrising a residual, re-ordering the integrals
        dict(name="add-30-300", op="add", occ="15", vir="50,50,50"),
        dict(name="copy-300", op="copy", occ="15", vir="50,50,50", perm="0,2,1,3"),
        # a whole iteration as a program replays it
        dict(name="ccd-30-300-modular", op="ccd", occ="15", vir="50,50,50", mode="modular", slices=13),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cut(rng, total, most):
    """`total` orbitals of one spin in up to `most` blocks of uneven size."""
    n = rng.randint(1, max(1, min(most, total // 4)))
    w = [rng.uniform(0.6, 1.4) for _ in range(n)]
    sizes = [max(1, int(total * x / sum(w))) for x in w]
    sizes[0] += total - sum(sizes)
    return ",".join(str(s) for s in sizes)


def _like_sized(case):
    """Whether the contracted block pairs of a modular case are all long (about
    a thousand elements) or all short, as blocks of like size give."""
    o, v = ([int(x) for x in case[k].split(",")] for k in ("occ", "vir"))
    for op, left in (("ladder", v), ("ring", o)):
        k = [x * y for x in left for y in v]
        if case["op"] in (op, "ccd") and not (all(x >= 1024 for x in k) or all(x < 1021 for x in k)):
            return False
    return True


def draw(rng):
    while True:
        c = _draw(rng)
        if c.get("mode") != "modular" or c["op"] == "fock" or _like_sized(c):
            return c


def _draw(rng):
    op = rng.choice(["ladder", "ladder", "ladder", "ladder", "ring", "ring", "fock", "copy", "add", "symm", "dot",
                     "ccd"])
    if op in ("copy", "dot"):
        c = dict(op=op, occ="4", vir=_cut(rng, _log_int(rng, 10, 140), 3))
        c["perm"] = ",".join(str(p) for p in rng.choice([(0, 2, 1, 3), (2, 3, 0, 1), (3, 1, 2, 0), (1, 0, 3, 2)])
                             ) if op == "copy" else "1,0,3,2"
        return c
    if op in ("add", "symm", "fock"):
        c = dict(op=op, occ=_cut(rng, _log_int(rng, 3, 20), 2), vir=_cut(rng, _log_int(rng, 12, 140), 3))
        if op == "fock":
            c.update(mode=rng.choice(["fp64", "fp64", "modular"]), add=rng.random() < 0.5)
            c["slices"] = 13 if c["mode"] == "modular" else 0
        return c
    if op == "ccd":
        mode = rng.choice(["fp64", "modular"])
        return dict(op=op, occ=_cut(rng, _log_int(rng, 3, 14), 2), vir=_cut(rng, _log_int(rng, 12, 100), 3),
                    mode=mode, slices=13 if mode == "modular" else 0)
    if op == "ring":
        mode = rng.choice(["fp64", "modular"])
        c = dict(op=op, mode=mode, slices=13 if mode == "modular" else 0, add=rng.random() < 0.5)
        if rng.random() < 0.7:
            n = rng.choice([4, 8])
            c.update(irreps=True, occ=",".join(str(rng.randint(1, 6)) for _ in range(n)),
                     vir=",".join(str(_log_int(rng, 2, 36)) for _ in range(n)))
            if not c["add"] and rng.random() < 0.4:
                c["symm"] = True
        else:
            c.update(occ=_cut(rng, _log_int(rng, 3, 16), 2), vir=_cut(rng, _log_int(rng, 12, 110), 3))
        return c
    mode = rng.choice(["fp64", "fp64", "modular", "modular", "bf16", "fp8", "int8"])
    slices = {"fp64": 0, "modular": 13, "bf16": rng.choice([3, 4, 7]), "fp8": rng.choice([4, 8]), "int8": 7}[mode]
    return dict(op=op, occ=_cut(rng, _log_int(rng, 4, 20), 2), vir=_cut(rng, _log_int(rng, 12, 118), 3), mode=mode,
                slices=slices, add=rng.random() < 0.25)


# ---------------------------------------------------------------- spaces

class Space:
    """A spin-blocked tensor space: block extents per dimension (alpha blocks,
    then beta blocks), permutational (anti)symmetry, as many beta indices in
    `bra` as in `ket`, and labels whose product must be the first irrep."""

    def __init__(self, sizes, perms, bra, ket, labels=None):
        self.sizes, self.perms, self.bra, self.ket, self.labels = sizes, perms, bra, ket, labels
        self.dims = [sum(s) for s in sizes]
        self.n = len(sizes)

    def spec(self):
        splits = [[int(x) for x in np.cumsum(s)[:-1]] for s in self.sizes]
        return BTSpec(dims=list(self.dims), splits=splits, perms=list(self.perms), part_pdims=[2] * self.n,
                      part_forbidden=spin_forbidden([(self.bra, self.ket)], self.n),
                      labels=None if self.labels is None else [list(x) for x in self.labels], label_nirrep=8)

    def permuted(self, p):
        """The space of B, B[y] = A[x] with y[d] = x[p[d]]."""
        inv = [p.index(d) for d in range(self.n)]
        perms = [(tuple(inv[q[p[d]]] for d in range(self.n)), c) for q, c in self.perms]
        return Space([self.sizes[x] for x in p], perms, [inv[d] for d in self.bra], [inv[d] for d in self.ket],
                     None if self.labels is None else [self.labels[x] for x in p])

    def group(self):
        g = [(tuple(range(self.n)), 1.0)]
        for p, c in g:
            for q, cq in self.perms:
                r = tuple(p[k] for k in q)
                if all(r != x for x, _ in g):
                    g.append((r, c * cq))
        return g

    def _spin(self, d, b):
        return int(b >= len(self.sizes[d]) // 2)

    def blocks(self):
        """(start, extent) per dimension and arena offset of every canonical
        block, and the arena's length: canonical is the smallest block index
        of an orbit; blocks start on multiples of four elements."""
        nb = [len(s) for s in self.sizes]
        starts = [np.concatenate([[0], np.cumsum(s)]) for s in self.sizes]
        grp = [p for p, _ in self.group()]
        out, off = [], 0
        for b in product(*[range(x) for x in nb]):
            if sum(self._spin(d, b[d]) for d in self.bra) != sum(self._spin(d, b[d]) for d in self.ket):
                continue
            if self.labels is not None:
                x = 0
                for d in range(self.n):
                    x ^= self.labels[d][b[d]]
                if x:
                    continue
            if any(tuple(b[k] for k in p) < b for p in grp):
                continue
            ext = [self.sizes[d][b[d]] for d in range(self.n)]
            out.append(([int(starts[d][b[d]]) for d in range(self.n)], ext, off))
            off += (math.prod(ext) + 3) // 4 * 4
        return out, off

    def nelems(self):
        return sum(math.prod(e) for _, e, _ in self.blocks()[0])

    def values(self, seed, scale, ranges):
        """The seeded inputs at the index ranges, as the library fills them:
        a sum of twelve 32-bit uniforms from splitmix64 per element of the
        symmetry group, signed; no spin or label rule applied."""
        dev = torch.device("cuda")
        x = [torch.arange(a, b, device=dev).reshape([-1 if k == d else 1 for k in range(self.n)])
             for d, (a, b) in enumerate(ranges)]
        key = _mix_int(seed)
        v = None
        for p, c in self.group():
            lin = torch.zeros((), dtype=torch.int64, device=dev)
            for d in range(self.n):
                lin = lin * self.dims[d] + x[p[d]]
            lin = lin * 6 + _signed(key)
            s = torch.zeros_like(lin)
            for r in range(6):
                h = _mix(lin + r)
                s += (h & 0xFFFFFFFF) + ((h >> 32) & 0xFFFFFFFF)
            s -= 6 << 32
            v = s if v is None else (v + s if c > 0 else v - s)
        return v.double() * (scale * 2.3283064365386963e-10)

    def dense(self, seed, scale, first=None):
        """The whole tensor (first index in the range `first`), with zeros where a rule forbids."""
        r0 = first or (0, self.dims[0])
        out = torch.zeros([r0[1] - r0[0]] + self.dims[1:], dtype=torch.float64, device="cuda")
        lab = None
        if self.labels is not None:
            lab = [torch.tensor(np.repeat(self.labels[d], self.sizes[d]), device="cuda") for d in range(self.n)]
        for s in product(range(2), repeat=self.n):
            if sum(s[d] for d in self.bra) != sum(s[d] for d in self.ket):
                continue
            rng = [(s[d] * self.dims[d] // 2, (s[d] + 1) * self.dims[d] // 2) for d in range(self.n)]
            lo, hi = max(rng[0][0], r0[0]), min(rng[0][1], r0[1])
            step = max(1, (1 << 26) // math.prod(b - a for a, b in rng[1:]))
            for a in range(lo, hi, step):
                cut = [(a, min(hi, a + step))] + rng[1:]
                v = self.values(seed, scale, cut)
                if lab is not None:
                    x = 0
                    for d in range(self.n):
                        x = x ^ lab[d][cut[d][0]:cut[d][1]].reshape([-1 if k == d else 1 for k in range(self.n)])
                    v = torch.where(x == 0, v, 0.0)
                out[tuple(slice(p - (r0[0] if d == 0 else 0), q - (r0[0] if d == 0 else 0))
                          for d, (p, q) in enumerate(cut))] = v
        return out

    def pack(self, block):
        """The arena whose canonical blocks block(starts, extents) gives."""
        blocks, n = self.blocks()
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        for st, ext, off in blocks:
            out[off:off + math.prod(ext)] = block(st, ext).reshape(-1)
        return out

    def pack_dense(self, x):
        return self.pack(lambda st, ext: x[tuple(slice(a, a + e) for a, e in zip(st, ext))])


def _signed(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _mix_int(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _mix(z):
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * _signed(0x94D049BB133111EB)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


ANTI_01, ANTI_23 = ((1, 0, 2, 3), -1.0), ((0, 1, 3, 2), -1.0)


def _spaces(case):
    o = [int(x) for x in case["occ"].split(",")] * 2
    v = [int(x) for x in case["vir"].split(",")] * 2
    lo = lv = None
    if case.get("irreps"):
        lo, lv = [b % (len(o) // 2) for b in range(len(o))], [b % (len(v) // 2) for b in range(len(v))]

    def lab(s):
        return None if lo is None else [lo if c == "o" else lv for c in s]

    def four(s, perms):
        return Space([o if c == "o" else v for c in s], perms, (0, 1), (2, 3), lab(s))

    return dict(t=four("oovv", [ANTI_01, ANTI_23]), V=four("vvvv", [ANTI_01, ANTI_23]), W=four("ovvo", []),
                x=four("oovv", []), x01=four("oovv", [ANTI_01]),
                f=Space([v, v], [((1, 0), 1.0)], (0,), (1,), None if lv is None else [lv, lv]))


def _eps(sp):
    """Orbital energies (hartree): the same for both spins, occupied below virtual ones."""
    o, v = sp.dims[0] // 2, sp.dims[2] // 2
    eo, ev = -np.linspace(2.0, 0.4, o), np.linspace(0.1, 3.5, v)
    return np.concatenate([eo, eo]), np.concatenate([ev, ev])


# ---------------------------------------------------------------- the program

_CTX = []


def _context():
    if not _CTX:
        _CTX.append(core.Context(torch.cuda.current_device()))
    return _CTX[0]


class _Handles:
    """The library objects of one state, released with it."""

    def __init__(self):
        self.own = []

    def keep(self, x):
        self.own.append(x)
        return x

    def tensor(self, space):
        return self.keep(core.block_tensor(_context(), space.spec()))

    def __del__(self):
        for x in reversed(self.own):
            x.close()


class _Arena:
    """A block tensor's device memory for torch, with its owner kept alive."""

    def __init__(self, handles, bt):
        self.handles = handles
        self.__cuda_array_interface__ = dict(shape=(bt.nelems,), typestr="<f8", data=(bt.device_ptr(), False),
                                             version=3, strides=None)


class _State:
    def __init__(self, handles, call, outputs):
        self.handles, self.call = handles, call
        self.outputs = [torch.as_tensor(_Arena(handles, x), device="cuda") if isinstance(x, core.block_tensor) else x
                        for x in outputs]


def _contraction(h, case, sp, a, b):
    if case["op"] == "ladder":
        c = core.contraction2(2, 2, 2).contract(2, 2).contract(3, 3)
        return h.keep(core.btod_contract2(c, a, b, kc=0.5))
    if case["op"] == "ring":
        c = core.contraction2(2, 2, 2, [0, 3, 1, 2]).contract(1, 0).contract(3, 2)
        return h.keep(core.btod_contract2(c, a, b))
    return h.keep(core.btod_contract2(core.contraction2(3, 1, 1).contract(3, 0), a, b))


def _amplitudes(h, sp, seed):
    """Doubles amplitudes: antisymmetrised integrals over orbital energies."""
    t = h.tensor(sp["t"])
    t.fill_seeded(seed, T_SCALE)
    eo, ev = _eps(sp["t"])
    t.denominator(np.concatenate([eo, eo, ev, ev]), nocc=2)
    return t


def _prepare_ccd(h, case, sp, seed):
    ctx, mode, ns = _context(), MODES[case["mode"]], case["slices"]
    t = _amplitudes(h, sp, seed)
    v, w = h.tensor(sp["V"]), h.tensor(sp["W"])
    v.fill_seeded(seed + 1, V_SCALE)
    w.fill_seeded(seed + 2, V_SCALE)
    ladder = _contraction(h, dict(op="ladder"), sp, t, v)
    ring = _contraction(h, dict(op="ring"), sp, t, w)
    l, g = h.keep(ladder.make_result()), h.keep(ring.make_result())
    x, r = h.keep(t.permuted((0, 2, 1, 3))), h.tensor(sp["t"])
    eo, ev = _eps(sp["t"])
    eps = np.concatenate([eo, eo, ev, ev])
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    copy = core.btod_copy(t, (0, 2, 1, 3))
    combine = core.btod_add(l, None, 1.0)
    for p, c in (((0, 1, 2, 3), 0.5), ((1, 0, 2, 3), -0.5), ((0, 1, 3, 2), -0.5), ((1, 0, 3, 2), 0.5)):
        combine.add_op(g, p, c)

    def step():
        copy.perform(x)
        ladder.perform(l, mode=mode, nslices=ns)
        ring.perform(g, mode=mode, nslices=ns)
        combine.perform(r)
        r.denominator(eps, nocc=2)
        check(lib().ltg_dotprod_async(r.h, None, t.h, None, energy.data_ptr()))

    step()
    ctx.synchronize()
    ctx.graph_begin()
    try:
        step()
    finally:
        graph = h.keep(ctx.graph_end())
    return _State(h, graph.launch, [x, r, energy])


def prepare(case, seed):
    h, sp, op, ctx = _Handles(), _spaces(case), case["op"], _context()
    seed = 10 * seed + 1
    if op == "ccd":
        return _prepare_ccd(h, case, sp, seed)
    if op in ("ladder", "ring", "fock"):
        a = _amplitudes(h, sp, seed)
        b = h.tensor(sp[{"ladder": "V", "ring": "W", "fock": "f"}[op]])
        b.fill_seeded(seed + 1, V_SCALE)
        c = _contraction(h, case, sp, a, b)
        mode, ns = MODES[case["mode"]], case["slices"]
        if case.get("symm"):
            r = h.keep(c.make_symmetrized(False, (0, 1)))
            return _State(h, lambda: c.perform_symmetrized(r, False, (0, 1), mode=mode, nslices=ns), [r])
        r = h.keep(c.make_result())
        if case.get("add"):
            r.fill_seeded(seed + 2, T_SCALE)
        d = 1.0 if case.get("add") else None
        return _State(h, lambda: c.perform(r, d, mode=mode, nslices=ns), [r])
    if op == "copy":
        perm = tuple(int(p) for p in case["perm"].split(","))
        a = h.tensor(sp["V"])
        a.fill_seeded(seed, V_SCALE)
        b = h.keep(a.permuted(perm))
        o = core.btod_copy(a, perm)
        return _State(h, lambda: o.perform(b), [b])
    if op == "dot":
        a, b = h.tensor(sp["V"]), h.tensor(sp["V"])
        a.fill_seeded(seed, V_SCALE)
        b.fill_seeded(seed + 1, V_SCALE)
        o = core.btod_dotprod(a, None, b, tuple(int(p) for p in case["perm"].split(",")))
        out = [0.0]
        s = _State(h, lambda: out.__setitem__(0, o.calculate()), [])
        s.outputs = out
        return s
    x = h.tensor(sp["x"])
    x.fill_seeded(seed, V_SCALE)
    if op == "symm":
        o = core.btod_symmetrize(x, False, (0, 1))
        r = h.keep(o.make_result())
    else:
        o = core.btod_add(x, None, 1.0).add_op(x, (1, 0, 2, 3), -1.0).add_op(x, (0, 1, 3, 2), -0.5)
        o.add_op(x, (1, 0, 3, 2), 0.5)
        r = h.tensor(sp["x"])
    return _State(h, lambda: o.perform(r), [r])


def run(state):
    state.call()
    return list(state.outputs)


# ---------------------------------------------------------------- what a pass cannot do without

def _flops(case, sp):
    """Multiply-adds over the allowed spins and labels, each contracted pair
    of antisymmetric indices once."""
    o = [int(x) for x in case["occ"].split(",")]
    v = [int(x) for x in case["vir"].split(",")]
    if case["op"] == "fock":
        return 2.0 * sp["x01"].nelems() * sum(v)
    if case["op"] == "ladder":
        n, total = sum(v), 0
        for st, ext, _ in sp["t"].blocks()[0]:
            same = (st[2] >= n) == (st[3] >= n)
            total += math.prod(ext) * (n * (n - 1) // 2 if same else n * n)
        return 2.0 * total
    # ring: (k, c) carries the spin change and the label product of (i, a)
    irreps = bool(case.get("irreps"))
    pairs = {}
    for sk, sc in product(range(2), repeat=2):
        for (x, no), (y, nv) in product(enumerate(o), enumerate(v)):
            key = (sc - sk, x ^ y if irreps else 0)
            pairs[key] = pairs.get(key, 0) + no * nv
    start = {}
    for d in (0, 2):
        pos = np.concatenate([[0], np.cumsum(sp["x"].sizes[d])])
        half = len(sp["x"].sizes[d]) // 2
        start[d] = {int(p): (int(b >= half), b % half) for b, p in enumerate(pos[:-1])}
    total = 0
    for st, ext, _ in sp["x"].blocks()[0]:
        (si, li), (sa, la) = start[0][st[0]], start[2][st[2]]
        total += math.prod(ext) * pairs.get((si - sa, li ^ la if irreps else 0), 0)
    return 2.0 * total


def work(case):
    sp, op = _spaces(case), case["op"]
    if op == "copy":
        return dict(bytes=16.0 * sp["V"].nelems(), flops=0.0)
    if op == "dot":
        return dict(bytes=16.0 * sp["V"].nelems(), flops=2.0 * sp["V"].nelems())
    if op in ("add", "symm"):
        r = sp["x"].nelems() if op == "add" else sp["x01"].nelems()
        return dict(bytes=8.0 * (sp["x"].nelems() + r), flops=(7.0 if op == "add" else 2.0) * r)
    t = sp["t"].nelems()
    if op == "ccd":
        f = _flops(dict(case, op="ladder"), sp) + _flops(dict(case, op="ring"), sp)
        return dict(bytes=8.0 * (sp["V"].nelems() + sp["W"].nelems() + 2 * t + sp["t"].permuted([0, 2, 1, 3]).nelems()),
                    flops=f)
    b = sp[{"ladder": "V", "ring": "W", "fock": "f"}[op]].nelems()
    r = {"ladder": sp["t"], "ring": sp["x01"] if case.get("symm") else sp["x"], "fock": sp["x01"]}[op].nelems()
    return dict(bytes=8.0 * (t + b + r * (2 if case.get("add") else 1)), flops=_flops(case, sp))


# ---------------------------------------------------------------- the same in dense FP64

def _dense_t(sp, seed):
    eo, ev = (torch.tensor(e, device="cuda") for e in _eps(sp["t"]))
    t = sp["t"].dense(seed, T_SCALE)
    return t / (eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, :, None] - ev)


def _dense_ladder(sp, t, seed):
    o, v = t.shape[0], t.shape[2]
    t2 = t.reshape(o * o, v * v)
    out = torch.empty_like(t)
    step = max(1, int(4e8) // v ** 3)
    for a in range(0, v, step):
        n = min(v, a + step) - a
        slab = sp["V"].dense(seed, V_SCALE, (a, a + n))
        out[:, :, a:a + n] = (0.5 * (t2 @ slab.reshape(n * v, v * v).T)).reshape(o, o, n, v)
    return out


def _dense_ring(sp, t, seed):
    return torch.einsum("ikac,kbcj->ijab", t, sp["W"].dense(seed, V_SCALE))


def exact(case, seed):
    sp, op = _spaces(case), case["op"]
    seed = 10 * seed + 1
    if op == "copy":
        p = [int(x) for x in case["perm"].split(",")]
        inv = [p.index(d) for d in range(4)]

        def block(st, ext):
            src = [(st[inv[d]], st[inv[d]] + ext[inv[d]]) for d in range(4)]
            return sp["V"].values(seed, V_SCALE, src).permute(p)
        return [sp["V"].permuted(p).pack(block)]
    if op == "dot":
        # <V, P V'> over the canonical blocks of V, each as often as its orbit
        total, grp = 0.0, [q for q, _ in sp["V"].group()]
        for st, ext, _ in sp["V"].blocks()[0]:
            rng = [(s, s + e) for s, e in zip(st, ext)]
            orbit = {tuple(rng[k] for k in q) for q in grp}
            x = sp["V"].values(seed, V_SCALE, rng)
            y = sp["V"].values(seed + 1, V_SCALE, [rng[k] for k in (1, 0, 3, 2)]).permute(1, 0, 3, 2)
            total += len(orbit) * float(torch.dot(x.reshape(-1), y.reshape(-1)))
        return [total]
    if op in ("add", "symm"):
        x = sp["x"].dense(seed, V_SCALE)
        if op == "symm":
            return [sp["x01"].pack_dense(x - x.permute(1, 0, 2, 3))]
        y = x - x.permute(1, 0, 2, 3)
        return [sp["x"].pack_dense(y - 0.5 * x.permute(0, 1, 3, 2) + 0.5 * x.permute(1, 0, 3, 2))]
    t = _dense_t(sp, seed)
    if op == "ladder":
        r, space = _dense_ladder(sp, t, seed + 1), sp["t"]
    elif op == "ring":
        r, space = _dense_ring(sp, t, seed + 1), sp["x"]
        if case.get("symm"):
            r, space = r - r.permute(1, 0, 2, 3), sp["x01"]
    elif op == "fock":
        r, space = torch.einsum("ijad,dc->ijac", t, sp["f"].dense(seed + 1, V_SCALE)), sp["x01"]
    else:
        l, g = _dense_ladder(sp, t, seed + 1), _dense_ring(sp, t, seed + 2)
        g = g - g.permute(1, 0, 2, 3)
        g = g - g.permute(0, 1, 3, 2)
        eo, ev = (torch.tensor(e, device="cuda") for e in _eps(sp["t"]))
        r = (l + 0.5 * g) / (eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, :, None] - ev)
        perm = [0, 2, 1, 3]
        return [sp["t"].permuted(perm).pack_dense(t.permute(perm)), sp["t"].pack_dense(r),
                torch.sum(r * t).reshape(1)]
    if case.get("add"):
        r = r + space.dense(seed + 2, T_SCALE)
    return [space.pack_dense(r)]
