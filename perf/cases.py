"""Performance cases: what a user of this engine has it do, through its
public entry points (``rtspmspm_b200.Engine``).

Inputs are made on the GPU with torch, with the shapes and value distributions
of ``rtspmspm_b200.gen`` (the generators there draw on the host, which takes far
longer than the products themselves).  A case names one sparsity pattern, so
that results of every seed have one size; the seed renumbers the rows and
columns of the random matrices, puts the COO entries in another order and
draws all values.

A case is a dict of plain values.  ``kind`` says what it runs:

* ``er``      C = A*B, Erdos-Renyi A (rows x inner) and B (inner x cols),
              Poisson entries per row, values U(-1, 1); B is A when ``square``
* ``stencil`` C = A*A, A the 27-point stencil on a g^3 grid
* ``rmat``    C = A*A, A an R-MAT graph (0.57, 0.19, 0.19, 0.05), values U(0, 1)
* ``batch``   independent uneven Erdos-Renyi products in one call
* ``coo``     unsorted COO with duplicates to CSR
* ``mlp``     one forward and backward pass of the row-size predictor

and, for the products, ``call`` how: ``multiply`` (C on the GPU),
``host`` (C read back with ``Result.to_host``), ``reuse`` (values of an
existing C recomputed) or ``into_host`` (C delivered into pinned buffers).
"""
import math
import zlib

import numpy as np
import torch

from rtspmspm_b200 import DeviceCsr, Engine, HostCsr
from rtspmspm_b200 import gen

DEV = "cuda"
MLP_LAYERS = ((8, 64), (64, 64), (64, 2))


# ---- cases -----------------------------------------------------------------


def listed():
    return [
        # the smallest call: a ragged rectangular product from device inputs,
        # checked as by default, with C read back to the host at once
        dict(name="tiny rect, to host", kind="er", rows=777, inner=1201, cols=345, mean_a=5.0, mean_b=4.0,
             square=False, algo="learned", bits=64, trusted=False, call="host"),
        # a small product in a loop of a program that trusts its inputs: launches and waits count
        dict(name="er 4096", kind="er", rows=4096, inner=4096, cols=4096, mean_a=8.0, mean_b=8.0, square=True,
             algo="learned", bits=32, trusted=True, call="multiply"),
        # odd sizes, 64-bit row pointers, inputs checked: an ordinary rectangular product
        dict(name="rect 50021, checked", kind="er", rows=50021, inner=30011, cols=70001, mean_a=11.0, mean_b=13.0,
             square=False, algo="learned", bits=64, trusted=False, call="multiply"),
        # about 1,024 products per row, nearly all of distinct columns
        dict(name="er 65536 x 32, plain", kind="er", rows=65536, inner=65536, cols=65536, mean_a=32.0, mean_b=32.0,
             square=True, algo="plain", bits=32, trusted=True, call="multiply"),
        # the benchmark's headline product: a PDE stencil squared
        dict(name="stencil 96, learned", kind="stencil", g=96, algo="learned", bits=32, trusted=True,
             call="multiply"),
        # the exact two-pass method on an odd grid
        dict(name="stencil 61, plain", kind="stencil", g=61, algo="plain", bits=64, trusted=False, call="multiply"),
        # new values on a known structure: a solver's set-up phase run again
        dict(name="stencil 96, new values", kind="stencil", g=96, algo="plain", bits=32, trusted=True, call="reuse"),
        # end to end from pinned host memory and back
        dict(name="stencil 64, host to host", kind="stencil", g=64, algo="learned", bits=32, trusted=True,
             call="into_host"),
        # a power-law graph squared: hub rows of millions of products beside rows of a few; the largest case
        dict(name="rmat 18", kind="rmat", scale=18, edges=16, algo="learned", bits=32, trusted=True,
             call="multiply"),
        # uneven independent products in one call, replayed from a graph
        dict(name="batch of 20", kind="batch", count=20, lo=1024, hi=65536, mean_lo=2.0, mean_hi=32.0,
             algo="learned", graph=True),
        # assembly: 2^26 unsorted entries to CSR on the GPU
        dict(name="coo 2^26", kind="coo", n=1 << 26, rows=1 << 22, cols=1 << 22),
        # training the row-size predictor: one minibatch forward and backward
        dict(name="predictor step 4096", kind="mlp", rows=4096),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["er", "er", "er", "stencil", "stencil", "rmat", "batch", "coo", "mlp"])
    algo = rng.choice(["learned", "learned", "plain"])
    bits = rng.choice([32, 64])
    trusted = rng.random() < 0.7
    if kind == "er":
        square = rng.random() < 0.5
        rows = _log_int(rng, 600, 131072)
        inner = rows if square else _log_int(rng, 600, 131072)
        cols = rows if square else _log_int(rng, 300, 262144)
        mean_a = round(rng.uniform(2.0, 32.0), 2)
        mean_b = mean_a if square else round(rng.uniform(2.0, 32.0), 2)
        call = "host" if rows < 2000 else rng.choice(["multiply", "multiply", "reuse"])
        return dict(kind=kind, rows=rows, inner=inner, cols=cols, mean_a=mean_a, mean_b=mean_b, square=square,
                    algo=algo, bits=bits, trusted=trusted, call=call)
    if kind == "stencil":
        call = rng.choice(["multiply", "multiply", "reuse", "into_host"])
        g = _log_int(rng, 8, 64 if call == "into_host" else 96)
        return dict(kind=kind, g=g, algo=algo, bits=bits, trusted=trusted, call=call)
    if kind == "rmat":
        return dict(kind=kind, scale=rng.randint(10, 17), edges=rng.randint(4, 16), algo=algo, bits=bits,
                    trusted=trusted, call=rng.choice(["multiply", "multiply", "reuse"]))
    if kind == "batch":
        lo = rng.randint(64, 2048)
        mean_lo = round(rng.uniform(2.0, 8.0), 2)
        return dict(kind=kind, count=rng.randint(3, 21), lo=lo, hi=_log_int(rng, 4 * lo, 65536), mean_lo=mean_lo,
                    mean_hi=round(rng.uniform(mean_lo, 32.0), 2), algo=algo, graph=rng.random() < 0.7)
    if kind == "coo":
        n = _log_int(rng, 1 << 12, 1 << 26)
        return dict(kind=kind, n=n, rows=_log_int(rng, max(16, n // 64), max(64, n)),
                    cols=_log_int(rng, max(16, n // 64), max(64, n)))
    return dict(kind=kind, rows=_log_int(rng, 200, 16384))


# ---- inputs ----------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _from_keys(rows, cols, key, values):
    """Sorted unique row * cols + col keys to (row_ptr int64, col int32, val)."""
    r = torch.div(key, cols, rounding_mode="floor")
    rp = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(r, minlength=rows), 0, out=rp[1:])
    return rows, cols, rp, (key - r * cols).to(torch.int32), values


def _pattern(case):
    """The generator of a case's pattern: the same for every seed and name."""
    text = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    return _generator(zlib.crc32(text.encode()))


def _renumber(n, g):
    return torch.randperm(n, device=DEV, generator=g)


def _erdos_renyi(rows, cols, mean, pattern, row_of, col_of, g):
    """Poisson(mean) entries a row drawn from `pattern`, then rows and columns
    renumbered by row_of / col_of and values drawn from `g`."""
    counts = torch.poisson(torch.full((rows,), float(mean), device=DEV), generator=pattern).to(torch.int64)
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), counts)
    c = torch.randint(0, cols, (r.numel(),), device=DEV, generator=pattern)
    key = torch.unique(row_of[r] * cols + col_of[c])
    return _from_keys(rows, cols, key, torch.rand(key.numel(), device=DEV, generator=g) * 2 - 1)


def _er_pair(rows, inner, cols, mean_a, mean_b, square, pattern, g):
    row_of = _renumber(rows, g)
    if square:
        a = _erdos_renyi(rows, rows, mean_a, pattern, row_of, row_of, g)
        return a, a
    mid = _renumber(inner, g)
    a = _erdos_renyi(rows, inner, mean_a, pattern, row_of, mid, g)
    return a, _erdos_renyi(inner, cols, mean_b, pattern, mid, _renumber(cols, g), g)


def _stencil(n, g):
    idx = torch.arange(n * n * n, device=DEV)
    x, y, z = idx % n, (idx // n) % n, idx // (n * n)
    d = torch.arange(27, device=DEV)
    dx, dy, dz = d % 3 - 1, (d // 3) % 3 - 1, d // 9 - 1
    ok = torch.ones((idx.numel(), 27), dtype=torch.bool, device=DEV)
    for v, dv in ((x, dx), (y, dy), (z, dz)):
        t = v[:, None] + dv
        ok &= (t >= 0) & (t < n)
    col = (idx[:, None] + dx + n * dy + n * n * dz)[ok]
    rp = torch.zeros(idx.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(ok.sum(1), 0, out=rp[1:])
    # off-diagonal N(0, 1); the diagonal dominates its row
    v = torch.zeros(ok.shape, device=DEV)
    v[ok] = torch.randn(col.numel(), device=DEV, generator=g)
    v[:, 13] = 0
    v[:, 13] = 26 + v.abs().sum(1)
    return idx.numel(), idx.numel(), rp, col.to(torch.int32), v[ok]


def _rmat(scale, edges, pattern, g):
    n, ne = 1 << scale, edges << scale
    r = torch.zeros(ne, dtype=torch.int64, device=DEV)
    c = torch.zeros(ne, dtype=torch.int64, device=DEV)
    for lvl in range(scale):
        u = torch.rand(ne, device=DEV, generator=pattern)
        bit = 1 << (scale - 1 - lvl)
        r += (u >= 0.76) * bit
        c += (((u >= 0.57) & (u < 0.76)) | (u >= 0.95)) * bit
    key = torch.unique(r * n + c)
    return _from_keys(n, n, key, torch.rand(key.numel(), device=DEV, generator=g))


def _matrices(case, seed):
    """(A, B) as (rows, cols, row_ptr, col, val); B is A for a square."""
    g = _generator(seed)
    if case["kind"] == "stencil":
        a = _stencil(case["g"], g)
        return a, a
    if case["kind"] == "rmat":
        a = _rmat(case["scale"], case["edges"], _pattern(case), g)
        return a, a
    return _er_pair(case["rows"], case["inner"], case["cols"], case["mean_a"], case["mean_b"], case["square"],
                    _pattern(case), g)


def _batch_shapes(case):
    """The products' shapes, log-uniform in size."""
    rng = np.random.default_rng(case["count"] * 7919 + case["lo"])
    out = []
    for _ in range(case["count"]):
        rows, inner, cols = (gen.log_uniform_int(rng, case["lo"], case["hi"]) for _ in range(3))
        mean_a, mean_b = (float(rng.uniform(case["mean_lo"], case["mean_hi"])) for _ in range(2))
        out.append((rows, inner, cols, mean_a, mean_b))
    return out


def _batch(case, seed):
    g, pattern = _generator(seed), _pattern(case)
    return [_er_pair(*shape, False, pattern, g) for shape in _batch_shapes(case)]


def _coo(case, seed):
    g, pattern = _generator(seed), _pattern(case)
    r = torch.randint(0, case["rows"], (case["n"],), device=DEV, dtype=torch.int32, generator=pattern)
    c = torch.randint(0, case["cols"], (case["n"],), device=DEV, dtype=torch.int32, generator=pattern)
    order = _renumber(case["n"], g)
    return r[order], c[order], torch.rand(case["n"], device=DEV, generator=g)


def _mlp(case, seed):
    """(parameters, features, targets): weights as initialised for training
    (representable in BF16, the width the predictor keeps them in), features
    and targets of the sizes that rows of real products have."""
    g = torch.Generator().manual_seed(int(seed))
    parts = []
    for i, o in MLP_LAYERS:
        lim = math.sqrt(6.0 / i)
        parts += [(torch.rand(i * o, generator=g) * 2 - 1) * lim, torch.rand(o, generator=g) * 0.2 - 0.1]
    params = torch.cat(parts).to(torch.bfloat16).float()
    feats = torch.rand(case["rows"], 8, generator=g)
    nnz = 15 * torch.rand(case["rows"], generator=g)
    targets = torch.stack([nnz, torch.clamp(torch.ceil(nnz + 1.3), 5, 13)], 1)
    return params, feats.to(DEV), targets.to(DEV)


def _device(m, bits):
    rows, cols, rp, col, val = m
    return DeviceCsr(rows, cols, rp if bits == 64 else rp.to(torch.int32), col, val)


class _Engine(Engine):
    """The program's engine, closed with the last of what it made."""

    def __del__(self):
        self.close()


def prepare(case, seed):
    eng = _Engine(0)
    kind = case["kind"]
    s = {"case": case, "eng": eng}
    if kind == "coo":
        s["coo"] = _coo(case, seed)
    elif kind == "mlp":
        params, s["feats"], s["targets"] = _mlp(case, seed)
        eng.mlp_set_params(params.numpy())
    elif kind == "batch":
        pairs = _batch(case, seed)
        s["As"] = [_device(a, 32) for a, _ in pairs]
        s["Bs"] = [_device(b, 32) for _, b in pairs]
    else:
        a, b = _matrices(case, seed)
        if case["call"] == "into_host":
            host = gen.Csr(a[0], a[1], a[2].cpu().numpy(), a[3].cpu().numpy(), a[4].cpu().numpy())
            s["A"] = s["B"] = HostCsr(host, index_bits=case["bits"], pinned=True)
            cap = max(1, 5 * case["g"] - 6) ** 3
            s["rp"] = torch.empty(host.rows + 1, dtype=torch.int64, pin_memory=True)
            s["col"] = torch.empty(cap, dtype=torch.int32, pin_memory=True)
            s["val"] = torch.empty(cap, dtype=torch.float32, pin_memory=True)
        else:
            s["A"] = _device(a, case["bits"])
            s["B"] = s["A"] if b is a else _device(b, case["bits"])
        if case["call"] == "reuse":
            # the structure comes from an earlier product of other values
            old = DeviceCsr(s["A"].rows, s["A"].cols, s["A"].row_ptr, s["A"].col_idx, torch.ones_like(s["A"].val))
            torch.cuda.synchronize()
            s["C"], _ = eng.multiply(old, s["B"], algo=case["algo"], skip_validation=True)
    torch.cuda.synchronize()
    return s


# ---- the calls -------------------------------------------------------------


class _Array:
    """Device memory of a result, for torch.as_tensor (no copy)."""

    def __init__(self, keep, ptr, n, kind):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr or 0, False), "version": 3}


def _view(C):
    s = C.s
    if s.nnz == 0:
        col, val = torch.empty(0, dtype=torch.int32, device=DEV), torch.empty(0, device=DEV)
    else:
        col = torch.as_tensor(_Array(C, s.col_idx, s.nnz, "<i4"), device=DEV)
        val = torch.as_tensor(_Array(C, s.val, s.nnz, "<f4"), device=DEV)
    rp = torch.as_tensor(_Array(C, s.row_ptr, s.rows + 1, "<i%d" % (s.index_bits // 8)), device=DEV)
    return {"row_ptr": rp, "col_idx": col, "val": val}


def run(s):
    case, eng = s["case"], s["eng"]
    kind = case["kind"]
    if kind == "coo":
        return _view(eng.coo_to_csr(case["rows"], case["cols"], *s["coo"]))
    if kind == "mlp":
        loss, grads = eng.mlp_grad(s["feats"], s["targets"])
        return {"loss": np.array(loss, np.float32), "grads": grads}
    if kind == "batch":
        out, _ = eng.multiply_batched(s["As"], s["Bs"], use_graph=case["graph"], skip_validation=True,
                                      algo=case["algo"])
        return [_view(C) for C in out]
    opts = dict(algo=case["algo"], skip_validation=case["trusted"])
    if case["call"] == "into_host":
        nnz, _ = eng.multiply_into_host(s["A"], s["B"], s["rp"], s["col"], s["val"], blocks=8, **opts)
        return {"row_ptr": s["rp"], "col_idx": s["col"][:nnz], "val": s["val"][:nnz]}
    if case["call"] == "reuse":
        eng.multiply_reuse(s["A"], s["B"], s["C"], skip_validation=case["trusted"])
        return _view(s["C"])
    C, _ = eng.multiply(s["A"], s["B"], **opts)
    if case["call"] == "host":
        h = C.to_host()
        return {"row_ptr": h.row_ptr, "col_idx": h.col_idx, "val": h.val}
    return _view(C)


# ---- what a pass cannot do without -----------------------------------------


def _er_sizes(rows, inner, cols, mean_a, mean_b):
    """(nnz A, nnz B, products, nnz C) of an Erdos-Renyi product, on average."""
    na = rows * inner * -math.expm1(-mean_a / inner)
    nb = inner * cols * -math.expm1(-mean_b / cols)
    products = na * nb / inner
    return na, nb, products, rows * cols * -math.expm1(-products / rows / cols)


def _csr_bytes(rows, nnz):
    return 8 * nnz + 4 * (rows + 1)


def work(case):
    """Bytes: each input read once and C written once (CSR, 32-bit row
    pointers).  Flops: a multiply and an add for each product."""
    kind = case["kind"]
    if kind == "coo":
        out = case["rows"] * case["cols"] * -math.expm1(-case["n"] / case["rows"] / case["cols"])
        return {"bytes": 12 * case["n"] + _csr_bytes(case["rows"], out), "flops": case["n"] - out}
    if kind == "mlp":
        params = sum(i * o + o for i, o in MLP_LAYERS)
        return {"bytes": 40 * case["rows"] + 6 * params, "flops": 6 * case["rows"] * params}
    if kind == "batch":
        shapes, b, f = _batch_shapes(case), 0.0, 0.0
        for rows, inner, cols, ma, mb in shapes:
            na, nb, products, nc = _er_sizes(rows, inner, cols, ma, mb)
            b += _csr_bytes(rows, na) + _csr_bytes(inner, nb) + _csr_bytes(rows, nc)
            f += 2 * products
        return {"bytes": b, "flops": f}
    same = True
    if kind == "stencil":
        rows = inner = case["g"] ** 3
        na, products, nc = ((3 * case["g"] - 2) ** 3, (9 * case["g"] - 10) ** 3, (5 * case["g"] - 6) ** 3)
        nb = na
    elif kind == "rmat":
        # fits to the merged graphs of scales 10 to 18 and 4 to 16 edges a
        # vertex, within a tenth of their counted sizes
        rows = inner = 1 << case["scale"]
        e = case["edges"] / 16
        na = nb = (case["edges"] << case["scale"]) * (1 - 0.129 * e ** 0.63 * 0.83 ** (case["scale"] - 14))
        products = 2.93e9 * 2.78 ** (case["scale"] - 18) * e ** 1.72
        nc = 1.275e9 * 2.88 ** (case["scale"] - 18) * e ** 1.33
    else:
        rows, inner, same = case["rows"], case["inner"], case["square"]
        na, nb, products, nc = _er_sizes(rows, inner, case["cols"], case["mean_a"], case["mean_b"])
    b = _csr_bytes(rows, na) + (0 if same else _csr_bytes(inner, nb)) + _csr_bytes(rows, nc)
    return {"bytes": b, "flops": 2 * products}


# ---- the same in 64 bits ---------------------------------------------------

_CHUNK = 1 << 26  # products expanded at a time


def _product64(a, b, row_type):
    """C = A*B with every product and sum in 64 bits, or None when it is too
    large to expand quickly."""
    rows, _, arp, acol, aval = a
    _, cols, brp, bcol, bval = b
    blen = brp[1:] - brp[:-1]
    each = blen[acol.long()]  # products of each entry of A
    ends = torch.zeros(each.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(each, 0, out=ends[1:])
    row_ends = ends[arp]
    total = int(row_ends[-1])
    if total > 6 * 10 ** 9:
        return None
    bounds, at, re = [0], 0, row_ends.cpu().numpy()
    while at < rows:
        nxt = int(np.searchsorted(re, re[at] + _CHUNK, side="right")) - 1
        at = min(rows, max(at + 1, nxt))
        bounds.append(at)
    row_of = torch.repeat_interleave(torch.arange(rows, device=DEV), arp[1:] - arp[:-1])
    counts = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    col_out, val_out = [], []
    for r0, r1 in zip(bounds, bounds[1:]):
        p0, p1 = int(arp[r0]), int(arp[r1])
        n = each[p0:p1]
        if p1 == p0 or int(n.sum()) == 0:
            continue
        src = torch.repeat_interleave(torch.arange(p0, p1, device=DEV), n)
        q = brp[acol[src].long()] + (torch.arange(src.numel(), device=DEV) + ends[p0] - ends[src])
        key, order = torch.sort((row_of[src] - r0) * cols + bcol[q].long())
        v = (aval[src].double() * bval[q].double())[order]
        head = torch.ones(key.numel(), dtype=torch.bool, device=DEV)
        head[1:] = key[1:] != key[:-1]
        seg = torch.cumsum(head, 0) - 1
        key = key[head]
        val_out.append(torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, seg, v))
        r = torch.div(key, cols, rounding_mode="floor")
        counts[r0 + 1:r1 + 1] += torch.bincount(r, minlength=r1 - r0)
        col_out.append((key - r * cols).to(torch.int32))
    rp = torch.cumsum(counts, 0).to(row_type)
    if not col_out:
        return {"row_ptr": rp, "col_idx": torch.empty(0, dtype=torch.int32), "val": torch.empty(0).double()}
    return {"row_ptr": rp, "col_idx": torch.cat(col_out), "val": torch.cat(val_out)}


def _coo64(case, seed):
    r, c, v = _coo(case, seed)
    key, order = torch.sort(r.long() * case["cols"] + c.long())
    head = torch.ones(key.numel(), dtype=torch.bool, device=DEV)
    head[1:] = key[1:] != key[:-1]
    seg = torch.cumsum(head, 0) - 1
    key = key[head]
    val = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, seg, v[order].double())
    rows, cols, rp, col, val = _from_keys(case["rows"], case["cols"], key, val)
    return {"row_ptr": rp, "col_idx": col, "val": val}


def _mlp64(case, seed):
    """Loss 0.5 * mean over rows of (e0^2 + e1^2 / 4) and its gradient."""
    params, feats, targets = _mlp(case, seed)
    p = params.double().to(DEV).requires_grad_()
    x, at = feats.double(), 0
    for n, (i, o) in enumerate(MLP_LAYERS):
        w, bias = p[at:at + i * o].view(i, o), p[at + i * o:at + i * o + o]
        at += i * o + o
        x = x @ w + bias
        x = torch.relu(x) if n < 2 else x
    e = x - targets.double()
    loss = 0.5 * (e[:, 0].square() + 0.25 * e[:, 1].square()).mean()
    loss.backward()
    return {"loss": loss.detach(), "grads": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "coo":
        return _coo64(case, seed)
    if kind == "mlp":
        return _mlp64(case, seed)
    if kind == "batch":
        out = [_product64(a, b, torch.int64) for a, b in _batch(case, seed)]
        return None if any(x is None for x in out) else out
    a, b = _matrices(case, seed)
    wide = case["call"] in ("host", "into_host")
    return _product64(a, b, torch.int64 if wide else torch.int32)
