"""The calls that users of this library make, with sizes, for timing.

A case is a dict of plain values: `kind` names the call, the rest its sizes.
All matrices are kernel matrices on random points (1D sorted, 2D / 3D along
the Morton curve), the inputs the library is used on; sizes and tolerances
follow the library's benchmark workloads and tests.

    listed()            the cases themselves
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, trees and buffers a program holds before the call
    run(state)          one pass through the public entry points
    work(case)          bytes and flops one pass cannot do without
    exact(case, seed)   the result in 64 bits without this library
"""
import math

import numpy as np
import torch

from hmat_lib_b200.hodlr import DeviceTree, Tree, matmat_batched

KINDS = {"gaussian": 0, "matern32": 1, "exponential": 2}


def listed():
    return [
        # H x on a small tree, the inner step of an iterative method: launch latency
        dict(name="matvec_1d_n1024", kind="product", op="N", precision=0, n=1024, dim=1,
             kernel="gaussian", length=0.2, diag=1.0, height=3, tol=1e-10, k=1),
        # H x on a large tree: the stored factors are read once
        dict(name="matvec_2d_n32768", kind="product", op="N", precision=0, n=32768, dim=2,
             kernel="matern32", length=0.1, diag=1e-2, height=8, tol=1e-8, k=1),
        # the benchmark's product, FP64 and on the int8 tensor cores
        dict(name="matmat_2d_n32768_k256", kind="product", op="N", precision=0, n=32768, dim=2,
             kernel="matern32", length=0.1, diag=1e-2, height=8, tol=1e-8, k=256),
        dict(name="mixed_2d_n32768_k256", kind="product", op="N", precision=1, n=32768, dim=2,
             kernel="matern32", length=0.1, diag=1e-2, height=8, tol=1e-8, k=256),
        # H^T X and X H of an odd size: ragged leaves, a few right-hand sides
        dict(name="matmat_TL_2d_n10007_k33", kind="product", op="TL", precision=0, n=10007, dim=2,
             kernel="exponential", length=0.2, diag=1e-2, height=6, tol=1e-6, k=33),
        # many uneven trees in one call (sizes, lengths and columns drawn per tree)
        dict(name="batch_1d_96_mixed", kind="batch", precision=1, count=96, mix=2, tol=1e-8),
        # H_A H_B with recompression
        dict(name="hxh_1d_n16384", kind="hxh", n=16384, height=7, tol=1e-8),
        # construction from the dense matrix, the benchmark's tree, and its first product
        dict(name="build_2d_n32768", kind="build", n=32768, dim=2, kernel="matern32", length=0.1,
             diag=1e-2, height=8, tol=1e-8, k=32),
        # construction from 3D points alone (large ranks), and its first product
        dict(name="points_3d_n8192", kind="points", n=8192, dim=3, kernel="exponential",
             length=0.15, diag=1e-2, height=6, tol=1e-8, k=32),
        # construction of many uneven trees in one call, and their first products
        dict(name="build_batch_1d_48", kind="build_batch", count=48, mix=2, tol=1e-8,
             k=16),
        # factorisation and solve of a regularised kernel system
        dict(name="solve_2d_n16384_k64", kind="solve", n=16384, dim=2, kernel="matern32",
             length=0.1, diag=1.0, height=7, tol=1e-8, k=64),
        # the C API on host arrays: construction, H v, H X, H^T X, X H of a small odd matrix
        dict(name="host_1d_n1021_k20", kind="host", n=1021, dim=1, kernel="gaussian", length=0.2,
             diag=1.0, height=3, tol=1e-10, k=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _height(rng, n):
    """Leaves of about 64 to 192 rows."""
    return max(1, int(round(math.log2(n / rng.uniform(70.0, 170.0)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "batch", "hxh", "build", "points",
                       "build_batch", "solve", "host"])
    tol = rng.choice([1e-6, 1e-8, 1e-8, 1e-10])
    kernel = rng.choice(sorted(KINDS))
    length = round(math.exp(rng.uniform(math.log(0.05), math.log(0.5))), 4)
    diag = rng.choice([1e-2, 1.0])
    c = dict(kind=kind, kernel=kernel, length=length, diag=diag, tol=tol)
    if kind == "product":
        c.update(op=rng.choice(["N", "N", "T", "L", "TL"]), precision=rng.choice([0, 0, 1]),
                 dim=rng.choice([1, 2, 2, 3]))
        c["n"] = _log_int(rng, 600, 8000 if c["dim"] == 3 else 32768)
        c["height"] = _height(rng, c["n"])
        if c["precision"]:   # the int8 path takes leaves of whole 32-row blocks
            c["n"] = max(1, round(c["n"] / 2 ** c["height"] / 32)) * 32 * 2 ** c["height"]
        c["k"] = 1 if rng.random() < 0.2 else _log_int(rng, 2, 256)
    elif kind in ("batch", "build_batch"):
        c = dict(kind=kind, count=_log_int(rng, 4, 64 if kind == "batch" else 40),
                 mix=rng.randrange(1 << 20), tol=tol)
        if kind == "batch":
            c["precision"] = rng.choice([0, 1])
        else:
            c["k"] = _log_int(rng, 1, 32)
    elif kind == "hxh":
        c = dict(kind=kind, n=_log_int(rng, 700, 16384), tol=rng.choice([1e-6, 1e-8, 1e-10]))
        c["height"] = _height(rng, c["n"])
    elif kind in ("build", "points", "solve"):
        c["dim"] = rng.choice([1, 2, 2, 3])
        hi = {"build": 24000, "points": 16384, "solve": 14000}[kind]
        c["n"] = _log_int(rng, 700, 6000 if c["dim"] == 3 else hi)
        c["height"] = _height(rng, c["n"])
        c["k"] = _log_int(rng, 1, 64)
        if kind == "solve":
            c["diag"] = 1.0
    else:
        c["dim"] = rng.choice([1, 2])
        c["n"] = _log_int(rng, 300, 3000)
        c["height"] = _height(rng, c["n"])
        c["k"] = _log_int(rng, 1, 100)
    return c


# ---- inputs ------------------------------------------------------------------------

def _points(n, dim, rng):
    """n x dim random points: sorted in 1D, along the Morton curve otherwise."""
    p = rng.random((n, dim))
    if dim == 1:
        return np.sort(p, axis=0)
    q = (p * 65536).astype(np.int64)
    code = np.zeros(n, dtype=np.int64)
    for b in range(16):
        for a in range(dim):
            code |= ((q[:, a] >> b) & 1) << (b * dim + a)
    return p[np.argsort(code, kind="stable")]


def _columns(pts, c0, c1, kernel, length, diag):
    """Columns c0 .. c1 - 1 of the kernel matrix (n x (c1 - c0), pts on the GPU)."""
    r2 = 0.0
    for a in range(pts.shape[1]):
        r2 = r2 + (pts[:, None, a] - pts[None, c0:c1, a]).square_()
    if kernel == "gaussian":
        v = r2.mul_(-0.5 / length ** 2).exp_()
    else:
        t = r2.sqrt_().mul_((math.sqrt(3.0) if kernel == "matern32" else 1.0) / length)
        v = torch.exp(-t)
        if kernel == "matern32":
            v.mul_(t.add_(1.0))
    i = torch.arange(c0, c1, device=v.device)
    v[i, i - c0] += diag
    return v


def _dense(pts, kernel, length, diag):
    """The kernel matrix on the GPU: symmetric, so its layout is column-major too."""
    n = pts.shape[0]
    a = torch.empty(n, n, dtype=torch.float64, device="cuda")
    for c0 in range(0, n, 2048):
        c1 = min(n, c0 + 2048)
        a[c0:c1] = _columns(pts, c0, c1, kernel, length, diag).t()
    return a


def _apply(pts, kernel, length, diag, x):
    """K X with x of shape (k, n), block by block; the result as (k, n)."""
    n = pts.shape[0]
    y = torch.empty_like(x)
    for c0 in range(0, n, 2048):
        c1 = min(n, c0 + 2048)
        y[:, c0:c1] = x @ _columns(pts, c0, c1, kernel, length, diag)
    return y


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _normal(rng, *shape):
    return _cuda(rng.standard_normal(shape))


def _kernel_of(case):
    return case["kernel"], case["length"], case["diag"]


def _batch_items(case, rng):
    """The uneven batch: sorted 1D points, exponential kernels, leaf 128.  `mix`
    names the drawn sizes and columns, the seed the points and lengths."""
    sizes = np.random.default_rng(case["mix"])
    items = []
    for _ in range(case["count"]):
        n = int(sizes.choice([1024, 2048, 4096, 8192]))
        k = int(sizes.integers(16, 129))
        items.append(dict(n=n, length=float(rng.uniform(0.05, 0.5)), height=int(np.log2(n // 128)),
                          k=case.get("k") or k, pts=_points(n, 1, rng)))
    return items


_HXH = (("gaussian", 0.1, 1.0), ("matern32", 0.2, 1.0))


def _inputs(case, seed):
    """The numbers of a case (points and right-hand sides), from the seed alone."""
    rng = np.random.default_rng([seed, 20250])
    if case["kind"] in ("batch", "build_batch"):
        items = _batch_items(case, rng)
        return items, [_normal(rng, it["k"], it["n"]) for it in items]
    pts = _points(case["n"], case.get("dim", 1), rng)
    return pts, _normal(rng, case.get("k", 16), case["n"])


def _from_points(pts, kernel, length, diag, height, tol):
    d = _cuda(pts.T)   # column-major n x dim
    return DeviceTree.build_kernel(d.data_ptr(), pts.shape[0], pts.shape[1], KINDS[kernel], length,
                                   diag, height, tol)


_STREAM = []


def _stream():
    """The stream that the program does its products on."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    inp, x = _inputs(case, seed)
    st = dict(case=case, x=x)
    if kind == "product":
        st["tree"] = _from_points(inp, *_kernel_of(case), case["height"], case["tol"])
        if "L" in case["op"]:
            st["xl"] = x.t().contiguous()   # k x n column-major
            st["yl"] = torch.zeros_like(st["xl"])
        st["y"] = torch.zeros_like(x)
    elif kind == "batch":
        st["trees"] = [_from_points(it["pts"], "exponential", it["length"], 0.0, it["height"],
                                    case["tol"]) for it in inp]
        st["ks"], st["ns"] = [it["k"] for it in inp], [it["n"] for it in inp]
        st["y"] = torch.zeros(sum(k * n for k, n in zip(st["ks"], st["ns"])), dtype=torch.float64,
                              device="cuda")
        off = np.concatenate([[0], np.cumsum([k * n for k, n in zip(st["ks"], st["ns"])])])
        st["ys"] = [st["y"].data_ptr() + 8 * int(o) for o in off[:-1]]
    elif kind == "hxh":
        st["a"], st["b"] = (_from_points(inp, *m, case["height"], case["tol"]) for m in _HXH)
        st["y"] = torch.zeros_like(x)
    elif kind == "build":
        st["matrix"] = _dense(_cuda(inp), *_kernel_of(case))
        st["y"] = torch.zeros_like(x)
    elif kind == "points":
        st["pts"] = _cuda(inp.T)
        st["y"] = torch.zeros_like(x)
    elif kind == "build_batch":
        st["items"] = inp
        st["matrices"] = [_dense(_cuda(it["pts"]), "exponential", it["length"], 0.0) for it in inp]
        st["y"] = torch.zeros(sum(v.numel() for v in x), dtype=torch.float64, device="cuda")
    elif kind == "solve":
        st["tree"] = _from_points(inp, *_kernel_of(case), case["height"], case["tol"])
        st["y"] = torch.zeros_like(x)
    elif kind == "host":
        st["matrix"] = _dense(_cuda(inp), *_kernel_of(case)).cpu().numpy().T
        st["x"] = np.asfortranarray(x.cpu().numpy().T)
        st["xl"] = np.asfortranarray(st["x"].T)
    torch.cuda.synchronize()
    return st


# ---- the calls ----------------------------------------------------------------------

def _matmat(tree, st, op=0, precision=0, x="x", y="y"):
    c = st["case"]
    n = c["n"]
    k = c.get("k", 16)
    ld = k if op == 2 else n
    tree.matmat(st[x].data_ptr(), k, ld, st[y].data_ptr(), ld, op=op, precision=precision,
                stream=_stream())
    return st[y]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "product":
        p = case["precision"]
        out = {}
        if "N" in case["op"]:
            out["n"] = _matmat(st["tree"], st, 0, p)
        if "T" in case["op"]:
            out["t"] = _matmat(st["tree"], st, 1, p)
        if "L" in case["op"]:
            out["l"] = _matmat(st["tree"], st, 2, p, "xl", "yl")
        return out
    if kind == "batch":
        matmat_batched(st["trees"], [v.data_ptr() for v in st["x"]], st["ks"], st["ns"], st["ys"],
                       st["ns"], precision=case["precision"], stream=_stream())
        return st["y"]
    if kind == "hxh":
        st["out"] = st["a"].hxh(st["b"], case["tol"])
        return {"ranks": st["out"].ranks(), "y": _matmat(st["out"], st)}
    if kind in ("build", "points"):
        n = case["n"]
        if kind == "build":
            st["out"] = DeviceTree.build(st["matrix"].data_ptr(), n, n, case["height"], case["tol"],
                                         stream=_stream())
        else:
            st["out"] = DeviceTree.build_kernel(st["pts"].data_ptr(), n, case["dim"],
                                                KINDS[case["kernel"]], case["length"], case["diag"],
                                                case["height"], case["tol"], stream=_stream())
        return {"ranks": st["out"].ranks(), "y": _matmat(st["out"], st)}
    if kind == "build_batch":
        ns = [it["n"] for it in st["items"]]
        st["out"] = DeviceTree.build_batched([a.data_ptr() for a in st["matrices"]], ns, ns,
                                             [it["height"] for it in st["items"]], case["tol"],
                                             stream=_stream())
        at = st["y"].data_ptr()
        ys = []
        for n in ns:
            ys.append(at)
            at += 8 * n * case["k"]
        matmat_batched(st["out"], [v.data_ptr() for v in st["x"]], [case["k"]] * len(ns), ns, ys,
                       ns, stream=_stream())
        return {"ranks": np.concatenate([t.ranks() for t in st["out"]]), "y": st["y"]}
    if kind == "solve":
        n, k = case["n"], case["k"]
        st["factor"] = st["tree"].factorize(stream=_stream())
        st["factor"].solve(st["x"].data_ptr(), k, n, st["y"].data_ptr(), n, stream=_stream())
        return st["y"]
    if kind == "host":
        t = Tree.from_dense(st["matrix"], case["height"], case["tol"])
        return {"v": t.matvec(st["x"][:, 0]), "n": t.matmat(st["x"], "N"),
                "t": t.matmat(st["x"], "T"), "l": t.matmat(st["xl"], "L")}
    raise ValueError(kind)


# ---- work and exact results --------------------------------------------------------

def _tree_numbers(case, spec, n, pts):
    """(stored doubles, [(depth, rows + columns, rows * columns, rank)] per block)."""
    t = _from_points(pts, *spec, case["height"], case["tol"])
    ranks, storage = t.ranks(), t.info()["storage"]
    t.free()
    blocks = []
    for d in range(case["height"]):
        size = n / 2 ** (d + 1)
        first = 2 * (2 ** d - 1)
        blocks += [(d, 2 * size, size * size, int(s)) for s in ranks[first:first + 2 ** (d + 1)]]
    return storage, blocks


def _build_work(n, storage, blocks, reads):
    """Input read once, factors written once; a sketch of each block and its adjoint product."""
    return {"bytes": reads + 8.0 * storage, "flops": 4.0 * sum(mn * s for _, _, mn, s in blocks)}


def work(case):
    kind = case["kind"]
    rng = np.random.default_rng([0, 20250])
    if kind in ("batch", "build_batch"):
        w = {"bytes": 0.0, "flops": 0.0}
        for it in _batch_items(case, rng):
            n, k = it["n"], it["k"]
            sub = dict(height=it["height"], tol=case["tol"])
            storage, blocks = _tree_numbers(sub, ("exponential", it["length"], 0.0), n, it["pts"])
            if kind == "build_batch":
                b = _build_work(n, storage, blocks, 8.0 * n * n)
                w = {q: w[q] + b[q] for q in w}
            w["bytes"] += 8.0 * storage * (kind == "batch") + 16.0 * n * k
            w["flops"] += 2.0 * k * storage
        return w
    n, k = case["n"], case.get("k", 16)
    pts = _points(n, case.get("dim", 1), rng)
    if kind == "hxh":
        w = {"bytes": 0.0, "flops": 0.0}
        for spec in _HXH:
            storage, blocks = _tree_numbers(case, spec, n, pts)
            w["bytes"] += 8.0 * storage * 1.5   # the result is about as large as either factor
            w["flops"] += 2.0 * sum(s * storage / 2 ** (d + 1) for d, _, _, s in blocks)
        return w
    storage, blocks = _tree_numbers(case, _kernel_of(case), n, pts)
    product = {"bytes": 8.0 * storage + 16.0 * n * k, "flops": 2.0 * k * storage}
    if kind == "product":
        ops = len(case["op"])
        return {q: ops * v for q, v in product.items()}
    if kind == "solve":
        # leaf inverses, each level's basis solved through the deeper ones, one solve
        leaf = n / 2 ** case["height"]
        f = 2.0 * n * leaf ** 2 + 2.0 * sum(s * storage / 2 ** (d + 1) for d, _, _, s in blocks)
        return {"bytes": product["bytes"], "flops": f + product["flops"]}
    b = _build_work(n, storage, blocks, 8.0 * n * n if kind != "points" else 8.0 * n * case["dim"])
    times = 3.0 + 1.0 / k if kind == "host" else 1.0
    return {"bytes": b["bytes"] + times * 16.0 * n * k, "flops": b["flops"] + times * product["flops"]}


def exact(case, seed):
    kind = case["kind"]
    inp, x = _inputs(case, seed)
    if kind in ("batch", "build_batch"):
        y = torch.cat([_apply(_cuda(it["pts"]), "exponential", it["length"], 0.0, v).reshape(-1)
                       for it, v in zip(inp, x)])
        return y if kind == "batch" else {"ranks": None, "y": y}
    pts = _cuda(inp)
    if kind == "hxh":
        return {"ranks": None, "y": _apply(pts, *_HXH[0], _apply(pts, *_HXH[1], x))}
    if kind == "solve":
        return torch.linalg.solve(_dense(pts, *_kernel_of(case)), x.t()).t().contiguous()
    y = _apply(pts, *_kernel_of(case), x)   # the matrix is symmetric: H^T X is the same
    if kind == "product":
        return {op.lower(): y.t().contiguous() if op == "L" else y for op in case["op"]}
    if kind in ("build", "points"):
        return {"ranks": None, "y": y}
    h = y.cpu().numpy().T
    return {"v": h[:, 0].copy(), "n": np.asfortranarray(h), "t": np.asfortranarray(h), "l": h.T.copy()}
