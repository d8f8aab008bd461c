"""Performance cases of the matrix product over compressed containers.

Every case goes through the library's public binding (iarray_b200.py): the operands are
compressed containers in GPU memory (or frames in host memory where the call takes those), made
once by prepare(); run() is one call sequence as a program makes it, and its result is read
back whole, as dense device data (decode_to_device) or as the bytes of a frame.

Case fields: kind, dtype, sizes (m, k, n), the partitions (chunk and block extents along m, k
and n: cm ck cn, bm bk bn), form ("native" / "split"), encoder of the result ("liblz4", the
library's default, or "parallel"), data (the values' distribution).  The operands are always
written by the liblz4-identical encoder, as files written by the reference are.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "iron-array_b200"))

import ctypes  # noqa: E402

import iarray_b200 as ia  # noqa: E402

TORCH = {"f64": torch.float64, "f32": torch.float32}
NUMPY = {"f64": np.float64, "f32": np.float32}
FORMS = {"native": ia.FORM_NATIVE, "split": ia.FORM_SPLIT}
ENCODERS = {"liblz4": ia.ENCODER_LIBLZ4, "parallel": ia.ENCODER_PARALLEL}

#: Most multiply-add work of a drawn product (the 8192^3 case does 1.1e12 flop) and most items of
#: a drawn operand (the 20000^2 matrix has 4e8).
MOST_FLOPS = {"native": 4e11, "split": 1.09e12}
MOST_ITEMS = 4e8


def listed():
    return [
        # the smallest call: a few chunks with ragged edges; launches, synchronisations and the
        # latency of single streams count
        dict(name="gemm_f64_300", kind="opt_gemm", dtype="f64", m=300, k=257, n=200, cm=128, ck=128, cn=128,
             bm=32, bk=32, bn=32, form="native", encoder="liblz4", data="scaled"),
        # the plain matrix product of the benchmark's first configuration, all defaults
        dict(name="matmul_f64_1000", kind="matmul", dtype="f64", m=1000, k=1000, n=1000, cm=500, ck=500, cn=500,
             bm=100, bk=100, bn=100, form="native", encoder="liblz4", data="uniform", ta=False, tb=False),
        # the reference's own perf tool sizes (tools/perf_matmul.c), ragged, all defaults
        dict(name="gemm_f64_4056", kind="opt_gemm", dtype="f64", m=4056, k=3230, n=3712, cm=1014, ck=1000, cn=928,
             bm=170, bk=125, bn=116, form="native", encoder="liblz4", data="scaled"),
        # the benchmark's headline: split precision, both operands about 0.5 GB compressed
        dict(name="gemm_f64_split_8192", kind="opt_gemm", dtype="f64", m=8192, k=8192, n=8192, cm=2048, ck=2048,
             cn=2048, bm=256, bk=256, bn=256, form="split", encoder="parallel", data="scaled"),
        # single precision through the panel product, a transposed view as the left operand,
        # blocks whose rows are no multiple of 4 items
        dict(name="matmul_f32_t_5000", kind="matmul", dtype="f32", m=5000, k=3500, n=6000, cm=1250, ck=875, cn=1500,
             bm=125, bk=175, bn=150, form="native", encoder="liblz4", data="normal", ta=True, tb=False),
        # the benchmark's single-precision configuration in the split form (six BF16 products)
        dict(name="gemm_f32_split_16384", kind="opt_gemm", dtype="f32", m=16384, k=4096, n=16384, cm=4096, ck=4096,
             cn=4096, bm=512, bk=512, bn=512, form="split", encoder="parallel", data="normal"),
        # the benchmark's matrix-vector configuration: a smooth 1.6 GB matrix
        dict(name="gemv_f32_20000", kind="gemv", dtype="f32", m=20000, k=20000, cm=4000, ck=4000, bm=500, bk=500,
             form="native", encoder="liblz4", data="smooth"),
        # the reference's matrix-vector perf tool sizes (tools/perf_matmul_vec.c)
        dict(name="gemv_f64_6000", kind="gemv", dtype="f64", m=4000, k=6000, cm=1000, ck=1500, bm=100, bk=150,
             form="native", encoder="liblz4", data="uniform"),
        # a batch of ragged products replayed as one graph (the first problems' range of the
        # benchmark's batch: extents in [64, 2048])
        dict(name="batch_f64_40", kind="batch", count=40, lo=64, hi=2048, shapes=5, cm=512, ck=512, cn=512, bm=128,
             bk=128, bn=128, dtype="f64", form="split", encoder="parallel", data="uniform"),
        # a product as an operand of an element-wise expression: max(alpha ab + bias, 0)
        dict(name="expr_f64_1500", kind="expr", dtype="f64", m=1500, k=1200, n=1800, cm=500, ck=400, cn=600, bm=100,
             bk=100, bn=120, form="native", encoder="liblz4", data="uniform"),
        # writing an array: dense device data to a frame in host memory
        dict(name="store_f32_4000", kind="store", dtype="f32", m=4000, n=3000, cm=1000, cn=1000, bm=100, bn=200,
             form="native", encoder="liblz4", data="smooth"),
        # frames in host memory to a frame in host memory, pipelined over row bands
        dict(name="cframes_f64_split_4096", kind="cframes", dtype="f64", m=4096, k=4096, n=4096, cm=1024, ck=1024,
             cn=1024, bm=256, bk=256, bn=256, form="split", encoder="liblz4", data="scaled"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _part(rng, n):
    """A chunk extent and a block extent for an axis of n items: half the time multiples of 4."""
    chunk = max(1, min(n, _log(rng, max(1, min(n, max(48, n // 5))), min(n, 4096))))
    block = max(1, min(chunk, _log(rng, max(1, min(chunk, max(24, chunk // 12))), min(chunk, 512))))
    if rng.random() < 0.5 and chunk >= 32:
        chunk -= chunk % 16
        block = max(16, block - block % 16) if chunk >= 16 else block
    return chunk, min(block, chunk)


def draw(rng):
    kind = rng.choice(["opt_gemm", "opt_gemm", "matmul", "gemv", "batch", "expr", "store", "cframes"])
    dtype = rng.choice(["f64", "f32"]) if kind not in ("batch", "expr") else "f64"
    form = rng.choice(["native", "split"])
    c = dict(kind=kind, dtype=dtype, form=form, encoder=rng.choice(["liblz4", "parallel"]),
             data=rng.choice(["uniform", "scaled", "smooth", "normal", "ramp", "sparse"]))
    if kind == "gemv":
        while True:
            m, k = _log(rng, 100, 20000), _log(rng, 100, 20000)
            if m * k <= MOST_ITEMS:
                break
        (cm, bm), (ck, bk) = _part(rng, m), _part(rng, k)
        return dict(c, m=m, k=k, cm=cm, ck=ck, bm=bm, bk=bk, form="native")
    if kind == "store":
        m, n = _log(rng, 50, 5000), _log(rng, 50, 5000)
        (cm, bm), (cn, bn) = _part(rng, m), _part(rng, n)
        return dict(c, m=m, n=n, cm=cm, cn=cn, bm=bm, bn=bn, form="native", encoder="liblz4")
    if kind == "batch":
        b = rng.choice([32, 50, 64, 100, 128])
        ch = b * rng.randint(2, 4)
        return dict(c, count=rng.randint(4, 40), lo=64, hi=_log(rng, 300, 2048), shapes=rng.randrange(1000), cm=ch,
                    ck=ch, cn=ch, bm=b, bk=b, bn=b, data=rng.choice(["uniform", "scaled"]))
    lo, hi = (100, 12000) if kind in ("opt_gemm", "matmul") else (100, 4096)
    while True:
        m, k, n = (_log(rng, lo, hi) for _ in range(3))
        if 2.0 * m * k * n <= MOST_FLOPS[form]:
            break
    (cm, bm), (ck, bk), (cn, bn) = _part(rng, m), _part(rng, k), _part(rng, n)
    c = dict(c, m=m, k=k, n=n, cm=cm, ck=ck, cn=cn, bm=bm, bk=bk, bn=bn)
    if kind == "matmul":
        c.update(ta=rng.random() < 0.3, tb=rng.random() < 0.3)
    if kind == "cframes":
        # the result's bytes are compared: whole numbers, which every form multiplies exactly, and
        # the encoder whose bytes are those of the reference's codec
        c.update(data="whole", encoder="liblz4")
    return c


# ------------------------------------------------------------------------------------ inputs
def _values(case, seed, salt, rows, cols, block=(64, 64)):
    """rows x cols values on the GPU in the case's dtype, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt * 7919) & 0x7FFFFFFF)
    r = random.Random(int(seed) * 31 + salt)
    dt = TORCH[case["dtype"]]
    data = case["data"]
    if data in ("uniform", "scaled", "sparse"):
        x = torch.rand((rows, cols), generator=g, device="cuda", dtype=dt).mul_(2).sub_(1)
        if data == "scaled":
            x *= torch.exp2(torch.randint(-8, 9, (rows, cols), generator=g, device="cuda", dtype=torch.int8).to(dt))
        if data == "sparse":                       # nine of ten blocks are zero
            bi, bj = -(-rows // block[0]), -(-cols // block[1])
            keep = torch.rand((bi, bj), generator=g, device="cuda") < 0.1
            keep = keep.repeat_interleave(block[0], 0)[:rows].repeat_interleave(block[1], 1)[:, :cols]
            x *= keep
        return x
    if data == "whole":
        return torch.randint(-64, 65, (rows, cols), generator=g, device="cuda", dtype=torch.int8).to(dt)
    i = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None]
    j = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :]
    if data == "smooth":
        return (torch.sin(0.001 * i + r.uniform(0, 6)) + torch.cos(0.002 * j + r.uniform(0, 6))).to(dt)
    if data == "ramp":
        return (r.uniform(-1, 1) + (i * cols + j) * (r.uniform(1, 2) / (rows * cols))).to(dt)
    x = torch.randn((rows, cols), generator=g, device="cuda", dtype=dt)
    x += (0.1 * torch.sin(0.003 * (i + j) + r.uniform(0, 6))).to(dt)
    return x


def _container(ctx, x, chunk, block):
    """A container of the device array x (one or two dimensions)."""
    d, s, p = ia.dtshape(x.shape, NUMPY["f64" if x.dtype == torch.float64 else "f32"]), ia.storage(chunk, block), ctypes.c_void_p()
    ia.check(ia.lib().iarray_b200_encode_from_device(ctx.ptr, ctypes.byref(d), x.data_ptr(), x.shape[-1],
                                                     ctypes.byref(s), ctypes.byref(p)), "encode_from_device")
    return ia.Container(ctx, p)


def _batch_shapes(case):
    r = random.Random(case["shapes"])
    return [tuple(r.randint(case["lo"], case["hi"]) for _ in range(3)) for _ in range(case["count"])]


def _operands(case, seed):
    """The dense operands on the GPU, in the order the calls take them."""
    kind = case["kind"]
    if kind == "batch":
        return [(_values(case, seed, 2 * i, m, k), _values(case, seed, 2 * i + 1, k, n))
                for i, (m, k, n) in enumerate(_batch_shapes(case))]
    if kind == "store":
        return [_values(case, seed, 0, case["m"], case["n"], (case["bm"], case["bn"]))]
    m, k = case["m"], case["k"]
    a = _values(case, seed, 0, *((k, m) if case.get("ta") else (m, k)), (case["bm"], case["bk"]))
    if kind == "gemv":
        return [a, _values(dict(case, data="uniform"), seed, 1, 1, k).reshape(-1)]
    n = case["n"]
    # only the left operand is block-sparse
    cb = dict(case, data="uniform") if case["data"] == "sparse" else case
    b = _values(cb, seed, 1, *((n, k) if case.get("tb") else (k, n)), (case["bk"], case["bn"]))
    if kind == "expr":
        return [a, b, _values(dict(case, data="uniform"), seed, 2, m, n)]
    return [a, b]


def _pinned(n):
    return torch.zeros(n, dtype=torch.uint8).pin_memory()


def prepare(case, seed):
    kind = case["kind"]
    ctx = ia.Context()                     # defaults: native form, liblz4-identical encoder
    ops = _operands(case, seed)
    torch.cuda.synchronize()               # the library's stream reads them
    s = dict(case, ctx=ctx)
    dt = TORCH[case["dtype"]]
    if kind == "store":
        m, n = case["m"], case["n"]
        s.update(x=ops[0], frame=_pinned(m * n * ops[0].element_size() * 2 + (1 << 22)).numpy())
    elif kind == "batch":
        pa, pb = ((case["cm"], case["ck"]), (case["bm"], case["bk"])), ((case["ck"], case["cn"]), (case["bk"], case["bn"]))
        As = [_container(ctx, a, *pa) for a, _ in ops]
        Bs = [_container(ctx, b, *pb) for _, b in ops]
        sizes = _batch_shapes(case)
        ctx.set_form(FORMS[case["form"]])
        ctx.set_encoder(ENCODERS[case["encoder"]])
        s["batch"] = ia.Batch(ctx, As, Bs, [(case["cm"], case["cn"])] * len(As), [(case["bm"], case["bn"])] * len(As))
        flat = torch.empty(sum(m * n for m, _, n in sizes), device="cuda", dtype=dt)
        s["out"], at = [], 0
        for m, _, n in sizes:
            s["out"].append(flat[at:at + m * n].view(m, n))
            at += m * n
        s["flat"] = flat
    else:
        ca, ba = (case["cm"], case["ck"]), (case["bm"], case["bk"])
        if case.get("ta"):
            ca, ba = ca[::-1], ba[::-1]
        s["a"] = _container(ctx, ops[0], ca, ba)
        if kind == "gemv":
            s["b"] = _container(ctx, ops[1], (case["ck"],), (case["bk"],))
            s["out"] = torch.empty(case["m"], device="cuda", dtype=dt)
        else:
            cb, bb = (case["ck"], case["cn"]), (case["bk"], case["bn"])
            if case.get("tb"):
                cb, bb = cb[::-1], bb[::-1]
            s["b"] = _container(ctx, ops[1], cb, bb)
            if case.get("ta"):
                s["a_stored"], s["a"] = s["a"], s["a"].transpose()
            if case.get("tb"):
                s["b_stored"], s["b"] = s["b"], s["b"].transpose()
            if kind != "cframes":
                s["out"] = torch.empty((case["m"], case["n"]), device="cuda", dtype=dt)
        if kind == "expr":
            cc, bc = (case["cm"], case["cn"]), (case["bm"], case["bn"])
            s["bias"] = _container(ctx, ops[2], cc, bc)
            e = ia.Expression(ctx, NUMPY[case["dtype"]])
            e.bind_matmul("ab", s["a"], s["b"])
            e.bind("bias", s["bias"])
            e.bind_scalar("alpha", 1.5)
            e.bind_out((case["m"], case["n"]), NUMPY[case["dtype"]], cc, bc)
            e.compile("max(alpha * ab + bias, 0)")
            s["expr"] = e
        if kind == "cframes":
            for x in ("a", "b"):
                f = _pinned(s[x].cframe_len()).numpy()
                s[x].to_cframe_into(f)
                s.pop(x).free()
                s["f" + x] = f
            isz = 8 if case["dtype"] == "f64" else 4
            ext = [-(-case[x] // case["c" + x]) * (-(-case["c" + x] // case["b" + x]) * case["b" + x]) for x in "mn"]
            chunks = -(-case["m"] // case["cm"]) * -(-case["n"] // case["cn"])
            s["frame"] = _pinned(ext[0] * ext[1] * isz + 64 * chunks + (1 << 16)).numpy()
        ctx.set_form(FORMS[case["form"]])
        ctx.set_encoder(ENCODERS[case["encoder"]])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "store":
        c = _container(ctx, s["x"], (s["cm"], s["cn"]), (s["bm"], s["bn"]))
        return {"length": c.to_cframe_into(s["frame"]), "frame": s["frame"]}
    if kind == "cframes":
        out, n = ia.opt_gemm_cframes(ctx, s["fa"], s["fb"], (s["cm"], s["cn"]), (s["bm"], s["bn"]), out=s["frame"])
        return {"length": n, "frame": out}
    if kind == "batch":
        for c, o in zip(s["batch"].run(), s["out"]):
            c.decode_to_device(o.data_ptr(), o.shape[1])
        return s["flat"]
    if kind == "gemv":
        c = ia.opt_gemv(ctx, s["a"], s["b"], (s["cm"],), (s["bm"],))
    elif kind == "expr":
        c = s["expr"].eval()
    else:
        product = ia.opt_gemm if kind == "opt_gemm" else ia.matmul
        c = product(ctx, s["a"], s["b"], (s["cm"], s["cn"]), (s["bm"], s["bn"]))
    c.decode_to_device(s["out"].data_ptr(), s["out"].shape[-1])
    return s["out"]


def _items(case):
    """Items read and written by one pass, and its multiply-adds."""
    kind = case["kind"]
    if kind == "batch":
        sizes = _batch_shapes(case)
        return sum(m * k + k * n + m * n for m, k, n in sizes), sum(m * k * n for m, k, n in sizes)
    if kind == "store":
        return 2 * case["m"] * case["n"], 0
    m, k, n = case["m"], case["k"], case.get("n", 1)
    return m * k + k * n + m * n * (2 if kind == "expr" else 1), m * k * n


def work(case):
    """Operands read once and the result written once at their dense sizes (a container's
    compressed size is 0.92 to 0.96 of its padded dense size for uniform, scaled and normal
    values and about half of it for smooth ones)."""
    items, madds = _items(case)
    return {"bytes": items * (8 if case["dtype"] == "f64" else 4), "flops": 2.0 * madds}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("store", "cframes"):       # bytes of a frame
        return None
    ops = _operands(case, seed)
    if kind == "batch":
        return torch.cat([(a.double() @ b.double()).reshape(-1) for a, b in ops])
    a, b = ops[0].double(), ops[1].double()
    if case.get("ta"):
        a = a.t()
    if case.get("tb"):
        b = b.t()
    y = a @ b
    if kind == "expr":
        y = torch.clamp_min(1.5 * y + ops[2].double(), 0)
    return y
