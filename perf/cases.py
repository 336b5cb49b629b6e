"""Workloads that stand for what programs do with this library, each run
through its public entry points (the C ABI, bound by tapp_b200): single
products from a handful of multiplications to trillions, a batched product and
a served mix. A case is a dict of plain values:

  kind "product": D[d] = alpha * sum op(A[a]) op(B[b]) + beta * C[d], one
      TAPP_execute_product. a, b, d: the labels, one letter per mode; ext: the
      extents, "a=16 b=16"; storage, c_storage: element types of A, B and of
      C, D; prec: the TAPP precision; f32_mode, f64_mode: the executor's
      options (tapp_b200.h); wait: the call returns when D is there, as a
      caller of the reference has it, else it is queued on the stream; values:
      how A, B and C are distributed; view: A is a window of a larger buffer
      with its first mode running backwards and its last one broadcast, and D
      is stored with its last mode fastest.
  kind "batched": `batches` products of one plan, one
      TAPP_execute_batched_product.
  kind "served": `requests` products of the served mix, queued on a server and
      drained.

All tensors are dense and column-major unless a view is asked for.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "reference-implementation_b200"))

import tapp_b200  # noqa: E402
from tapp_b200.server import Server  # noqa: E402
from tapp_b200.workloads import served_stream  # noqa: E402

TYPES = {"f32": (tapp_b200.TAPP_F32, torch.float32, np.float32), "f64": (tapp_b200.TAPP_F64, torch.float64, np.float64),
         "c32": (tapp_b200.TAPP_C32, torch.complex64, np.complex64),
         "c64": (tapp_b200.TAPP_C64, torch.complex128, np.complex128),
         "f16": (tapp_b200.TAPP_F16, torch.float16, None), "bf16": (tapp_b200.TAPP_BF16, torch.bfloat16, None)}
PRECS = {"default": tapp_b200.TAPP_DEFAULT_PREC, "f32": tapp_b200.TAPP_F32F32_ACCUM_F32,
         "f64": tapp_b200.TAPP_F64F64_ACCUM_F64, "f16_f32": tapp_b200.TAPP_F16F16_ACCUM_F32,
         "bf16_f32": tapp_b200.TAPP_BF16BF16_ACCUM_F32}
ROUNDED = {"f16_f32": torch.float16, "bf16_f32": torch.bfloat16}  # the precisions that round their operands
STORAGE_NAME = {v[0]: k for k, v in TYPES.items()}


def product(name, a, b, d, ext, storage="f32", prec="f32", alpha=1.0, beta=0.5, values="uniform", wait=False,
            c_storage="", f32_mode=0, f64_mode=0, conj_a=False, conj_b=False, view=False):
    case = {"name": name, "kind": "product", "a": a, "b": b, "d": d,
            "ext": " ".join("%s=%d" % (k, ext[k]) for k in sorted(ext)), "storage": storage,
            "c_storage": c_storage or storage, "prec": prec, "alpha": alpha, "beta": beta, "values": values,
            "wait": wait, "f32_mode": f32_mode, "f64_mode": f64_mode, "conj_a": conj_a, "conj_b": conj_b, "view": view}
    if not name:
        del case["name"]
    return case


def all_of(labels, n):
    return {x: n for x in labels}


def listed():
    return [
        # the smallest call a program makes: a few values, the default executor, wait for the result (the size of the
        # reference's own tests and of a loop over small blocks)
        product("tiny_f64", "aebf", "fced", "abcd", all_of("abcdef", 4), "f64", "f64", 1.3, 0.7, wait=True),
        # the reference's plain binary contraction, every extent 16, called and waited for
        product("dense16_f32", "aebf", "fced", "abcd", all_of("abcdef", 16), "f32", "f32", 1.3, 0.7, wait=True),
        # every class of index in one product: Hadamard, diagonal, unary, a backward and a broadcast stride, conj(B)
        product("mixed_c32", "ahkku", "khcv", "ahc", {"a": 40, "h": 12, "k": 24, "u": 6, "c": 36, "v": 5}, "c32",
                "default", 0.4, -0.7, wait=True, conj_b=True, view=True),
        # the large dense contraction (M = N = K = 4096) in the precisions it is run in: 16-bit tensor cores ...
        product("dense64_bf16", "acid", "dbcj", "abij", all_of("abcdij", 64), "f32", "bf16_f32", values="outliers"),
        # ... binary32 results from the tensor cores ...
        product("dense64_split", "acid", "dbcj", "abij", all_of("abcdij", 64), "f32", "f32", values="outliers", f32_mode=1),
        # ... and plain binary32, what a caller gets who asks for nothing
        product("dense64_f32", "acid", "dbcj", "abij", all_of("abcdij", 64), "f32", "f32", values="outliers"),
        # double precision as a coupled-cluster code contracts, native arithmetic: the largest work here
        product("double160_f64", "abef", "efij", "abij", {"a": 160, "b": 160, "e": 160, "f": 160, "i": 40, "j": 40},
                "f64", "default", 1.0, 1.0, values="loguniform"),
        # complex double with conj(A) on the integer tensor cores, 8 slices (as accurate as native)
        product("sliced96_c64", "abef", "efij", "abij", {"a": 96, "b": 96, "e": 96, "f": 96, "i": 40, "j": 40}, "c64",
                "default", 1.0, 1.0, values="loguniform", f64_mode=8, conj_a=True),
        # a Tucker mode-n product, the commonest request of the served mix, with odd extents and an odd rank
        product("tucker_f32", "abcd", "rc", "abrd", {"a": 77, "b": 190, "c": 133, "d": 61, "r": 33}, "f32", "f32", 0.7, 0.3),
        # a batched Hadamard product with a short contraction, operands stored in unlike orders
        product("hadamard_f32", "abkcd", "ckab", "dcba", {"a": 72, "b": 8, "k": 69, "c": 74, "d": 67}, "f32", "f32", 0.9, -0.3),
        # many equal products of middle size in one call
        {"name": "batched512_bf16", "kind": "batched", "batches": 64, "m": 512, "n": 512, "k": 512, "storage": "f32",
         "prec": "bf16_f32", "f32_mode": 0, "alpha": 1.0, "beta": 0.5},
        # the served mix: uneven products of four types, queued at once and drained
        {"name": "served48", "kind": "served", "requests": 48, "stream": 5, "tensor_mib": 64},
    ]


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["tiny", "dense", "mixed", "large", "double", "tucker", "hadamard", "batched", "served"])
    scal = dict(alpha=round(rng.uniform(-1, 1), 3), beta=round(rng.uniform(-1, 1), 3))
    if kind == "tiny":
        storage = rng.choice(["f32", "f64", "c32"])
        return product("", "aebf", "fced", "abcd", {x: rng.randint(2, 6) for x in "abcdef"}, storage,
                       {"f32": "f32", "f64": "f64", "c32": "default"}[storage], wait=True, **scal)
    if kind == "dense":
        return product("", "aebf", "fced", "abcd", {x: log_int(rng, 7, 28) for x in "abcdef"}, "f32", "f32", wait=True, **scal)
    if kind == "mixed":
        ext = {"a": rng.randint(20, 60), "h": rng.randint(6, 16), "k": rng.randint(12, 32), "u": rng.randint(2, 8),
               "c": rng.randint(20, 48), "v": rng.randint(2, 6)}
        return product("", "ahkku", "khcv", "ahc", ext, "c32", "default", wait=True, conj_b=True, view=True, **scal)
    if kind == "large":
        prec, mode = rng.choice([("bf16_f32", 0), ("f16_f32", 0), ("f32", 1), ("f32", 0)])
        storage = {"bf16_f32": rng.choice(["f32", "bf16"]), "f16_f32": rng.choice(["f32", "f16"]), "f32": "f32"}[prec]
        step = rng.choice([1, 4, 8])
        ext = {x: log_int(rng, 20, 64) // step * step for x in "abcdij"}
        return product("", "acid", "dbcj", "abij", ext, storage, prec, c_storage="f32", f32_mode=mode,
                       alpha=1.0, beta=0.5, values="outliers" if storage == "f32" else "uniform")
    if kind == "double":
        storage = rng.choice(["f64", "c64"])
        ext = {x: log_int(rng, 32, 112 if storage == "f64" else 80) for x in "abef"}
        ext.update(i=rng.randint(12, 40), j=rng.randint(12, 40))
        return product("", "abef", "efij", "abij", ext, storage, "default", 1.0, 1.0, values="loguniform",
                       f64_mode=rng.choice([0, 0, 7, 8]), conj_a=storage == "c64")
    if kind == "tucker":
        storage, prec = rng.choice([("f32", "f32"), ("f32", "f32"), ("f32", "bf16_f32"), ("f64", "default"), ("c32", "default")])
        order = rng.choice([3, 4])
        while True:
            e = [rng.randint(8, 256) for _ in range(order)]
            if math.prod(e) <= (1 << 27):
                break
        core, n = "abcd"[:order], rng.randrange(order)
        ext = dict(zip(core, e), r=rng.randint(4, 64))
        return product("", core, "r" + core[n], core.replace(core[n], "r"), ext, storage, prec, **scal)
    if kind == "hadamard":
        while True:
            ext = {x: log_int(rng, 4, 96) for x in "abkcd"}
            if math.prod(ext.values()) <= 200_000_000 and ext["a"] * ext["b"] * ext["c"] >= 256:
                break
        orders = ["".join(rng.sample(x, len(x))) for x in ("abkcd", "abkc", "abcd")]
        storage = rng.choice(["f32", "f32", "f64", "c32"])
        return product("", *orders, ext, storage, "f32" if storage == "f32" else "default", **scal)
    if kind == "batched":
        prec, mode = rng.choice([("bf16_f32", 0), ("f16_f32", 0), ("f32", 1)])
        m, n, k = (log_int(rng, 96, 640) // 8 * 8 + rng.choice([0, 0, 3]) for _ in range(3))
        return {"kind": "batched", "batches": rng.randint(4, 64), "m": m, "n": n, "k": k, "storage": "f32", "prec": prec,
                "f32_mode": mode, "alpha": 1.0, "beta": 0.5}
    return {"kind": "served", "requests": rng.randint(12, 48), "stream": rng.randrange(1 << 20),
            "tensor_mib": rng.choice([16, 32, 64])}


# ---------------------------------------------------------------------------
# inputs

def values(n, dtype, how, gen):
    """n values: uniform in [-1, 1] (real and imaginary parts), normal with 1% of them scaled by 1e3, or of log-uniform
    magnitude in [1e-8, 1] with random sign or phase"""
    real = {torch.complex64: torch.float32, torch.complex128: torch.float64}.get(dtype, dtype)
    if real in (torch.float16, torch.bfloat16):
        real = torch.float32
    rand = lambda: torch.rand(n, dtype=real, device="cuda", generator=gen)  # noqa: E731
    if how == "outliers":
        x = torch.randn(n, dtype=real, device="cuda", generator=gen)
        return x.mul_(torch.where(rand() < 0.01, 1e3, 1.0).to(real)).to(dtype)
    if how == "loguniform":
        mag = rand().mul_(-8 * math.log(10)).exp_()
        if dtype.is_complex:
            return torch.polar(mag, rand().mul_(2 * math.pi))
        return mag.mul_(torch.where(rand() < 0.5, -1.0, 1.0).to(real))
    if dtype.is_complex:
        return torch.complex(rand().mul_(2).sub_(1), rand().mul_(2).sub_(1))
    return rand().mul_(2).sub_(1).to(dtype)


def colmajor(ext):
    s, at = [], 1
    for e in ext:
        s.append(at)
        at *= e
    return s


class Operand:
    """One tensor in device memory: what TAPP is told of it (type, extents, strides, address of coordinate 0)."""

    def __init__(self, storage, ext, strides=None, how=None, gen=None, pad=0):
        self.storage, self.ext = storage, list(ext)
        self.strides = strides or colmajor(ext)
        low = sum(s * (e - 1) for s, e in zip(self.strides, self.ext) if s < 0)
        high = sum(s * (e - 1) for s, e in zip(self.strides, self.ext) if s > 0)
        self.base = pad - low
        dtype = TYPES[storage][1]
        n = high - low + 1 + pad
        self.flat = values(n, dtype, how, gen) if how else torch.zeros(n, dtype=dtype, device="cuda")

    @property
    def ptr(self):
        return self.flat.data_ptr() + self.base * self.flat.element_size()

    def tensor(self):
        """The tensor by its coordinates: a view, a copy where a stride is negative."""
        back = [k for k, s in enumerate(self.strides) if s < 0]
        start = self.base + sum(self.strides[k] * (self.ext[k] - 1) for k in back)
        t = self.flat.as_strided(self.ext, [abs(s) for s in self.strides], start)
        return t.flip(back) if back else t


def extents(case):
    return {k: int(v) for k, v in (x.split("=") for x in case["ext"].split())}


def operands(case, seed):
    """A, B, C and D of a product from the seed"""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    ext = extents(case)
    e = lambda labels: [ext[x] for x in labels]  # noqa: E731
    sa, sd, pad = None, None, 0
    if case["view"]:
        outer = ext[case["a"][0]] + 4
        sa = [-1] + [outer * math.prod(e(case["a"][1:k])) for k in range(1, len(case["a"]) - 1)] + [0]
        last, rest = ext[case["d"][-1]], e(case["d"][:-1])
        pad = 2
        sd = [last * s for s in colmajor([rest[0]] + rest[1:])] + [1]
    how = case["values"]
    return [Operand(case["storage"], e(case["a"]), sa, how, gen, pad), Operand(case["storage"], e(case["b"]), None, how, gen),
            Operand(case["c_storage"], e(case["d"]), None, how, gen), Operand(case["c_storage"], e(case["d"]), sd)]


def scalar(storage, v):
    return np.array([v], dtype=TYPES[storage][2])


class Plan:
    """Tensor infos and product object, as a program keeps them between calls"""

    def __init__(self, ops, labels, prec, conj=(False, False)):
        self.lib = tapp_b200.load()
        self.infos = []
        for o in ops:
            err, h = self.lib.tensor_info(TYPES[o.storage][0], o.ext, o.strides)
            if err:
                raise RuntimeError("TAPP_create_tensor_info: %d" % err)
            self.infos.append(h)
        err, self.plan = self.lib.create_product(0, [int(conj[0]), int(conj[1]), 0, 0], self.infos, labels, prec)
        if err:
            raise RuntimeError("TAPP_create_tensor_product: %d" % err)

    def __del__(self):
        self.lib.lib.TAPP_destroy_tensor_product(self.plan)
        for h in self.infos:
            self.lib.lib.TAPP_destroy_tensor_info(h)


class Executor:
    def __init__(self, wait, f32_mode=0, f64_mode=0):
        self.lib = tapp_b200.load()
        self.handle = self.lib.create_executor()
        if not wait:
            self.lib.set_stream(self.handle, torch.cuda.current_stream().cuda_stream)
            self.lib.set_int(self.handle, tapp_b200.ATTR_ASYNC, 1)
        if f32_mode:
            self.lib.set_int(self.handle, tapp_b200.ATTR_F32_MODE, f32_mode)
        if f64_mode:
            self.lib.set_int(self.handle, tapp_b200.ATTR_F64_MODE, f64_mode)

    def __del__(self):
        self.lib.lib.TAPP_destroy_executor(self.handle)


def check(err):
    if err:
        raise RuntimeError("TAPP error %#x: %s" % (err, tapp_b200.load().explain(err)))


class Product:
    def __init__(self, case, seed):
        self.ops = operands(case, seed)
        labels = [[ord(x) for x in case[k]] for k in "abdd"]
        self.plan = Plan(self.ops, labels, PRECS[case["prec"]], (case["conj_a"], case["conj_b"]))
        self.executor = Executor(case["wait"], case["f32_mode"], case["f64_mode"])
        self.alpha, self.beta = (scalar(case["c_storage"], case[k]) for k in ("alpha", "beta"))
        self.out = self.ops[3].tensor()
        self.args = (self.plan.plan, self.executor.handle, self.alpha.ctypes.data, self.ops[0].ptr, self.ops[1].ptr,
                     self.beta.ctypes.data, self.ops[2].ptr, self.ops[3].ptr)
        self.execute = self.plan.lib.execute

    def run(self):
        check(self.execute(*self.args))
        return self.out


def batch_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    m, n, k, num = case["m"], case["n"], case["k"], case["batches"]
    dtype = TYPES[case["storage"]][1]
    return [values(num * x, dtype, "uniform", gen).view(num, x) for x in (m * k, k * n, m * n)]


class Batched:
    def __init__(self, case, seed):
        m, n, k, num = case["m"], case["n"], case["k"], case["batches"]
        self.bufs = batch_inputs(case, seed)
        self.bufs.append(torch.zeros_like(self.bufs[2]))
        shapes = [Operand(case["storage"], x) for x in ([m, k], [k, n], [m, n], [m, n])]
        self.plan = Plan(shapes, [[ord(x) for x in y] for y in ("ak", "kb", "ab", "ab")], PRECS[case["prec"]])
        self.executor = Executor(False, case["f32_mode"])
        self.alpha, self.beta = (scalar(case["storage"], case[x]) for x in ("alpha", "beta"))
        lists = [(ctypes.c_void_p * num)(*[b[i].data_ptr() for i in range(num)]) for b in self.bufs]
        self.status = ctypes.c_ssize_t(0)
        self.args = (self.plan.plan, self.executor.handle, ctypes.byref(self.status), num, self.alpha.ctypes.data, lists[0],
                     lists[1], self.beta.ctypes.data, lists[2], lists[3])
        self.execute = self.plan.lib.lib.TAPP_execute_batched_product

    def run(self):
        check(self.execute(*self.args))
        return self.bufs[3]


def served_specs(case):
    return served_stream(np.random.default_rng(case["stream"]), case["requests"], max_tensor_bytes=case["tensor_mib"] << 20)


def served_operands(spec, gen):
    storage = STORAGE_NAME[spec.storage]
    return [Operand(storage, spec.extents[k], None, "uniform" if k < 3 else None, gen) for k in range(4)]


class Served:
    def __init__(self, case, seed):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        self.keep, self.calls, self.outs = [], [], []
        for spec in served_specs(case):
            ops = served_operands(spec, gen)
            plan = Plan(ops, [list(x) for x in spec.idx], spec.prec)
            real = ops[0].flat.dtype.is_complex
            alpha, beta = (scalar(ops[3].storage, v if real else np.real(v)) for v in (spec.alpha, spec.beta))
            self.keep.append((ops, plan, alpha, beta))
            self.calls.append((plan.plan, alpha.ctypes.data, ops[0].ptr, ops[1].ptr, beta.ctypes.data, ops[2].ptr, ops[3].ptr))
            self.outs.append(ops[3].tensor())
        torch.cuda.synchronize()  # the server works on streams of its own
        self.server = Server(tapp_b200.load(), 64 << 30, n_streams=8, max_in_flight=64)

    def run(self):
        submit = self.server.submit
        for call in self.calls:
            check(submit(*call)[0])
        check(self.server.drain())
        self.server.reset_stats()
        return self.outs

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()


def prepare(case, seed):
    return {"product": Product, "batched": Batched, "served": Served}[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it has to give

def size_of(storage):
    return {"f16": 2, "bf16": 2, "f32": 4, "f64": 8, "c32": 8, "c64": 16}[storage]


def product_work(a, b, d, ext, storage, c_storage):
    """Every addressed element once (a label in two modes of a tensor addresses its diagonal), two operations for each
    product of two real numbers"""
    count = lambda labels: math.prod(ext[x] for x in set(labels))  # noqa: E731
    terms = count(d) * count([x for x in set(a) & set(b) if x not in d])
    return {"bytes": (count(a) + count(b)) * size_of(storage) + 2 * count(d) * size_of(c_storage),
            "flops": (8 if storage in ("c32", "c64") else 2) * terms}


def work(case):
    if case["kind"] == "product":
        a = case["a"][:-1] if case["view"] else case["a"]  # a broadcast mode holds nothing of its own
        return product_work(a, case["b"], case["d"], extents(case), case["storage"], case["c_storage"])
    if case["kind"] == "batched":
        one = product_work("ak", "kb", "ab", {"a": case["m"], "b": case["n"], "k": case["k"]}, case["storage"], case["storage"])
        return {k: v * case["batches"] for k, v in one.items()}
    total = {"bytes": 0, "flops": 0}
    for s in served_specs(case):
        total["bytes"] += sum(s.nbytes(k) for k in range(4))
        total["flops"] += s.flops()
    return total


def wide(t, prec):
    """A tensor in 64 bits, rounded first where the precision rounds its operands"""
    if prec in ROUNDED:
        t = t.to(ROUNDED[prec])
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def exact_product(ops, labels, prec, alpha, beta, conj=(False, False)):
    if prec in ROUNDED:
        alpha, beta = (float(torch.tensor(x).to(ROUNDED[prec])) for x in (alpha, beta))
    elif ops[3].storage in ("f32", "c32"):
        alpha, beta = (complex(np.complex64(x)) if isinstance(x, complex) else float(np.float32(x)) for x in (alpha, beta))
    A, B, C = (wide(o.tensor(), prec) for o in ops[:3])
    A, B = (x.conj() if c else x for x, c in zip((A, B), conj))
    return alpha * torch.einsum("%s,%s->%s" % labels, A, B) + beta * C


def exact(case, seed):
    if case["kind"] == "product":
        return exact_product(operands(case, seed), (case["a"], case["b"], case["d"]), case["prec"], case["alpha"],
                             case["beta"], (case["conj_a"], case["conj_b"]))
    if case["kind"] == "batched":
        m, n, k, num = case["m"], case["n"], case["k"], case["batches"]
        A, B, C = (wide(x, case["prec"]) for x in batch_inputs(case, seed))
        D = case["alpha"] * torch.bmm(B.view(num, n, k), A.view(num, k, m)).view(num, -1) + case["beta"] * C
        return D
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = []
    for spec in served_specs(case):
        ops = served_operands(spec, gen)
        real = spec.storage not in (tapp_b200.TAPP_C32, tapp_b200.TAPP_C64)
        alpha, beta = (v.real if real else v for v in (complex(spec.alpha), complex(spec.beta)))
        labels = tuple("".join(chr(97 + x) for x in spec.idx[k]) for k in (0, 1, 3))
        prec = "bf16_f32" if spec.prec == tapp_b200.TAPP_BF16BF16_ACCUM_F32 else "f32"
        out.append(exact_product(ops, labels, prec, alpha, beta))
    return out
