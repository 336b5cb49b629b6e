"""GPU parity of every form of the element path's row kernels (generic.cu:
k_element_rows, k_warp_rows and the one-output kernels beside them), each
asserted through tapp_b200_describe_plan before it runs: 8 and 4 rows of a
step, neighbours and spread over the mode that is walked first, the varying
operand A or B, operands of every kind of load, sums longer than the offset
tables. Checked against the oracle's binary64 sums (helpers.error_bound, a
sample of the outputs) and, bit for bit, against the grouped launch, which
takes one output at a time.
"""
import numpy as np
import pytest

from helpers import error_bound, run_on_device
from test_dispatch_cpu import field
from test_gpu_rows import grouped_bits, product
from test_gpu_simt import describe

pytestmark = pytest.mark.gpu

# storage, precision: stored as computed, rounded, 16 bits of both kinds
TYPES = [(0, 0), (0, 6), (1, -1), (2, -1), (3, -1), (2, 6), (4, 5), (5, -1)]


def check(tapp, oracle, case, kernel, rows, spread=None, along=None):
    ex = tapp.create_executor()
    text = describe(tapp, case, ex)
    assert (field(text, "kernel"), field(text, "rows")) == (kernel, str(rows)), text
    if rows > 1:
        assert (field(text, "spread"), field(text, "along")) == (str(int(spread)), along), text
    run = case.copy()
    assert run_on_device(tapp, run, ex) == 0
    tapp.lib.TAPP_destroy_executor(ex)
    outputs = int(np.prod(case.D.extents))
    err, D64, scale, offs = oracle.execute_f64(case.copy(), samples=np.random.default_rng(3).integers(0, outputs, 4096))
    assert err == 0
    got = run.D.copy()
    got.buf = got.buf[got.base + offs]
    from helpers import d_values
    assert (np.abs(d_values(got) - D64) <= error_bound(case, scale, D64)).all()
    one, two = grouped_bits(tapp, case)
    assert run.D.buf.view(np.uint8).tobytes() == one == two


# groups of 8 with a remainder of 1, 5 and none; groups of 4 where 8 leave the GPU idle; the mode walked last
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("d,a,rows", [(9, 300, 8), (21, 180, 8), (16, 200, 8), (5, 250, 4)])
def test_neighbouring_rows_of_a_thread(tapp, oracle, gpu, storage, prec, d, a, rows):
    case = product(d, storage, prec, "abkd", "bka", "abd", {"a": a, "b": 401, "d": d, "k": 3})
    check(tapp, oracle, case, "element", rows, False, "A")


@pytest.mark.parametrize("storage,prec", [(0, 0), (3, -1), (5, 6)])
def test_rows_of_a_thread_along_b(tapp, oracle, gpu, storage, prec):
    case = product(8, storage, prec, "bka", "abkd", "abd", {"a": 300, "b": 401, "d": 11, "k": 3})
    check(tapp, oracle, case, "element", 8, False, "B")


# the mode that only one operand has is walked first: 8 or 4 rows spread over it, with short last groups
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("d,rows", [(57, 8), (61, 8), (64, 8), (29, 4), (32, 4)])
def test_rows_spread_over_the_first_mode(tapp, oracle, gpu, storage, prec, d, rows):
    case = product(d, storage, prec, "dabk", "abk", "dab", {"a": 150, "b": 131, "d": d, "k": 2})
    check(tapp, oracle, case, "element", rows, True, "A")


@pytest.mark.parametrize("storage,prec", [(0, 0), (2, -1), (4, 5)])
def test_rows_spread_along_b(tapp, oracle, gpu, storage, prec):
    case = product(58, storage, prec, "abk", "dabk", "dab", {"a": 150, "b": 131, "d": 58, "k": 2})
    check(tapp, oracle, case, "element", 8, True, "B")


# rows of a warp: 8 and 4, along A's or B's mode
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("d,a,rows", [(9, 40, 8), (6, 16, 4)])
@pytest.mark.parametrize("swap", [False, True])
def test_rows_of_a_warp(tapp, oracle, gpu, storage, prec, d, a, rows, swap):
    ab = ("kab", "kabd") if swap else ("kabd", "kab")
    case = product(d, storage, prec, *ab, "abd", {"a": a, "b": 51, "d": d, "k": 99})
    check(tapp, oracle, case, "warpdot", rows, False, "B" if swap else "A")


# one row a step: a contraction longer than the offset tables (512 terms), in a thread and in a warp with unary modes
@pytest.mark.parametrize("storage,prec", TYPES)
def test_contraction_longer_than_the_tables(tapp, oracle, gpu, storage, prec):
    check(tapp, oracle, product(1, storage, prec, "abk", "abk", "ab", {"a": 200, "b": 191, "k": 517}), "element", 1)
    check(tapp, oracle, product(2, storage, prec, "abku", "kab", "ab", {"a": 30, "b": 29, "k": 517, "u": 5}), "warpdot", 1)


# unary modes of all that the tables hold (128 values) and longer, in a thread and in a warp
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("u", [128, 131])
def test_unary_modes_around_the_tables(tapp, oracle, gpu, storage, prec, u):
    rows = 0 if u > 128 and (prec in (5, 6) or storage >= 4) else 1
    check(tapp, oracle, product(3, storage, prec, "abu", "abv", "ab", {"a": 200, "b": 191, "u": u, "v": 3}), "element", rows)
    check(tapp, oracle, product(4, storage, prec, "ahku", "khv", "ah", {"a": 40, "h": 39, "k": 17, "u": u, "v": 3}), "warpdot", rows)


# rows of a warp with unary modes: 8 rows, and one where the runs along u fill lines
@pytest.mark.parametrize("storage,prec", TYPES)
def test_rows_of_a_warp_with_unary_modes(tapp, oracle, gpu, storage, prec):
    ext = {"a": 90, "h": 110, "k": 19, "u": 3, "v": 5}
    check(tapp, oracle, product(7, storage, prec, "uahk", "khv", "ah", ext), "warpdot", 8, False, "A")
    check(tapp, oracle, product(8, storage, prec, "uahk", "khv", "ah", dict(ext, u=33)), "warpdot", 1)


# one term: threads without tables
@pytest.mark.parametrize("storage,prec", TYPES)
def test_one_term(tapp, oracle, gpu, storage, prec):
    check(tapp, oracle, product(5, storage, prec, "abd", "ba", "dab", {"a": 60, "b": 71, "d": 13}), "element", 0)


# operands that are converted as they are loaded
@pytest.mark.parametrize("types,prec", [((0, 5, 0, 0), -1), ((1, 1, 0, 0), 0), ((3, 2, 3, 3), -1), ((4, 4, 2, 2), -1)])
def test_converted_operands(tapp, oracle, gpu, types, prec):
    from tapp_b200.case import alloc, fill_uniform, scalar, Case
    def tensors(labels, ext):
        out = []
        for k, (x, t) in enumerate(zip(labels, types)):
            e = [ext[c] for c in x]
            out.append(alloc(t, e, [int(np.prod(e[:j])) for j in range(len(e))], [ord(c) for c in x]))
            if k < 3:
                fill_uniform(out[-1], np.random.default_rng(k))
        return out
    for labels, ext, kernel in ((("abkd", "bka", "abd", "abd"), {"a": 300, "b": 401, "d": 9, "k": 3}, "element"),
                                (("kabd", "kab", "abd", "abd"), {"a": 40, "b": 51, "d": 9, "k": 99}, "warpdot")):
        case = Case(*tensors(labels, ext), scalar(types[3], 0.7), scalar(types[3], 0.3), prec)
        check(tapp, oracle, case, kernel, 0)


# complex operands aligned to their real part only, which the planner cannot see: one output at a time as well
@pytest.mark.parametrize("storage", [2, 3])
@pytest.mark.parametrize("a,b,d,ext", [("abkd", "bka", "abd", {"a": 300, "b": 401, "d": 9, "k": 3}),
                                       ("kabd", "kab", "abd", {"a": 40, "b": 51, "d": 9, "k": 99})])
def test_complex_operands_aligned_to_their_parts(tapp, oracle, gpu, storage, a, b, d, ext):
    import torch
    case = product(6, storage, -1, a, b, d, ext)
    one, _ = grouped_bits(tapp, case)
    shift, dev, ptrs = (4 if storage == 2 else 8), [], []
    for t in (case.A, case.B, case.C, case.D):
        raw = np.zeros(t.buf.nbytes + shift, dtype=np.uint8)
        raw[shift:] = t.buf.view(np.uint8)
        dev.append(torch.from_numpy(raw).cuda())
        ptrs.append(dev[-1].data_ptr() + shift + t.base * t.itemsize)
    ex = tapp.create_executor()
    assert case.run(tapp, executor=ex, A_ptr=ptrs[0], B_ptr=ptrs[1], C_ptr=ptrs[2], D_ptr=ptrs[3]) == 0
    torch.cuda.synchronize()
    tapp.lib.TAPP_destroy_executor(ex)
    assert dev[3].cpu().numpy()[shift:].tobytes() == one
