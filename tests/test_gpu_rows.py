"""GPU parity of the element path with several outputs per thread or per warp
(generic.cu: k_element_rows, k_warp_rows): batched products with one mode that
only one operand has, at extents around the group sizes, in unlike orders.
The oracle bound is helpers.error_bound; the bits must be those of the kernel
that takes one output at a time (a batch of two runs it in the grouped launch).
"""
import ctypes
import numpy as np
import pytest

import tapp_b200
from test_gpu_parity import check_against_f64
from test_gpu_simt import describe, spec_case

pytestmark = pytest.mark.gpu

TYPES = [(0, 0), (0, 6), (1, -1), (2, -1), (3, -1)]


def product(seed, storage, prec, a, b, d, ext):
    e = lambda labels: [ext[x] for x in labels]
    i = lambda labels: [ord(x) for x in labels]
    return spec_case(np.random.default_rng(seed), storage, prec, (e(a), e(b), e(d), e(d)), (i(a), i(b), i(d), i(d)))


def grouped_bits(tapp, case):
    """D of the case run as a batch of two, which the grouped element launch computes one output at a time."""
    import torch
    ts = (case.A, case.B, case.C, case.D)
    dev = [[torch.from_numpy(t.buf.view(np.uint8).copy()).cuda() for t in ts] for _ in range(2)]
    infos = [tapp.tensor_info(t.dtype, t.extents, t.strides)[1] for t in ts]
    err, plan = tapp.create_product(0, [t.op for t in ts], infos, [t.idx for t in ts], case.prec)
    assert err == 0
    lists = [(ctypes.c_void_p * 2)(*[dev[k][j].data_ptr() for k in range(2)]) for j in range(4)]
    ex, st = tapp.create_executor(), ctypes.c_ssize_t(0)
    assert tapp.lib.TAPP_execute_batched_product(plan, ex, ctypes.byref(st), 2, case.alpha.ctypes.data, lists[0], lists[1],
                                                 case.beta.ctypes.data, lists[2], lists[3]) == 0
    torch.cuda.synchronize()
    tapp.lib.TAPP_destroy_executor(ex)
    tapp.lib.TAPP_destroy_tensor_product(plan)
    return dev[0][3].cpu().numpy().tobytes(), dev[1][3].cpu().numpy().tobytes()


def check(tapp, oracle, case, kernel):
    from helpers import run_on_device
    ex = tapp.create_executor()
    assert f"kernel={kernel}" in describe(tapp, case, ex)
    check_against_f64(tapp, oracle, case, device=True, executor=ex)
    run = case.copy()
    assert run_on_device(tapp, run, ex) == 0
    tapp.lib.TAPP_destroy_executor(ex)
    one, two = grouped_bits(tapp, case)
    assert run.D.buf.view(np.uint8).tobytes() == one == two


# the mode d is A's alone, walked last or first; the batch is large enough for 4 rows a thread at most
# (test_gpu_row_forms.py has the others)
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("d,batch", [(3, 200), (8, 160), (21, 110), (5, 300)])
@pytest.mark.parametrize("a,b,o", [("abkd", "bka", "dab"), ("abkd", "kab", "abd"), ("dabk", "abk", "dab")])
def test_outputs_of_a_thread(tapp, oracle, gpu, storage, prec, d, batch, a, b, o):
    case = product(d + batch, storage, prec, a, b, o, {"a": batch, "b": 401, "d": d, "k": 5})
    check(tapp, oracle, case, "element")


# the operand that varies may be B
@pytest.mark.parametrize("storage,prec", [(0, 0), (3, -1)])
def test_outputs_of_a_thread_along_b(tapp, oracle, gpu, storage, prec):
    check(tapp, oracle, product(9, storage, prec, "bka", "abkd", "dab", {"a": 120, "b": 401, "d": 9, "k": 6}), "element")


# one warp for several outputs: the contraction contiguous in A, rows along A's own mode d or B's own mode e, with and
# without unary modes u (A) and v (B)
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("d,k", [(3, 64), (9, 70), (21, 131)])
def test_outputs_of_a_warp(tapp, oracle, gpu, storage, prec, d, k):
    check(tapp, oracle, product(d + k, storage, prec, "kabd", "kab", "dab", {"a": 40, "b": 51, "d": d, "k": k}), "warpdot")


@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("a,b", [("ahku", "khev"), ("ahk", "kehv"), ("uahk", "keh")])
@pytest.mark.parametrize("sizes", [(40, 12, 24, 36), (13, 30, 9, 11)])
def test_outputs_of_a_warp_with_unary_modes(tapp, oracle, gpu, storage, prec, a, b, sizes):
    ext = dict(zip("ahke", sizes), u=6, v=5)
    case = product(sum(sizes), storage, prec, a, b, "ahe", ext)
    # fewer than 64 loads an output stay with one thread per output
    check(tapp, oracle, case, "warpdot" if ext["k"] * ((6 if "u" in a else 1) + (5 if "v" in b else 1)) >= 64 else "element")
