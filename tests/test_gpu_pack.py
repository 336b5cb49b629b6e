"""GPU parity of the 16-byte operand packs (tc.cu: k_pack_runs, k_pack_cols) and
of the TMA epilogue's boxes, at the edges of their tiles, against the oracle
with the bounds of test_gpu_tc.py.
"""
import numpy as np
import pytest

from test_gpu_parity import check_against_f64
from test_gpu_simt import spec_case
from test_gpu_tc import SPLIT_REL, tc_executor, path_of

pytestmark = pytest.mark.gpu


# A and B contiguous along their rows or the contraction; rows and contractions that fill a tile of 32 x 256 or 64 x 128,
# part of one, and several; D's first two modes multiples of 32 (TMA boxes) and not
@pytest.mark.parametrize("prec,split", [(6, False), (5, False), (0, True)])
@pytest.mark.parametrize("M,N,K", [(4, 64, 36), (68, 132, 260), (132, 68, 124), (64, 36, 520), (288, 96, 256)])
@pytest.mark.parametrize("a_t,b_t", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_matrix_edges(tapp, oracle, gpu, prec, split, M, N, K, a_t, b_t):
    rng = np.random.default_rng(M + 3 * N + 5 * K + prec + 2 * a_t + b_t)
    A = ([K, M], [2, 0]) if a_t else ([M, K], [0, 2])
    B = ([N, K], [1, 2]) if b_t else ([K, N], [2, 1])
    case = spec_case(rng, 0, prec, (A[0], B[0], [M, N], [M, N]), (A[1], B[1], [0, 1], [0, 1]))
    ex = tc_executor(tapp, split=split)
    assert "path=tc" in path_of(tapp, case, ex)
    check_against_f64(tapp, oracle, case, device=True, executor=ex, extra_rel=SPLIT_REL if split else 0.0)
    tapp.lib.TAPP_destroy_executor(ex)


# several row, contracted and batch modes, each a multiple of 4 along the contiguous one
@pytest.mark.parametrize("prec,split", [(6, False), (0, True)])
@pytest.mark.parametrize("a,b", [("mikjl", "kjnl"), ("kmjil", "nkjl"), ("jkmil", "lkjn")])
def test_several_modes(tapp, oracle, gpu, prec, split, a, b):
    ext = {"m": 12, "i": 9, "k": 20, "j": 8, "n": 68, "l": 3}
    e = lambda labels: [ext[x] for x in labels]
    i = lambda labels: [ord(x) for x in labels]
    case = spec_case(np.random.default_rng(len(a) + ord(a[0])), 0, prec, (e(a), e(b), e("minl"), e("minl")),
                     (i(a), i(b), i("minl"), i("minl")))
    ex = tc_executor(tapp, split=split)
    assert "path=tc" in path_of(tapp, case, ex)
    check_against_f64(tapp, oracle, case, device=True, executor=ex, extra_rel=SPLIT_REL if split else 0.0)
    tapp.lib.TAPP_destroy_executor(ex)
