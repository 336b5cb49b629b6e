"""GPU parity of the tiled GEMM over asynchronous copies (csrc/cuda/tile.cu)
at the edges of its tiles, slices, copy forms and splits, against the
oracle's binary64 evaluation with helpers.error_bound.
"""
import numpy as np
import pytest

import tapp_b200
from families import bounded_case
from helpers import d_values, error_bound
from test_gpu_parity import check_against_f64
from test_gpu_simt import simt_executor, spec_case

pytestmark = pytest.mark.gpu

TYPES = [(0, 0), (0, 6), (1, -1), (2, -1), (3, -1)]


# rows, columns, contraction: one of each; remainders of every tile and slice; contractions that one block walks,
# that 2, 4 and 8 blocks of a cluster share (some with an empty last share) and that go through the workspace
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (17, 16, 15), (130, 33, 65), (64, 65, 129), (257, 9, 200), (63, 61, 1040),
                                   (131, 129, 333), (20, 18, 4099)])
@pytest.mark.parametrize("a_t,b_t,d_t", [(0, 0, 0), (1, 0, 1), (0, 1, 1), (1, 1, 0)])
def test_matrix_edges(tapp, oracle, gpu, storage, prec, M, N, K, a_t, b_t, d_t):
    rng = np.random.default_rng(M * 7 + N * 5 + K + 10 * storage + prec + 4 * a_t + 2 * b_t + d_t)
    A = ([K, M], [2, 0]) if a_t else ([M, K], [0, 2])
    B = ([N, K], [1, 2]) if b_t else ([K, N], [2, 1])
    D = ([N, M], [1, 0]) if d_t else ([M, N], [0, 1])
    case = spec_case(rng, storage, prec, (A[0], B[0], D[0], D[0]), (A[1], B[1], D[1], D[1]))
    ex = simt_executor(tapp)
    check_against_f64(tapp, oracle, case, device=True, executor=ex)
    tapp.lib.TAPP_destroy_executor(ex)


# several modes per index class, Hadamard modes, windows of larger tensors, strides of both signs, every element op
@pytest.mark.parametrize("storage,prec", TYPES)
@pytest.mark.parametrize("seed", range(6))
def test_strided_products(tapp, oracle, gpu, storage, prec, seed):
    rng = np.random.default_rng(1000 * seed + 10 * storage + prec)
    case = bounded_case(rng, dtype=storage, prec=prec, n_contracted=1 + seed % 3, n_freeA=1 + seed % 2,
                        n_freeB=1 + (seed // 2) % 2, n_hadamard=(seed // 3) % 2, ext_choices=[2, 4, 9, 16, 33, 70],
                        ops=[seed & 1, (seed >> 1) & 1, 1, 0], subtensor=seed % 2 == 1, mixed=seed >= 4, max_work=4e6)
    ex = simt_executor(tapp)
    check_against_f64(tapp, oracle, case, device=True, executor=ex)
    tapp.lib.TAPP_destroy_executor(ex)


# complex operands aligned to their real part only, as C allows
@pytest.mark.parametrize("storage", [2, 3])
@pytest.mark.parametrize("a_t", [0, 1])
def test_complex_operands_aligned_to_their_parts(tapp, oracle, gpu, storage, a_t):
    import torch
    rng = np.random.default_rng(70 + storage + a_t)
    A = ([40, 66], [2, 0]) if a_t else ([66, 40], [0, 2])
    case = spec_case(rng, storage, -1, (A[0], [40, 35], [66, 35], [66, 35]), (A[1], [2, 1], [0, 1], [0, 1]))
    shift, dev, ptrs = (4 if storage == 2 else 8), [], []
    for t in (case.A, case.B, case.C, case.D):
        raw = np.zeros(t.buf.nbytes + shift, dtype=np.uint8)
        raw[shift:] = t.buf.view(np.uint8)
        dev.append(torch.from_numpy(raw).cuda())
        ptrs.append(dev[-1].data_ptr() + shift + t.base * t.itemsize)
    ex = simt_executor(tapp)
    assert case.run(tapp, executor=ex, A_ptr=ptrs[0], B_ptr=ptrs[1], C_ptr=ptrs[2], D_ptr=ptrs[3]) == 0
    torch.cuda.synchronize()
    tapp.lib.TAPP_destroy_executor(ex)
    run = case.copy()
    run.D.buf[:] = np.frombuffer(dev[3].cpu().numpy()[shift:].tobytes(), dtype=run.D.buf.dtype)
    e64, D64, scale = oracle.execute_f64(case.copy())
    assert e64 == 0
    assert (np.abs(d_values(run.D) - D64) <= error_bound(case, scale, D64)).all()


# a product gives the same bits in every run, also where ranks or splits are added
@pytest.mark.parametrize("storage", [0, 1, 2, 3])
@pytest.mark.parametrize("M,N,K", [(100, 90, 700), (20, 18, 6000)])
def test_same_bits_every_run(tapp, gpu, storage, M, N, K):
    from helpers import run_on_device
    case = spec_case(np.random.default_rng(5), storage, -1, ([M, K], [K, N], [M, N], [M, N]), ([0, 2], [2, 1], [0, 1], [0, 1]))
    ex = simt_executor(tapp)
    got = []
    for _ in range(3):
        run = case.copy()
        assert run_on_device(tapp, run, ex) == 0
        got.append(run.D.buf.tobytes())
    tapp.lib.TAPP_destroy_executor(ex)
    assert got[0] == got[1] == got[2]
    assert tapp_b200.load().launches() > 0


# products of many rows and up to 64 columns, with remainders in columns, rows and contraction, in whichever narrow or
# tiled kernel the rules give them (test_gpu_tile_forms.py has every tall tile)
@pytest.mark.parametrize("storage,prec", [(0, 0), (0, 6), (1, -1), (2, -1)])
@pytest.mark.parametrize("N", [1, 8, 11, 16, 23, 31, 36, 39, 48, 59, 64])
@pytest.mark.parametrize("M,a_t", [(38004, 0), (38002, 0), (37999, 0), (37999, 1)])
def test_tall_products(tapp, oracle, gpu, storage, prec, N, M, a_t):
    rng = np.random.default_rng(N + M + a_t + 10 * storage + prec)
    A = ([131, M], [2, 0]) if a_t else ([M, 131], [0, 2])
    case = spec_case(rng, storage, prec, (A[0], [N, 131], [M, N], [M, N]), (A[1], [1, 2], [0, 1], [0, 1]))
    ex = simt_executor(tapp)
    samples = np.random.default_rng(7).integers(0, M * N, 4096)
    from helpers import run_on_device
    run = case.copy()
    assert run_on_device(tapp, run, ex) == 0
    tapp.lib.TAPP_destroy_executor(ex)
    err, D64, scale, offs = oracle.execute_f64(case.copy(), samples=samples)
    assert err == 0
    assert (np.abs(run.D.buf[run.D.base + offs].astype(np.complex128) - D64) <= error_bound(case, scale, D64)).all()
