"""GPU parity of the tiled GEMM's forms that ordinary sizes do not reach
(csrc/cuda/tile.cu), each asserted through tapp_b200_describe_plan before it
runs: every tall tile with each way of copying its rows, alone and shared by
the ranks of a cluster, and C and D stored in other types than the operands in
every epilogue (whole tile, cluster, workspace). Against the oracle's binary64
sums with helpers.error_bound (a sample of the outputs where there are many).
"""
import numpy as np
import pytest

from helpers import d_values, error_bound, run_on_device
from tapp_b200.case import Case, alloc, fill_uniform, scalar
from test_dispatch_cpu import field
from test_gpu_simt import describe, simt_executor, spec_case

pytestmark = pytest.mark.gpu


def check(tapp, oracle, case, **want):
    ex = simt_executor(tapp)
    text = describe(tapp, case, ex)
    assert field(text, "kernel") == "tiled" and all(field(text, k) == str(v) for k, v in want.items()), text
    run = case.copy()
    assert run_on_device(tapp, run, ex) == 0
    tapp.lib.TAPP_destroy_executor(ex)
    outputs = int(np.prod(case.D.extents))
    err, D64, scale, offs = oracle.execute_f64(case.copy(), samples=np.random.default_rng(3).integers(0, outputs, 4096))
    assert err == 0
    run.D.buf = run.D.buf[run.D.base + offs]
    assert (np.abs(d_values(run.D) - D64) <= error_bound(case, scale, D64)).all()


def batched(storage, prec, M, N, K, L, a_along_k, d_columns):
    e = {"m": M, "n": N, "k": K, "l": L}
    labels = ("kml" if a_along_k else "mkl", "nkl", "nml" if d_columns else "mnl")
    labels += (labels[2],)
    return spec_case(np.random.default_rng(M + N + K + L), storage, prec, tuple([e[x] for x in y] for y in labels),
                     tuple([ord(x) for x in y] for y in labels))


# batches of few rows, which no narrow kernel takes: rows in 16-byte groups, in pairs, alone, and across the contraction
COPIES = [(500, False), (502, False), (501, False), (503, True)]


@pytest.mark.parametrize("prec", [0, 6])
@pytest.mark.parametrize("M,along", COPIES)
@pytest.mark.parametrize("N,L,tile", [(4, 460, "256x8"), (8, 460, "256x8"), (11, 460, "256x12"), (13, 230, "256x16"),
                                      (23, 230, "256x24"), (31, 140, "256x32"), (36, 140, "256x36"), (39, 140, "256x40"),
                                      (47, 140, "256x48"), (61, 140, "256x64")])
def test_tall_tiles(tapp, oracle, gpu, prec, M, along, N, L, tile):
    check(tapp, oracle, batched(0, prec, M, N, 21, L, along, N % 2), tile=tile, cluster=1, splits=1)


@pytest.mark.parametrize("M,along", COPIES)
@pytest.mark.parametrize("N,L,tile", [(5, 80, "128x8"), (15, 80, "128x16"), (22, 310, "128x24"), (43, 210, "128x48")])
def test_tall_complex_tiles(tapp, oracle, gpu, M, along, N, L, tile):
    if N == 43 and not along:
        tile = "64x64"  # wide as 48 columns only where A lies along the contraction
    check(tapp, oracle, batched(2, -1, M, N, 21, L, along, N % 2), tile=tile, cluster=1, splits=1)


# between one and one and a half tall tiles per SM, two ranks share a long contraction
@pytest.mark.parametrize("prec", [0, 6])
@pytest.mark.parametrize("N,tile", [(37, "256x40"), (63, "256x64")])
@pytest.mark.parametrize("d_columns", [False, True])
def test_tall_tiles_of_two_ranks(tapp, oracle, gpu, prec, N, tile, d_columns):
    check(tapp, oracle, batched(0, prec, 502, N, 261, 100, False, d_columns), tile=tile, cluster=2, splits=1)


# C and D in other types than A and B: whole tiles, clusters, splits through the workspace and their second kernel
@pytest.mark.parametrize("types,prec", [((0, 0, 4, 4), 0), ((0, 0, 5, 0), 0), ((0, 0, 0, 5), 6), ((0, 0, 1, 1), 0), ((0, 0, 4, 5), 5),
                                        ((1, 1, 0, 0), 1), ((1, 1, 1, 0), -1), ((2, 2, 3, 2), 0), ((2, 2, 0, 0), 0),
                                        ((3, 3, 2, 2), 1)])
@pytest.mark.parametrize("M,N,K,cluster,splits", [(1030, 1034, 33, "1", "1"), (130, 70, 300, None, "1"), (40, 36, 5000, "1", None)])
@pytest.mark.parametrize("d_columns", [False, True])
def test_other_storage_of_c_and_d(tapp, oracle, gpu, types, prec, M, N, K, cluster, splits, d_columns):
    rng = np.random.default_rng(M + N + K)
    shapes = [([M, K], [0, 2]), ([K, N], [2, 1])] + [([N, M], [1, 0]) if d_columns else ([M, N], [0, 1])] * 2
    ts = [alloc(t, e, [1, e[0]], i) for t, (e, i) in zip(types, shapes)]
    for t in ts[:3]:
        fill_uniform(t, rng)
    case = Case(*ts, scalar(types[3], 0.7), scalar(types[3], 0.3), prec)
    ex = simt_executor(tapp)
    text = describe(tapp, case, ex)
    tapp.lib.TAPP_destroy_executor(ex)
    if cluster is None:
        assert int(field(text, "cluster")) > 1, text
    if splits is None:
        assert int(field(text, "splits")) > 1, text
    check(tapp, oracle, case, **{k: v for k, v in (("cluster", cluster), ("splits", splits)) if v})


# where the buffers lie does not show in the bits: the same product 16-byte aligned and aligned to its elements only
@pytest.mark.parametrize("labels,ext,storage", [(("mk", "nk", "mn"), {"m": 10000, "n": 30, "k": 100}, 0),
                                                (("mk", "nk", "mn"), {"m": 3000, "n": 20, "k": 64}, 1),
                                                (("km", "kn", "mn"), {"m": 634, "n": 480, "k": 1536}, 0)])
def test_bits_do_not_depend_on_alignment(tapp, gpu, labels, ext, storage):
    import torch
    e, i = (lambda x: [ext[c] for c in x]), (lambda x: [ord(c) for c in x])
    case = spec_case(np.random.default_rng(9), storage, -1, tuple(e(x) for x in labels + labels[2:]),
                     tuple(i(x) for x in labels + labels[2:]))
    got = []
    for shift in (0, case.A.itemsize):
        dev, ptrs = [], []
        for t in (case.A, case.B, case.C, case.D):
            raw = np.zeros(t.buf.nbytes + shift, dtype=np.uint8)
            raw[shift:] = t.buf.view(np.uint8)
            dev.append(torch.from_numpy(raw).cuda())
            ptrs.append(dev[-1].data_ptr() + shift + t.base * t.itemsize)
        ex = simt_executor(tapp)
        assert case.run(tapp, executor=ex, A_ptr=ptrs[0], B_ptr=ptrs[1], C_ptr=ptrs[2], D_ptr=ptrs[3]) == 0
        torch.cuda.synchronize()
        tapp.lib.TAPP_destroy_executor(ex)
        got.append(dev[3].cpu().numpy()[shift:].tobytes())
    assert got[0] == got[1]
