"""Which CUDA-core kernel a product runs, as tapp_b200_describe_plan reports
it (no GPU): the rules of the element path and of the tiled GEMM, at sizes on
both sides of their lines.
"""
import re

import pytest

import tapp_b200
from tapp_b200.abi import TAPP_F32, TAPP_F64, TAPP_C32, TAPP_C64, TAPP_F16, TAPP_BF16


def plan_text(tapp, a, b, d, ext, types, prec, path=0):
    """The plan of D[d] = sum A[a] B[b] + C[d], one letter per mode, dense column-major; types of A, B, C, D"""
    infos = []
    for labels, t in zip((a, b, d, d), types):
        strides, at = [], 1
        for x in labels:
            strides.append(at)
            at *= ext[x]
        infos.append(tapp.tensor_info(t, [ext[x] for x in labels], strides)[1])
    err, plan = tapp.create_product(0, [0] * 4, infos, [[ord(x) for x in labels] for labels in (a, b, d, d)], prec)
    assert err == 0
    ex = tapp.create_executor()
    if path:
        tapp.set_int(ex, tapp_b200.ATTR_PATH, path)
    text = tapp.describe(plan, ex)
    tapp.lib.TAPP_destroy_executor(ex)
    tapp.lib.TAPP_destroy_tensor_product(plan)
    for h in infos:
        tapp.lib.TAPP_destroy_tensor_info(h)
    return text


def field(text, name):
    m = re.search(rf" {name}=(\S+)", text)
    return m and m[1]


# operands stored as computed, rounded or not, and 16-bit operands of either kind are loaded in groups; what is converted
# behind a switch is taken one output at a time, threads and warps alike
@pytest.mark.parametrize("types,prec,grouped", [
    ((TAPP_F32,) * 4, 0, True), ((TAPP_F32,) * 4, 6, True), ((TAPP_F16,) * 4, 5, True), ((TAPP_F16,) * 4, -1, True),
    ((TAPP_BF16, TAPP_F16, TAPP_F32, TAPP_F32), -1, True), ((TAPP_F64,) * 4, -1, True), ((TAPP_C32,) * 4, 6, True),
    ((TAPP_C64,) * 4, -1, True), ((TAPP_F32, TAPP_BF16, TAPP_F32, TAPP_F32), -1, False),
    ((TAPP_F64, TAPP_F64, TAPP_F32, TAPP_F32), 0, False), ((TAPP_F32, TAPP_F32, TAPP_F32, TAPP_F32), 1, False),
    ((TAPP_F16, TAPP_F16, TAPP_C32, TAPP_C32), -1, False), ((TAPP_C64, TAPP_C32, TAPP_C64, TAPP_C64), -1, False)])
def test_element_operands_loaded_in_groups(tapp, types, prec, grouped):
    ext = {"a": 500, "b": 401, "d": 9, "k": 5}
    t = plan_text(tapp, "abkd", "bka", "dab", ext, types, prec)
    assert field(t, "kernel") == "element" and field(t, "rows") == ("8" if grouped else "0"), t
    ext = {"a": 40, "b": 51, "d": 9, "k": 70}
    t = plan_text(tapp, "kabd", "kab", "dab", ext, types, prec)
    assert field(t, "kernel") == "warpdot" and field(t, "rows") == ("8" if grouped else "0"), t


# a single term is not worth filling offset tables for, unless outputs share loads of an operand
@pytest.mark.parametrize("a,b,ext,types,prec,rows", [
    ("abd", "ba", {"a": 78, "b": 25, "d": 19}, (TAPP_F32,) * 4, 0, "0"),
    ("abd", "ba", {"a": 780, "b": 250, "d": 19}, (TAPP_F32,) * 4, 0, "8"),
    ("abd", "ba", {"a": 780, "b": 250, "d": 19}, (TAPP_C32,) * 4, -1, "8"),
    ("abd", "ba", {"a": 780, "b": 250, "d": 19}, (TAPP_C32,) * 4, 6, "0"),
    ("abdk", "ba", {"a": 78, "b": 25, "d": 19, "k": 3}, (TAPP_F32,) * 4, 0, "1"),
    ("abdk", "bak", {"a": 78, "b": 25, "d": 19, "k": 2}, (TAPP_F32,) * 4, 0, "1")])
def test_one_term_takes_one_output_at_a_time(tapp, a, b, ext, types, prec, rows):
    t = plan_text(tapp, a, b, "abd", ext, types, prec)
    assert field(t, "kernel") == "element" and field(t, "rows") == rows, t


# groups that the mode fills no more than half are not formed
@pytest.mark.parametrize("d,k,types,rows", [
    (4, 3, (TAPP_F32,) * 4, "4"), (5, 3, (TAPP_F32,) * 4, "8"), (4, 3, (TAPP_F64,) * 4, "4"), (3, 3, (TAPP_F64,) * 4, "4"),
    (2, 3, (TAPP_F64,) * 4, "1"), (2, 3, (TAPP_F32,) * 4, "1"), (2, 3, (TAPP_BF16,) * 4, "1"),
    (2, 1, (TAPP_F32,) * 4, "0"), (3, 1, (TAPP_F32,) * 4, "4")])
def test_rows_fill_more_than_half_a_group(tapp, d, k, types, rows):
    t = plan_text(tapp, "abkd", "bka", "abd", {"a": 500, "b": 401, "d": d, "k": k}, types, -1)
    assert field(t, "kernel") == "element" and field(t, "rows") == rows, t


# unary modes beyond the offset tables are summed for one output a warp, in k_warpdot where each value is converted; and so
# are contiguous ones whose runs fill lines
@pytest.mark.parametrize("a,types,prec,u,v,rows", [
    ("ahku", (TAPP_F32,) * 4, 0, 128, 128, "8"), ("ahku", (TAPP_F32,) * 4, 0, 129, 3, "1"), ("ahku", (TAPP_F32,) * 4, 0, 3, 129, "1"),
    ("ahku", (TAPP_C64,) * 4, -1, 129, 3, "1"), ("ahku", (TAPP_F32,) * 4, 6, 129, 3, "0"), ("ahku", (TAPP_F16,) * 4, -1, 129, 3, "0"),
    ("ahku", (TAPP_F16,) * 4, -1, 128, 3, "8"), ("uahk", (TAPP_F32,) * 4, 0, 15, 3, "8"), ("uahk", (TAPP_F32,) * 4, 0, 16, 3, "1"),
    ("uahk", (TAPP_C32,) * 4, -1, 8, 3, "1"), ("uahk", (TAPP_F16,) * 4, -1, 31, 3, "8"), ("uahk", (TAPP_F16,) * 4, -1, 32, 3, "1")])
def test_long_unary_modes_take_one_row(tapp, a, types, prec, u, v, rows):
    t = plan_text(tapp, a, "khv", "ah", {"a": 150, "h": 120, "k": 33, "u": u, "v": v}, types, prec)
    assert field(t, "kernel") == "warpdot" and field(t, "rows") == rows, t


# up to 8 columns stay with the narrow kernels once their rows fill the GPU, from 9 columns the line rises with them
@pytest.mark.parametrize("t,prec,m,n,k,kernel", [
    (TAPP_F32, 0, 57771, 6, 100, "narrow"), (TAPP_F32, 6, 57771, 1, 300, "narrow"), (TAPP_F32, 0, 50001, 9, 100, "tiled"),
    (TAPP_F32, 0, 57771, 20, 100, "tiled"), (TAPP_F32, 0, 37001, 6, 100, "tiled"), (TAPP_F32, 0, 100001, 9, 100, "narrow"),
    (TAPP_F32, 0, 100001, 16, 100, "narrow"), (TAPP_F32, 0, 90001, 16, 100, "tiled"), (TAPP_F32, 0, 120001, 16, 100, "tiled"), (TAPP_F32, 0, 155001, 30, 100, "narrow"), (TAPP_F32, 0, 57771, 20, 64, "narrow"),
    (TAPP_C32, -1, 22347, 2, 245, "narrow"), (TAPP_C32, -1, 9001, 2, 245, "tiled"), (TAPP_C32, -1, 22347, 9, 245, "tiled"),
    (TAPP_C32, -1, 278581, 12, 138, "narrow"), (TAPP_C32, -1, 278581, 13, 138, "tiled"),
    (TAPP_F64, -1, 285869, 4, 117, "narrow"), (TAPP_F64, -1, 285869, 4, 222, "tiled"), (TAPP_F64, -1, 20001, 4, 117, "tiled"),
    (TAPP_F64, -1, 285869, 9, 117, "tiled")])
def test_narrow_kernels_keep_few_columns(tapp, t, prec, m, n, k, kernel):
    text = plan_text(tapp, "mk", "nk", "mn", {"m": m, "n": n, "k": k}, (t,) * 4, prec)
    got = field(text, "kernel")
    assert got == kernel or (kernel == "narrow" and got.startswith("narrow")), text
    assert (field(text, "tile") is not None) == (kernel == "tiled"), text


# tall tiles need rows for several warps an SM, and there are none where general ones do better
@pytest.mark.parametrize("t,m,n,tile", [
    (TAPP_F32, 57771, 12, "128x16"), (TAPP_F32, 230000, 12, "256x12"), (TAPP_F32, 100001, 20, "128x32"),
    (TAPP_F32, 120001, 20, "256x24"), (TAPP_F32, 50001, 33, "64x64"), (TAPP_F32, 70001, 33, "256x36"),
    (TAPP_F32, 50001, 40, "256x40"), (TAPP_F32, 60001, 48, "256x48"), (TAPP_F32, 500001, 50, "64x64"),
    (TAPP_F32, 500001, 60, "64x64"), (TAPP_F32, 40001, 64, "64x64"), (TAPP_F32, 60001, 64, "256x64"),
    (TAPP_C32, 30001, 8, "128x32"), (TAPP_C32, 40001, 8, "128x8"), (TAPP_C32, 20001, 16, "128x32"), (TAPP_C32, 30001, 16, "128x16"),
    (TAPP_C32, 100001, 24, "128x32"), (TAPP_C32, 160001, 24, "128x24"), (TAPP_C32, 500001, 25, "128x32"),
    (TAPP_C32, 500001, 40, "64x64"), (TAPP_C32, 500001, 45, "64x64")])
def test_tall_tiles_need_rows(tapp, t, m, n, tile):
    # a contraction beyond what the narrow kernels hold
    text = plan_text(tapp, "mk", "nk", "mn", {"m": m, "n": n, "k": 5000}, (t,) * 4, -1)
    assert (field(text, "kernel"), field(text, "tile")) == ("tiled", tile), text


# few tiles and a long contraction: splits through the workspace once 8 ranks of a cluster would walk some 10 slices each
@pytest.mark.parametrize("t,m,n,k,through_workspace", [
    (TAPP_C64, 384, 14, 1811, True), (TAPP_C64, 384, 14, 1025, True), (TAPP_C64, 384, 14, 1024, False),
    (TAPP_C32, 136, 38, 1903, True), (TAPP_C32, 136, 38, 1280, False), (TAPP_F64, 56, 91, 1400, True),
    (TAPP_F64, 56, 91, 1280, False), (TAPP_F32, 108, 37, 1420, True), (TAPP_F32, 108, 37, 1400, False), (TAPP_F32, 2048, 33, 1660, False)])
def test_long_contractions_of_few_tiles_are_split(tapp, t, m, n, k, through_workspace):
    text = plan_text(tapp, "mk", "nk", "mn", {"m": m, "n": n, "k": k}, (t,) * 4, -1, path=tapp_b200.PATH_SIMT)
    assert field(text, "kernel") == "tiled", text
    assert (int(field(text, "splits")) > 8, int(field(text, "cluster"))) == (through_workspace, 1 if through_workspace else 8), text


# from one to one and a half tiles per SM, long contractions are shared by two ranks
@pytest.mark.parametrize("t,l,k,cluster", [(TAPP_F32, 40, 900, 2), (TAPP_F32, 40, 512, 1), (TAPP_F32, 55, 900, 2), (TAPP_F32, 56, 900, 1),
                                           (TAPP_F64, 80, 900, 2), (TAPP_C64, 40, 900, 2)])
def test_little_more_than_a_tile_per_sm(tapp, t, l, k, cluster):
    text = plan_text(tapp, "mkl", "nkl", "mnl", {"m": 106, "n": 86, "k": k, "l": l}, (t,) * 4, -1)
    assert field(text, "kernel") == "tiled" and int(field(text, "cluster")) == cluster, text


# binary32 tiles of 128 x 128 also for fewer tiles where the contraction is long or an operand lies along it; both operands
# in 16-byte runs along a long contraction go to the kernel that loads runs (no tile)
@pytest.mark.parametrize("a,b,m,n,k,tile", [
    ("mk", "nk", 634, 480, 2832, "128x128"), ("mk", "nk", 634, 480, 1100, "128x128"), ("mk", "nk", 634, 480, 900, "64x64"),
    ("mk", "nk", 200, 180, 2832, "64x64"), ("mk", "nk", 634, 60, 2832, "64x64"), ("mk", "nk", 2000, 2000, 100, "128x128"),
    ("mk", "nk", 1500, 1400, 1100, "64x64"), ("km", "nk", 1500, 1400, 1100, "128x128"), ("mk", "kn", 1500, 1400, 1000, "64x64"),
    ("km", "kn", 634, 480, 512, "128x128"), ("km", "kn", 634, 480, 508, "64x64"), ("km", "kn", 300, 200, 600, "64x64"),
    ("km", "kn", 634, 480, 1536, None), ("km", "kn", 634, 480, 1537, "128x128"), ("km", "kn", 634, 480, 1532, "128x128"),
    ("km", "kn", 300, 200, 2048, None), ("km", "kn", 200, 200, 2048, "64x64"), ("km", "kn", 2000, 2000, 2048, "128x128")])
def test_wide_tiles_for_fewer_tiles(tapp, a, b, m, n, k, tile):
    text = plan_text(tapp, a, b, "mn", {"m": m, "n": n, "k": k}, (TAPP_F32,) * 4, 0, path=tapp_b200.PATH_SIMT)
    assert field(text, "tile") == tile, text
