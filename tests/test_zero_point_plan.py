"""Layout of products with zero points on the tensor cores, planned on the host."""
import ctypes

import pytest

INT_MAX = 2 ** 31 - 1
B200 = (74, 45, 33, 26, 22, 15, 15)  # clusters of 2 to 8 CTAs that run at once
SHAPES = [(16, 128, 17), (256, 4096, 24), (1024, 4096, 32), (4096, 4096, 128), (14336, 4096, 33), (28672, 256, 20), (2064, 2944, 65),
          (8192, 8192, 512), (4096, 14336, 100000)]


def plan(lib, n, k, m, gs, clusters=B200, max_split=8, sms=148, bits=4):
    out = (ctypes.c_int * 8)()
    assert lib.matgptq_b200_zp_plan(bits, gs, n, k, m, sms, (ctypes.c_int * 7)(*clusters), max_split, out) == 0
    return dict(zip(("path", "blocks", "ncols", "tiles", "split", "accumulators", "stages", "smem"), out))


@pytest.mark.parametrize("gs", [-1, 32, 128])
@pytest.mark.parametrize("n,k,m", SHAPES)
def test_a_device_that_cannot_tell_how_many_clusters_it_runs(lib, n, k, m, gs):
    # no limit known: the plan of a device on which every number of clusters runs at once
    unknown = plan(lib, n, k, m, gs, (INT_MAX,) * 7)
    assert unknown == plan(lib, n, k, m, gs, (2 ** 30,) * 7)
    assert unknown["split"] <= min(8, k // 128)


@pytest.mark.parametrize("gs", [-1, 32, 128])
@pytest.mark.parametrize("clusters", [B200, (INT_MAX,) * 7, (1,) * 7])
@pytest.mark.parametrize("n,k,m", SHAPES)
def test_a_plan_fits_the_kernel(lib, n, k, m, gs, clusters):
    for max_split in (1, 8):
        p = plan(lib, n, k, m, gs, clusters, max_split)
        assert p["blocks"] == -(-m // 64) and p["ncols"] % 16 == 0 and m <= p["blocks"] * p["ncols"] and p["ncols"] <= 64
        assert p["tiles"] in (4, 8, 16) and (p["tiles"] < 16 or p["ncols"] <= 32)
        assert 1 <= p["split"] <= min(max_split, k // 128)
        row_blocks, dcols = (2 if p["tiles"] == 16 else 1), -(-p["ncols"] // 32) * 32
        assert p["accumulators"] * row_blocks * dcols + p["stages"] * 64 * row_blocks <= 512  # columns of tensor memory
        assert 2 <= p["stages"] <= 6 and (p["tiles"] > 4 or p["stages"] >= 4) and p["smem"] <= 227 * 1024


GEMV, TENSOR = 1, 2


@pytest.mark.parametrize("gs,n,k,m,path", [
    (128, 4096, 4096, 16, GEMV), (128, 14336, 4096, 1, GEMV),
    # narrow layers: the passes run side by side, until they fill the device
    (128, 256, 4096, 17, GEMV), (32, 256, 4096, 128, GEMV), (128, 256, 4096, 160, TENSOR),
    (128, 1024, 4096, 17, GEMV), (32, 1024, 4096, 32, GEMV), (-1, 1024, 4096, 32, GEMV), (128, 1024, 4096, 33, TENSOR),
    (128, 1536, 1024, 32, GEMV), (128, 1536, 1024, 33, TENSOR),  # 288 CTAs of 296: clusters leave some of them over
    (128, 2048, 256, 64, GEMV), (128, 2048, 256, 96, TENSOR),
    # wide ones: two waves of passes from 17 rows on
    (128, 4096, 4096, 17, TENSOR), (128, 2048, 4096, 17, TENSOR), (32, 14336, 4096, 17, TENSOR), (128, 4096, 4096, 2 ** 24, TENSOR),
    # one scale per row: few blocks of in-features, or activations in pieces
    (-1, 4096, 256, 32, TENSOR), (128, 4096, 256, 32, GEMV), (-1, 512, 14336, 32, TENSOR), (128, 512, 14336, 32, GEMV)])
def test_path(lib, gs, n, k, m, path):
    assert plan(lib, n, k, m, gs)["path"] == path
    if m > 16:
        assert plan(lib, n, k, m, gs, sms=1)["path"] == TENSOR  # nothing runs side by side there


@pytest.mark.parametrize("bits", [2, 3, 4, 6, 8])
@pytest.mark.parametrize("gs", [-1, 32, 128])
def test_path_changes_once_as_the_batch_grows(lib, bits, gs):
    for n in (16, 272, 1024, 4096, 28672):
        for k in (128, 1024, 4096, 14336, 53248):
            paths = [plan(lib, n, k, m, gs, bits=bits)["path"] for m in (1, 16, 17, 32, 33, 64, 100, 300, 1000, 5000, 40000)]
            assert paths[:2] == [GEMV, GEMV] and paths == sorted(paths) and paths[-1] == TENSOR, (n, k, paths)


def test_refused(lib):
    out, clusters = (ctypes.c_int * 7)(), (ctypes.c_int * 7)(*B200)
    for args in [(5, 128, 1024, 1024, 32, 148, clusters, 8, out), (4, 64, 1024, 1024, 32, 148, clusters, 8, out), (4, 128, 1024, 1024, 0, 148, clusters, 8, out),
                 (4, 128, 1024, 1024, 32, 148, None, 8, out), (4, 128, 1024, 1024, 32, 148, clusters, 9, out),
                 (4, 128, 1024, 1024, 32, 148, (ctypes.c_int * 7)(*[0] * 7), 8, out), (4, 128, 1024, 1024, 32, 148, clusters, 8, None)]:
        assert lib.matgptq_b200_zp_plan(*args) != 0
