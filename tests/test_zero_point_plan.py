"""Layout of products with zero points on the tensor cores, planned on the host."""
import ctypes

import pytest

INT_MAX = 2 ** 31 - 1
B200 = (74, 45, 33, 26, 22, 15, 15)  # clusters of 2 to 8 CTAs that run at once
SHAPES = [(16, 128, 17), (256, 4096, 24), (1024, 4096, 32), (4096, 4096, 128), (14336, 4096, 33), (28672, 256, 20), (2064, 2944, 65),
          (8192, 8192, 512), (4096, 14336, 100000)]


def plan(lib, n, k, m, gs, clusters=B200, max_split=8, sms=148):
    out = (ctypes.c_int * 7)()
    assert lib.matgptq_b200_zp_plan(gs, n, k, m, sms, (ctypes.c_int * 7)(*clusters), max_split, out) == 0
    return dict(zip(("blocks", "ncols", "tiles", "split", "accumulators", "stages", "smem"), out))


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


def test_refused(lib):
    out, clusters = (ctypes.c_int * 7)(), (ctypes.c_int * 7)(*B200)
    for args in [(64, 1024, 1024, 32, 148, clusters, 8, out), (128, 1024, 1024, 16, 148, clusters, 8, out),
                 (128, 1024, 1024, 32, 148, None, 8, out), (128, 1024, 1024, 32, 148, clusters, 9, out),
                 (128, 1024, 1024, 32, 148, (ctypes.c_int * 7)(*[0] * 7), 8, out), (128, 1024, 1024, 32, 148, clusters, 8, None)]:
        assert lib.matgptq_b200_zp_plan(*args) != 0
