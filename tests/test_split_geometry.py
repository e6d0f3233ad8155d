"""The sizes that the split mat-vec (csrc/qmv_split.cuh) promises to take all have a geometry (host logic, no GPU)."""
import ctypes as C

import pytest

import mlx_native_b200 as mx
from mlx_native_b200 import _native

SMS = 148


def geometry(gtype, rows, k, n=4096, experts=0, misaligned=0):
    p = _native.QmmIdParams(rows, 1, n, k, experts, int(gtype), n * (k // gtype.block_values()) * gtype.block_bytes())
    ranks, tiles = C.c_uint32(), C.c_uint32()
    assert _native.lib().mlxn_debug_split_geometry(C.byref(p), misaligned, SMS, C.byref(ranks), C.byref(tiles)) == 0
    return ranks.value, tiles.value


# the largest K by activation rows; the kernels that take what is beyond are chosen by the same answer
@pytest.mark.parametrize("tname", ["Q4_0", "Q8_0", "Q6_K", "Q4_K"])
@pytest.mark.parametrize("rows,limit", [(1, 133120), (2, 65536), (3, 30720), (4, 30720), (5, 14336), (8, 14336)])
@pytest.mark.parametrize("misaligned", [0, 2])
def test_every_k_up_to_the_limit_has_a_geometry(tname, rows, limit, misaligned):
    gtype = mx.GgmlType[tname]
    qk = gtype.block_values()
    if tname == "Q4_K" and misaligned:
        assert geometry(gtype, rows, 4096, misaligned=misaligned) == (0, 0)
        return
    for k in range(qk, min(limit, 32768) + 1, qk):
        ranks, tiles = geometry(gtype, rows, k, misaligned=misaligned)
        assert ranks in (1, 2, 4, 8) and 1 <= tiles <= 4, (k, ranks, tiles)
    assert geometry(gtype, rows, limit // 256 * 256, misaligned=misaligned)[0] > 0
    assert geometry(gtype, rows, limit // 256 * 256 + 256, misaligned=misaligned) == (0, 0)


@pytest.mark.parametrize("tname", ["Q4_0", "Q8_0", "Q6_K", "Q4_K", "Q5_K"])
@pytest.mark.parametrize("pairs,limit", [(1, 16640), (2, 3840), (17, 3840), (256, 3840)])
def test_every_routed_k_up_to_the_limit_has_a_geometry(tname, pairs, limit):
    gtype = mx.GgmlType[tname]
    qk = gtype.block_values()
    for k in range(qk, limit // qk * qk + 1, qk):
        ranks, tiles = geometry(gtype, pairs, k, n=768, experts=16)
        assert ranks == 1 and 1 <= tiles <= 4, k
    assert geometry(gtype, pairs, limit // 256 * 256 + 256, n=768, experts=16) == (0, 0)
    assert geometry(gtype, 257, 2048, n=768, experts=16) == (0, 0)


# One, two and four rows: what was measured as the fastest geometry, or within 5 percent of it.  (The choice once went by a model of four shapes: Q8_0 10240 x 4096 over clusters
# of four took 16.9 us, on one CTA each 11.9, and 13.0 before the kernel had integers.)
@pytest.mark.parametrize("tname,rows,n,k,good", [
    ("Q8_0", 1, 10240, 4096, [(1, 3)]), ("Q6_K", 1, 10240, 4096, [(1, 3)]), ("Q4_0", 2, 10240, 4096, [(2, 4), (2, 3)]), ("Q4_0", 2, 12288, 4096, [(2, 3), (2, 4)]),
    ("Q6_K", 2, 14336, 4096, [(2, 4)]), ("Q8_0", 2, 14336, 4096, [(2, 4)]), ("Q4_K", 2, 10240, 4096, [(2, 3)]), ("Q4_0", 2, 8192, 12288, [(8, 4)]),
    ("Q6_K", 2, 4096, 12288, [(8, 4), (4, 4)]), ("Q4_K", 1, 11264, 4096, [(1, 3)]),
    ("Q4_0", 4, 6144, 4096, [(2, 3)]), ("Q8_0", 4, 12288, 4096, [(2, 3), (4, 4)]), ("Q8_0", 4, 8192, 5120, [(2, 2)]), ("Q4_K", 4, 4096, 8192, [(4, 2), (4, 3)])])
def test_geometry_of_few_rows(tname, rows, n, k, good):
    assert geometry(mx.GgmlType[tname], rows, k, n=n) in good
