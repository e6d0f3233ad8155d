"""Dense mat-mat (csrc/qmm.cu) where CTAs share tiles along K and where tiles have any multiple of 16 rows, and the routed form with two
CTAs per SM on rows that do not start on 16-byte boundaries, against the oracle."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import TYPES, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
TOL = 2e-5   # against f16 operands: only the order of the f32 sums differs


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


# With 148 SMs: more tiles than SMs in ranges that cut tiles (rows that do and do not start on 16-byte boundaries, K tails of 32 to 160
# values, n that is no multiple of the rows of a copy), tiles in halves (K of eight raw stages and more, an odd number of them), whole
# tiles (short K), and row counts at the edges of 16-row steps and of the 64-, 128- and 256-row kernels.
@pytest.mark.parametrize("tname,m,n,k", [
    ("Q8_0", 9, 19100, 2080), ("Q4_0", 70, 19000, 2400), ("Q8_0", 130, 19100, 1600), ("Q4_0", 300, 9729, 2208), ("Q6_K", 40, 19073, 4096),
    ("Q6_K", 33, 19074, 512), ("Q4_0", 16, 200, 2048), ("Q8_0", 17, 130, 2080), ("Q6_K", 65, 300, 2304), ("Q4_0", 81, 257, 2176),
    ("Q6_K", 129, 128, 4096), ("Q8_0", 145, 500, 2304), ("Q4_0", 333, 384, 2048), ("Q6_K", 241, 136, 2048), ("Q4_0", 256, 100, 256),
    ("Q8_0", 257, 640, 1024), ("Q4_0", 520, 300, 512), ("Q6_K", 1025, 256, 768), ("Q6_K", 257, 4096, 768), ("Q8_0", 600, 6400, 1056)])
def test_tiles(ctx, tname, m, n, k):
    gtype, otype = TYPES[tname]
    wq = normal_weights(n + k + m, n, k, otype)
    x = normal_acts(n + m, m, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmm_tc"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, f16_operands=True, nthreads=8)
    assert norm_err(y, y_ref, ad) <= TOL
    assert np.array_equal(y.view(np.uint32), ctx.matmul(gtype, wq, x, n, k).view(np.uint32))   # two addends: the order does not matter


# rows of 630, 1890, 162, 522, 340 and 1088 bytes: groups of 8, 8, 8, 8, 4 and 1; n that is no multiple of the group takes the other copies
@pytest.mark.parametrize("tname,T,top_k,E,n,k", [
    ("Q6_K", 40, 8, 16, 264, 768), ("Q6_K", 100, 2, 4, 130, 2304), ("Q4_0", 64, 8, 8, 136, 288), ("Q4_0", 33, 2, 3, 128, 928),
    ("Q8_0", 200, 1, 5, 132, 320), ("Q8_0", 37, 8, 128, 256, 1024)])
def test_routed(ctx, tname, T, top_k, E, n, k):
    gtype, otype = TYPES[tname]
    w = normal_weights(E + n, E * n, k, otype)
    x = normal_acts(T, T, k)
    rng = np.random.default_rng(T + n)
    ids = np.stack([rng.permutation(E)[:top_k] for _ in range(T)]).astype(np.uint32).reshape(-1)
    y, _ = ctx.matmul_id(gtype, w, w.size // E, x, ids, top_k, n, k, E)
    assert mx.last_kernel_name() == "qmm_tc_id"
    y_ref, ad = orc.qmatmul_id(otype, w, w.size // E, x, ids, top_k, n, k, E, f16_operands=True, nthreads=8)
    assert norm_err(y, y_ref, ad) <= TOL
