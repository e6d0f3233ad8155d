"""Mat-mats on pairs of SMs whose weight rows lie in tensor memory as in a raw stage (csrc/qmm_duo.cu: Q6_K rows off 16-byte boundaries), and Q4_K by
16-byte loads, against the f16-operand oracle."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MM_TOL, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


# every other row on a boundary (K = 1024, 3072: 840 and 2520 bytes), every fourth (512: 420) and eighth (256: 210); a last tile of rows that is part-filled;
# enough tiles that none is shared by two pairs, and few
@pytest.mark.parametrize("n,k,m", [(10238, 1024, 40), (10240, 1024, 33), (1030, 3072, 70), (10240, 512, 40), (520, 512, 300), (528, 256, 65)])
def test_dense(ctx, n, k, m):
    wq = normal_weights(n + k, n, k, orc.Q6_K)
    x = normal_acts(m, m, k)
    y = ctx.matmul(mx.GgmlType.Q6_K, wq, x, n, k)
    assert mx.last_mat_mat()[0] == "qmm_duo"
    rows = np.unique(np.concatenate([np.arange(48), np.arange(n - 48, n), np.arange(n // 2, n // 2 + 32)]))
    w = orc.dequantize(orc.Q6_K, wq).reshape(n, k)[rows].astype(np.float64)
    ref, ad = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    assert norm_err(y[:, rows], ref, ad) <= MM_TOL


@pytest.mark.parametrize("tname,n,k", [("Q6_K", 258, 1024), ("Q6_K", 260, 512), ("Q6_K", 264, 768), ("Q6_K", 136, 2048), ("Q4_K", 130, 768)])
def test_routed(ctx, tname, n, k):
    T, top_k, E = 70, 8, 12
    gtype, otype = (mx.GgmlType.Q6_K, orc.Q6_K) if tname == "Q6_K" else (mx.GgmlType.Q4_K, orc.Q4_K)
    w = normal_weights(n, E * n, k, otype)
    x = normal_acts(k, T, k)
    rng = np.random.default_rng(n)
    ids = np.concatenate([rng.permutation(E)[:top_k] for _ in range(T)]).astype(np.uint32)
    y, _ = ctx.matmul_id(gtype, w, w.size // E, x, ids, top_k, n, k, E)
    assert mx.last_mat_mat()[0] == "qmm_duo_id"
    y_ref, ad = orc.qmatmul_id(otype, w, w.size // E, x, ids, top_k, n, k, E, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MM_TOL
