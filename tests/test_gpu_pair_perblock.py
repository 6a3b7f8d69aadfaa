"""GPU: the per-block kernel on CTA pairs where its scale ring (runs of four k-blocks, two buffers) and its row stores begin and end."""
import ml_dtypes
import numpy as np
import pytest

from conftest import case_seed
from oracle import qbmm_oracle
from test_gpu_umma import E4M3, _fp8, _run

pytestmark = pytest.mark.gpu

CASES = [
    # batch, m, k, n, t1, t2, group_m, int8, bias, out
    (0, 256, 128, 256, False, True, 1, False, False, "bfloat16"),      # one k-block
    (0, 300, 640, 512, False, False, 1, False, False, "float16"),      # a run and one k-block; scalar scale loads; ragged rows
    (0, 2304, 384, 2560, False, True, 1, False, False, "bfloat16"),    # several tiles a pair: the ring runs on from tile to tile
    (0, 700, 1536, 1288, False, True, 1, False, False, "float32"),      # vector scale loads; last tile stored row by row
    (0, 512, 1152, 1301, True, True, 128, False, False, "bfloat16"),   # rows of odd length: no 16-byte pieces anywhere
    (3, 260, 512, 384, False, False, 1, False, False, "bfloat16"),     # batches, 384 = one and a half tiles
    (0, 520, 1152, 768, False, True, 1, True, True, "bfloat16"),       # int8: bit-exact
]


@pytest.mark.parametrize("tile_n", ["128", "256"])
@pytest.mark.parametrize("case", CASES, ids=[str(c) for c in CASES])
def test_scale_runs_and_row_stores(aclnn, case, tile_n, monkeypatch):
    """fp8: within the other per-block kernels' tolerance (fp32 summation order inside a k-block); int8 bit for bit."""
    from gpu_util import check_close

    batch, m, k, n, t1, t2, gm, is_int, has_bias, out_name = case
    rng = np.random.default_rng(case_seed(case))
    lead = (batch,) if batch else ()
    kb, mg, ng = -(-k // 128), -(-m // gm), -(-n // 128)
    sh1, sh2 = lead + ((k, m) if t1 else (m, k)), lead + ((n, k) if t2 else (k, n))
    if is_int:
        x1, x2 = rng.integers(-127, 128, sh1, dtype=np.int8), rng.integers(-127, 128, sh2, dtype=np.int8)
        lo = (1e-3, 1e-2)
    else:
        x1, x2 = _fp8(rng, sh1, E4M3), _fp8(rng, sh2, E4M3)
        lo = (0.5, 2)
    s1 = rng.uniform(*lo, lead + ((kb, mg) if t1 else (mg, kb))).astype(np.float32)
    s2 = rng.uniform(*lo, lead + ((ng, kb) if t2 else (kb, ng))).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32) if has_bias else None
    group = (gm << 32) | (128 << 16) | 128
    monkeypatch.setenv("OPSNN_QMM_PAIR", "1")
    monkeypatch.setenv("OPSNN_QMM_PB_BN", tile_n)
    got = _run(aclnn, x1, x2, s1, s2, bias, t1, t2, group, out_name, "qmm_umma_pair_perblock")
    pick = (lambda a, i: a[i]) if batch else (lambda a, i: a)
    for i in range(batch or 1):
        args = [pick(a, i) for a in (x1, x2, s1, s2)]
        want = qbmm_oracle.quant_matmul_v5(*args, bias, t1, t2, group, out_name)
        g = pick(got, i)
        if is_int:
            assert np.array_equal(g.view(np.uint16), want.view(np.uint16))
        else:
            check_close(g, want, qbmm_oracle.quant_matmul_v5(*args, None, t1, t2, group, "float32"), out_name)
    assert np_finite(got)


def np_finite(a):
    return bool(np.all(np.isfinite(a.astype(np.float32) if a.dtype == ml_dtypes.bfloat16 else a)))
