"""GPU: the split kernel of the dequant and per-block modes (weight columns as the MMA's M, k cut into pieces) against the oracle, at the
sizes where its tiles, pieces and ways of combining them begin and end. int8 sums are exact, so those outputs are bit-exact; fp8 differs by
fp32 summation order."""
import ml_dtypes
import numpy as np
import pytest

from conftest import case_seed
from oracle import qbmm_oracle

pytestmark = pytest.mark.gpu

E4M3, E5M2 = ml_dtypes.float8_e4m3fn, ml_dtypes.float8_e5m2

CASES = [
    # mode, batch, m, k, n, x2 stored (n,k), bias, out
    ("int8", (), 1, 4096, 256, True, "i32", "bfloat16"),       # one or two tiles, a piece per CTA of a cluster
    ("int8", (), 17, 2064, 2064, False, "f32", "bfloat16"),    # ragged k and n, x2 along n
    ("int8", (), 64, 512, 22000, True, None, "float16"),       # few k-blocks: a tile a CTA
    ("int8", (), 130, 4112, 272, True, "i32", "bfloat16"),     # two row tiles, few columns
    ("int8", (2,), 33, 1040, 656, True, None, "bfloat16"),     # batched
    ("fp8", (), 16, 6144, 1040, False, "f32", "float16"),
    ("fp8", (), 250, 2048, 528, True, None, "float32"),
    ("e5m2", (), 40, 1072, 20000, True, "f32", "bfloat16"),
    ("block", (), 1, 7168, 400, True, None, "bfloat16"),
    ("block", (), 48, 1152, 20096, False, None, "float16"),    # per-block, a tile a CTA
    ("block", (), 100, 3072, 640, True, None, "float32"),
    ("block", (3,), 20, 1088, 320, True, None, "bfloat16"),    # last k-block half full
    # a cluster's sums sent to their owners: rows that fours and owners do not divide, fewer fours than owners, one to four fours a thread
    ("fp8", (), 5, 1472, 1296, False, "f32", "float32"),
    ("int8", (), 30, 4096, 3088, True, "f32", "bfloat16"),
    # (bf16: these outputs are 1e-3 and less, and half a unit of fp16's subnormals, 3e-8, is 2 % of check_close's floor of 1.5e-6)
    ("fp8", (), 61, 2048, 4112, False, None, "bfloat16"),
    ("fp8", (), 64, 4096, 3072, True, "f32", "bfloat16"),
    ("int8", (), 83, 4096, 3072, True, "i32", "bfloat16"),
    ("int8", (2,), 21, 3072, 400, False, None, "bfloat16"),
    # more tiles of either shape than SMs: pieces across tiles, summed through workspace
    ("int8", (), 64, 384, 40960, True, "i32", "float16"),
    ("fp8", (), 20, 1040, 38416, True, "f32", "bfloat16"),
    ("block", (), 33, 640, 38416, True, None, "bfloat16"),
]


@pytest.mark.parametrize("case", CASES, ids=[str(c) for c in CASES])
def test_split_kernel_equals_oracle(aclnn, monkeypatch, case):
    monkeypatch.setenv("OPSNN_QMM_SPLIT", "1")
    _against_oracle(aclnn, case)


@pytest.mark.parametrize("halves", ["1", "2"])
@pytest.mark.parametrize("nk", [False, True])
@pytest.mark.parametrize("m,k,n", [(9, 4224, 1168), (50, 2176, 1296), (127, 1216, 400)])
def test_per_block_instances(aclnn, monkeypatch, m, k, n, nk, halves):
    """The instances of the per-block form: x2 in either order, 256 and 128 columns a tile, 32 and 64 sums a thread."""
    monkeypatch.setenv("OPSNN_QMM_SPLIT", "1")
    monkeypatch.setenv("OPSNN_QMM_SPLIT_HALVES", halves)
    _against_oracle(aclnn, ("block", (), m, k, n, nk, None, "bfloat16"))


@pytest.mark.parametrize("case", [
    # mode, batch, m, k, n, x2 stored (n,k), bias, out
    ("fp8", (), 5, 1472, 1296, False, "f32", "float32"),
    ("int8", (), 30, 4096, 3088, True, "f32", "bfloat16"),
    ("int8", (), 83, 4096, 3072, True, "i32", "bfloat16"),
    ("int8", (2,), 21, 3072, 400, False, None, "bfloat16"),
    ("int8", (), 128, 4096, 4096, True, None, "bfloat16"),
    ("fp8", (), 250, 2048, 528, True, None, "float32"),
    ("int8", (), 130, 4112, 272, True, "i32", "bfloat16"),
], ids=str)
@pytest.mark.parametrize("halves", ["1", "2"])
def test_sums_of_a_cluster_sent_or_fetched(aclnn, monkeypatch, case, halves):
    """Either way of bringing the pieces of a tile together, at shares that the host would and would not send: the same additions, the same bits."""
    monkeypatch.setenv("OPSNN_QMM_SPLIT", "1")
    monkeypatch.setenv("OPSNN_QMM_SPLIT_HALVES", halves)
    outs = []
    for push in ("0", "1"):
        monkeypatch.setenv("OPSNN_QMM_SPLIT_PUSH", push)
        outs.append(_against_oracle(aclnn, case))
    assert np.array_equal(outs[0].view(np.uint8), outs[1].view(np.uint8))


def _against_oracle(aclnn, case):
    import torch

    from gpu_util import check_close, desc, out_tensor, out_to_np

    mode, batch, m, k, n, nk, bias_kind, out_name = case
    rng = np.random.default_rng(case_seed(case))
    if mode == "int8":
        x1 = rng.integers(-127, 128, batch + (m, k), dtype=np.int8)
        x2 = rng.integers(-127, 128, batch + ((n, k) if nk else (k, n)), dtype=np.int8)
    else:
        dt = E5M2 if mode == "e5m2" else E4M3
        x1 = rng.standard_normal(batch + (m, k)).astype(np.float32).astype(E4M3)
        x2 = rng.standard_normal(batch + ((n, k) if nk else (k, n))).astype(np.float32).astype(dt)
    group = 0
    if mode == "block":
        kb, ng = -(-k // 128), -(-n // 128)
        s1 = rng.uniform(0.5, 2, batch + (m, kb)).astype(np.float32)
        s2 = rng.uniform(0.5, 2, batch + ((ng, kb) if nk else (kb, ng))).astype(np.float32)
        group = (1 << 32) | (128 << 16) | 128
    else:
        s1 = rng.uniform(1e-3, 1e-2, m).astype(np.float32) if not batch else None
        s2 = rng.uniform(1e-3, 1e-2, n).astype(np.float32)
    bias = {None: None, "i32": rng.integers(-1000, 1001, n).astype(np.int32), "f32": rng.uniform(-1, 1, n).astype(np.float32)}[bias_kind]
    want = qbmm_oracle.quant_matmul_v5(x1, x2, s1, s2, bias, False, nk, group, out_name)
    outs = []
    for _ in range(2):  # twice: the second call finds the workspace as the first left it
        out = out_tensor(batch + (m, n), out_name)
        aclnn.quant_matmul_v5(desc(aclnn, x1), desc(aclnn, x2), desc(aclnn, s1), desc(aclnn, s2), aclnn.Tensor(out.shape, out_name, out), desc(aclnn, bias),
                              False, nk, group)
        torch.cuda.synchronize()
        outs.append(out_to_np(out))
    assert aclnn.last_kernel_name() == ("qmm_umma_split_perblock" if mode == "block" else "qmm_umma_split_deq"), aclnn.last_kernel_name()
    assert np.array_equal(outs[0].view(np.uint8), outs[1].view(np.uint8))
    if mode == "int8":
        assert np.array_equal(outs[0].view(np.uint8), np.asarray(want).view(np.uint8))
    else:
        check_close(outs[0], want, qbmm_oracle.quant_matmul_v5(x1, x2, s1, s2, bias, False, nk, group, "float32"), out_name)
    return outs[0]


@pytest.mark.parametrize("mode,m,k,n,push", [("int8", 128, 4096, 4096, None),   # a cluster of pieces, their sums fetched
                                             ("int8", 64, 1024, 40960, None),   # more tiles than SMs: pieces across tiles
                                             ("block", 24, 7168, 400, None),     # per-block, pieces across tiles
                                             ("block", 24, 2048, 9216, None),    # a cluster
                                             ("int8", 64, 4096, 3072, "1"),      # a cluster's sums sent: two and sixteen pieces a tile
                                             ("int8", 21, 4096, 512, "1")])
def test_wait_that_runs_out_ends_the_call(aclnn, monkeypatch, mode, m, k, n, push):
    """The producer stops after its first k-block: every wait behind it runs out, all CTAs of a cluster still meet, nothing is written, later
    calls are refused until the condition is cleared, and then find tensor memory and workspace as they should."""
    import torch

    from gpu_util import DEV

    monkeypatch.setenv("OPSNN_QMM_SPLIT", "1")
    if push is not None:
        monkeypatch.setenv("OPSNN_QMM_SPLIT_PUSH", push)
    gen = torch.Generator(device=DEV).manual_seed(6)
    if mode == "int8":
        x, w = (torch.randint(-127, 128, s, generator=gen, device=DEV, dtype=torch.int8) for s in ((m, k), (n, k)))
        s1, s2 = (torch.rand(c, generator=gen, device=DEV) * 1e-2 for c in (m, n))
        group = 0
    else:
        x, w = (torch.randn(s, generator=gen, device=DEV).to(torch.float8_e4m3fn) for s in ((m, k), (n, k)))
        s1, s2 = (torch.rand((-(-c // g), k // 128), generator=gen, device=DEV) for c, g in ((m, 1), (n, 128)))
        group = (1 << 32) | (128 << 16) | 128

    def run():
        y = torch.full((m, n), -7777.0, dtype=torch.bfloat16, device=DEV)
        aclnn.quant_matmul_v5(*(aclnn.from_torch(t) for t in (x, w, s1, s2, y)), None, False, True, group)
        torch.cuda.synchronize()
        assert aclnn.last_kernel_name() == ("qmm_umma_split_perblock" if mode == "block" else "qmm_umma_split_deq")
        return y

    want = run()
    status = aclnn.lib().opsnn_qmm_umma_status
    assert status(1) == 0
    monkeypatch.setenv("OPSNN_TEST_SPLIT_STALL_KBLOCK", "1")
    monkeypatch.setenv("OPSNN_TEST_UMMA_POLL_LIMIT", "3000")
    bad = run()
    monkeypatch.delenv("OPSNN_TEST_SPLIT_STALL_KBLOCK")
    monkeypatch.delenv("OPSNN_TEST_UMMA_POLL_LIMIT")
    with pytest.raises(aclnn.AclnnError):
        run()
    code = status(1)  # read and cleared, which also restores the poll limit
    assert (code >> 8) in (2, 3), hex(code)
    assert bool((bad == -7777.0).all())
    assert torch.equal(run(), want) and status(1) == 0


def test_per_block_on_weights_stored_along_k(aclnn):
    """Few rows and a long k: the waits of the instances for x2 stored (n,k) gain by an out-of-line part of their own (with the one that all kernels
    of the file share such a call took as long as on (k,n), with its own 0.92 times). Up to five attempts, for a GPU whose clock moves."""
    import torch

    from gpu_util import DEV, least_times

    m, k, n = 9, 8448, 6144
    gen = torch.Generator(device=DEV).manual_seed(12)
    x = torch.randn((m, k), generator=gen, device=DEV).to(torch.float8_e4m3fn)
    s1 = torch.rand((m, k // 128), generator=gen, device=DEV)
    calls = {}
    for nk in (True, False):
        w = torch.randn((n, k) if nk else (k, n), generator=gen, device=DEV).to(torch.float8_e4m3fn)
        s2 = torch.rand((n // 128, k // 128) if nk else (k // 128, n // 128), generator=gen, device=DEV)
        y = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
        d = [aclnn.from_torch(t) for t in (x, w, s1, s2, y)]
        group = (1 << 32) | (128 << 16) | 128
        ws = torch.empty(max(1, aclnn.quant_matmul_v5(*d, None, False, nk, group)), dtype=torch.uint8, device=DEV)
        assert aclnn.last_kernel_name() == "qmm_umma_split_perblock"
        calls[nk] = lambda d=d, nk=nk, ws=ws, keep=(w, s2, y): aclnn.quant_matmul_v5(*d, None, False, nk, group, workspace=ws)
    ratios = []
    for _ in range(5):
        t = least_times(calls)
        ratios.append(t[True] / t[False])
        if ratios[-1] <= 0.96:
            return
    assert False, ratios


def test_fewer_columns_do_not_take_longer(aclnn):
    """A stream's pieces of a tile are added up by whoever arrives last: two tiles of 128 k-blocks, cut that way, took nine times as long as eight times
    the columns; cut into clusters they take less. Up to five attempts, for a GPU whose clock moves between the two."""
    import torch

    from gpu_util import DEV, least_times

    m, k = 16, 16384
    gen = torch.Generator(device=DEV).manual_seed(13)
    x = torch.randn((m, k), generator=gen, device=DEV).to(torch.float8_e4m3fn)
    s1 = torch.rand(m, generator=gen, device=DEV)
    calls = {}
    for n in (256, 2048):
        w = torch.randn((n, k), generator=gen, device=DEV).to(torch.float8_e4m3fn)
        s2 = torch.rand(n, generator=gen, device=DEV)
        y = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
        d = [aclnn.from_torch(t) for t in (x, w, s1, s2, y)]
        ws = torch.empty(max(1, aclnn.quant_matmul_v5(*d, None, False, True)), dtype=torch.uint8, device=DEV)
        assert aclnn.last_kernel_name() == "qmm_umma_split_deq"
        calls[n] = lambda d=d, ws=ws, keep=(w, s2, y): aclnn.quant_matmul_v5(*d, None, False, True, workspace=ws)
    ratios = []
    for _ in range(5):
        t = least_times(calls)
        ratios.append(t[256] / t[2048])
        if ratios[-1] <= 1.0:
            return
    assert False, ratios
