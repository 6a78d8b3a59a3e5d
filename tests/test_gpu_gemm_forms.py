"""The tcgen05 GEMM on every weight form it takes (one and two fp16 terms per weight, with and without mins), on columns that do
not fill its tiles and on calls whose K range is cut into parts, against the CUDA-core kernel (itself checked against the oracle); which
calls take it, and which of them are cut."""
import numpy as np
import pytest

from arcinferzero_b200 import synth as S

pytestmark = pytest.mark.gpu


def kernels_of(izb, call):
    """Names of the library kernels that `call` launches."""
    izb.profile_start()
    call()
    return set(izb.profile_stop())


def extremes(qt, rows):
    """Largest scales and quants of either sign in some rows: products up to 4096 must stay exact."""
    v = rows.copy()
    if qt == 14:
        v = v.reshape(v.shape[0], -1, 210)
        v[0, :, 0:192], v[0, :, 192:208] = 0xFF, 0x80   # quant 31, scale -128
        v[1, :, 0:192], v[1, :, 192:208] = 0x00, 0x80   # quant -32, scale -128: 4096
        v[2, :, 0:192], v[2, :, 192:208] = 0x00, 0x7F
    elif qt == 23:
        v = v.reshape(v.shape[0], -1, 136)
        v[0, :, 2:8], v[0, :, 8:] = 0x00, 0x00          # scale -32, codebook -127
        v[1, :, 2:8], v[1, :, 8:] = 0xFF, 0xFF          # scale 31, codebook 113
    elif qt in (12, 13):
        v = v.reshape(v.shape[0], -1, 144 if qt == 12 else 176)
        v[0, :, 4:] = 0xFF
    return v.reshape(rows.shape)


# (16, 16): the smallest calls; 144, 272: a part of the last column tile; 40 x 128 x 4096 and 130 x 144 x 2304: K cut into parts;
# 300 x 2432 x 512: more tiles than half the SMs, not cut
@pytest.mark.parametrize("qt", [12, 8, 2, 13, 14, 23])
@pytest.mark.parametrize("M,N,K", [(16, 16, 256), (16, 16, 1280), (130, 144, 2304), (40, 128, 4096), (129, 272, 768), (300, 2432, 512)])
def test_tensor_core_gemm_equals_core_gemm(izb, qt, M, N, K):
    """Which kernel ran is looked at: IZB_GEMM_AUTO may take the other one, and would then be compared with itself."""
    import torch
    W = izb.Weight(qt, extremes(qt, S.make_weight(qt, N, K, N + K + qt)), N, K)
    Mp = izb.pad_rows(M)
    x = torch.from_numpy(S.make_act(M, K, M + K)).cuda()
    x[0] = 1.0  # every int8 = 127
    aq, asc, _ = izb.quantize_act(x, Mp=Mp)
    impls = [izb.GEMM_AUTO, izb.GEMM_TC] if qt in (12, 8, 2) else [izb.GEMM_AUTO]  # (the per-16-scale types cannot name the kernel)
    for acc in (0, 1, 2):
        base = torch.from_numpy(np.random.default_rng(acc).standard_normal((Mp, N + 8)).astype(np.float32)).cuda()
        b = base.clone()
        izb.gemm(W, aq, asc, M=M, out=b, c_off=4, acc=acc, impl=izb.GEMM_CORE)
        for impl in impls:
            a = base.clone()
            ran = kernels_of(izb, lambda: izb.gemm(W, aq, asc, M=M, out=a, c_off=4, acc=acc, impl=impl))
            short = impl == izb.GEMM_AUTO and (qt not in (12, 8, 2) or N % 128 != 0) and K <= 512 << acc  # (may go to the CUDA cores, below)
            folded = qt in (12, 13) and impl == izb.GEMM_AUTO and acc == 0 and K >= 2048
            assert ("gemm_fold" if folded else "gemm_tc") in ran or short, (acc, impl, ran)
            assert ("gemm_fold" in ran) + ("gemm_tc" in ran) <= 1, (acc, impl, ran)
            assert ("split_reduce" in ran) == (impl == izb.GEMM_AUTO and acc == 0 and K >= 2048), (acc, impl, ran)
            ra, rb = a[:M, 4:N + 4].double(), b[:M, 4:N + 4].double()
            assert float((ra - rb).abs().max() / rb.abs().max()) < 1e-5, (acc, impl)
            assert torch.equal(a[:, :4], base[:, :4]) and torch.equal(a[:, N + 4:], base[:, N + 4:]) and torch.equal(a[M:], base[M:])
    want = izb.gemm(W, aq, asc)
    got = []
    ran = kernels_of(izb, lambda: got.append(izb.quant_matmul(W, x, M)[0]))
    assert "quant_prepare" in ran or K <= 512, ran
    assert ("gemm_fold" in ran) == (qt in (12, 13) and K >= 2048), ran
    assert torch.equal(got[0][:M], want[:M])
    assert izb.device_status(0) == 0
    W.close()


@pytest.mark.parametrize("qt", [13, 14, 23])
def test_scaled_products_are_exact(izb, qt):
    """scale * quant reaches 4096 and travels as one or two fp16 terms.  With unit factors and one block's activation scale at 1, the others at
    0, an output is that block's integer: equal to the CUDA-core kernel's (itself equal to the oracle's) bit for bit."""
    import torch
    M, N, K = 130, 144, 1280
    w = extremes(qt, S.make_weight(qt, N, K, qt)).copy()
    sb = w.reshape(N, K // 256, -1)
    at = 208 if qt == 14 else 0
    sb[:, :, at:at + 2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
    if qt == 13:
        sb[:, :, 2:4] = 0
    W = izb.Weight(qt, w, N, K)
    Mp = izb.pad_rows(M)
    x = torch.from_numpy(S.make_act(M, K, 7)).cuda()
    x[0], x[1] = 1.0, -1.0
    aq, asc, _ = izb.quantize_act(x, Mp=Mp)
    assert "gemm_tc" in kernels_of(izb, lambda: izb.gemm(W, aq, asc, M=M))
    largest = 0.0
    for b in range(K // 32):
        one = torch.zeros_like(asc)
        one[b] = 1.0
        got, want = izb.gemm(W, aq, one, M=M)[:M], izb.gemm(W, aq, one, M=M, impl=izb.GEMM_CORE)[:M]
        assert torch.equal(got, want) and torch.equal(got, got.round()), b
        largest = max(largest, float(got.abs().max()))
    assert largest > (2.0 ** 23 if qt != 13 else 2.0 ** 20)
    assert izb.device_status(0) == 0
    W.close()


# One wave of 64 x 64 tiles over a short K goes to the CUDA-core kernel, where the tensor-core kernel is the newcomer (part columns,
# per-16-scale types); the border in K depends on type and store mode.
@pytest.mark.parametrize("qt,M,N,K,acc,core", [(14, 64, 128, 256, 0, True), (14, 64, 128, 512, 0, False), (13, 64, 144, 512, 1, True), (23, 64, 144, 768, 1, False),
                                               (14, 64, 272, 1024, 2, True), (14, 64, 272, 1280, 2, False), (14, 1024, 1040, 256, 0, False), (8, 64, 144, 512, 0, True),
                                               (8, 64, 144, 768, 0, False), (2, 64, 144, 1024, 1, True), (8, 64, 144, 2048, 2, True), (12, 64, 144, 512, 1, True),
                                               (12, 64, 144, 512, 0, False), (12, 64, 128, 256, 0, False), (8, 64, 256, 256, 2, False)])
def test_short_calls_take_the_faster_kernel(izb, qt, M, N, K, acc, core):
    import torch
    W = izb.Weight(qt, S.make_weight(qt, N, K, N + K + qt), N, K)
    x = torch.from_numpy(S.make_act(M, K, M + K)).cuda()
    aq, asc, _ = izb.quantize_act(x)
    base = torch.from_numpy(np.random.default_rng(acc).standard_normal((M, N)).astype(np.float32)).cuda()
    want = izb.gemm(W, aq, asc, out=base.clone(), acc=acc, impl=izb.GEMM_CORE)
    a, b = base.clone(), base.clone()
    for out, call in ((a, lambda: izb.matmul(W, aq, asc, M, out=a, acc=acc)), (b, lambda: izb.quant_matmul(W, x, M, out=b, acc=acc))):
        ran = kernels_of(izb, call)
        assert ("gemm_tc" not in ran) == core, ran
        assert torch.equal(out, want) if core else float((out - want).abs().max() / want.abs().max()) < 1e-5
    assert torch.equal(a, b)
    W.close()


@pytest.mark.parametrize("qt", [12, 8, 14])
def test_sm_limit_changes_no_result(izb, qt):
    """The limit caps the grid of the GEMM; how a long K is cut into parts, and with it where sums are rounded, does not follow it."""
    import torch
    M, N, K = 40, 256, 4096
    W = izb.Weight(qt, S.make_weight(qt, N, K, 5), N, K)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 6)).cuda())
    want = izb.gemm(W, aq, asc)
    assert "split_reduce" in kernels_of(izb, lambda: izb.gemm(W, aq, asc))
    try:
        for sms in (100, 20, 3, 1):
            izb.set_sm_limit(0, sms)
            assert torch.equal(izb.gemm(W, aq, asc), want), sms
    finally:
        izb.set_sm_limit(0, 0)
    assert izb.device_status(0) == 0
    W.close()


@pytest.mark.parametrize("qt", [12, 8])
def test_named_kernel_is_not_cut(izb, qt):
    """Where IZB_GEMM_AUTO cuts K, IZB_GEMM_TC gives the sums of izb_gemm_noalloc, a row's sums do not depend on the rows beside it, and a
    gate projection followed by store mode 2 is store mode 3."""
    import torch
    M, N, K = 40, 256, 4096
    g, u = S.make_weight(qt, N, K, 5), S.make_weight(qt, N, K, 6)
    Wg, Wu, Wgu = izb.Weight(qt, g, N, K), izb.Weight(qt, u, N, K), izb.gateup_weight(qt, g, u, N, K)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 7)).cuda() * 0.02)
    assert "split_reduce" in kernels_of(izb, lambda: izb.gemm(Wg, aq, asc))
    named = izb.gemm(Wg, aq, asc, M=M, impl=izb.GEMM_TC)
    assert torch.equal(izb.gemm_noalloc(Wg, aq, asc, M=M, out=torch.zeros_like(named))[:M], named[:M])
    many = izb.gemm(Wg, aq.repeat(8, 1), asc.repeat(1, 8), impl=izb.GEMM_TC)
    assert torch.equal(many[:M], named[:M])
    assert torch.equal(izb.gemm(Wu, aq, asc, M=M, out=named, acc=2)[:M], izb.gemm(Wgu, aq, asc, M=M, acc=3)[:M])
    assert izb.device_status(0) == 0
    for W in (Wg, Wu, Wgu):
        W.close()


def test_selfcheck_runs_every_form():
    """The start-up check switches the tensor-core kernel for all weight forms, part columns and cut K: it must run them all.  (In a process
    of its own: the verdict is kept.)"""
    import os
    import subprocess
    import sys
    body = """
import torch, arcinferzero_b200 as izb
izb.profile_start()
izb.selfcheck(0)
ran = izb.profile_stop()
# five forms x (plain cut, adding, SwiGLU, plain uncut), two with block dots; two forms in the folded kernel, cut and uncut
assert ran["gemm_tc"]["launches"] == 22 and ran["gemm_fold"]["launches"] == 4 and ran["split_reduce"]["launches"] == 7, ran
assert sum(ran[k]["launches"] for k in ran if k.startswith("gemm_k16")) == 14, ran
assert izb.device_status(0) == 0
print("done")
"""
    r = subprocess.run([sys.executable, "-c", body], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
