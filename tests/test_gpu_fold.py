"""The folded GEMM (plain stores of Q4_K and Q5_K products of K >= 2048 under GEMM_AUTO): tiles of any number of token rows, part columns, K cut and not, extreme
and non-finite scales."""
import numpy as np
import pytest

from arcinferzero_b200 import synth as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def weights64(qt, rows, K):
    """The weights in 64 bits, exactly."""
    n, nsb = rows.shape[0], K // 256
    w, out = rows.reshape(n, nsb, -1), np.empty((n, nsb, 16, 16))
    for i in range(n):
        for s in range(nsb):
            if qt == 12:
                d, dmin, sc, mn, q = O.decode_q4k_sb(w[i, s])
                sc, mn = sc.repeat(2), mn.repeat(2)
            else:
                d, dmin, sc, mn, _, q = O.decode_generic_sb(qt, w[i, s])
            out[i, s] = d * sc[:, None].astype(np.float64) * q.reshape(16, 16) - dmin * mn[:, None].astype(np.float64)
    return out.reshape(n, K)


def exact(qt, rows, K, aq, asc):
    a = aq.astype(np.float64).reshape(len(aq), K // 32, 32) * asc.T[:, :, None].astype(np.float64)
    return a.reshape(len(aq), K) @ weights64(qt, rows, K).T


def run(izb, W, aq, asc, M, N, Mp):
    import torch
    out = torch.full((Mp, N + 8), float("nan"), device="cuda")
    izb.profile_start()
    izb.gemm(W, aq, asc, M=M, out=out, c_off=4)
    ran = izb.profile_stop()
    assert izb.device_status(0) == 0 and "gemm_fold" in ran and "gemm_tc" not in ran, ran
    got = out.cpu().numpy()
    assert np.isnan(got[:, :4]).all() and np.isnan(got[:, N + 4:]).all() and np.isnan(got[M:]).all()
    return got[:M, 4:N + 4]


# 9 .. 145 rows: one tile of each height, two tiles of unequal ones; 144: a part column tile; 20000 columns: more than one round, K not cut
@pytest.mark.parametrize("qt", [12, 13])
@pytest.mark.parametrize("M,N,K", [(9, 128, 2048), (16, 128, 2304), (33, 128, 2048), (64, 256, 2560), (97, 128, 2048), (128, 128, 2048), (129, 256, 2048), (145, 128, 4096),
                                   (300, 144, 2304), (40, 20000, 2048), (700, 4096, 2048)])
def test_fold_against_64_bits(izb, qt, M, N, K):
    """Bound: the activations keep 22 bits of a superblock's largest, the superblock's sum is cut once below 2^-23 of itself, and K / 256 such sums are
    added in f32: some 2e-7 of the result's norm; 4e-7 leaves room for the spread."""
    import torch
    w = S.make_weight(qt, N, K, N + K)
    W = izb.Weight(qt, w, N, K)
    Mp = izb.pad_rows(M)
    x = S.make_act(M, K, M + K)
    x.reshape(M, -1, 32)[:, ::3] *= 40.0  # superblocks whose blocks differ in scale
    aq, asc, _ = izb.quantize_act(torch.from_numpy(x).cuda(), Mp=Mp)
    got = run(izb, W, aq, asc, M, N, Mp)
    cols = np.unique(np.linspace(0, N - 1, 96).astype(int))
    ref = exact(qt, w[cols], K, aq[:M].cpu().numpy(), asc[:, :M].cpu().numpy())
    err = np.linalg.norm(got[:, cols] - ref) / np.linalg.norm(ref)
    assert err < 4e-7, err
    core = izb.gemm(W, aq, asc, M=M, impl=izb.GEMM_CORE).cpu().numpy()[:M]
    assert np.abs(got - core).max() / np.abs(core).max() < 1e-5
    both, q, _ = izb.quant_matmul(W, torch.from_numpy(x).cuda(), M)
    assert torch.equal(q, aq) and (both.cpu().numpy()[:M] == got).all()  # the pre-pass with the quantiser in it
    W.close()


def test_rows_do_not_depend_on_the_tile(izb):
    import torch
    N, K = 10240, 2048  # (80 column tiles: K is not cut)
    W = izb.Weight(12, np.tile(S.make_weight(12, 256, K, 1), (N // 256, 1)), N, K)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(400, K, 2)).cuda())
    want = izb.gemm(W, aq, asc, M=400)[:400]
    for M in (16, 48, 80, 112, 128, 160, 272):
        assert torch.equal(izb.gemm(W, aq[:M].contiguous(), asc[:, :M].contiguous(), M=M)[:M], want[:M]), M
    W.close()


@pytest.mark.parametrize("qt", [12, 13])
def test_fold_scales_at_the_ends_of_their_range(izb, qt):
    """Activation scales of 0, denormal, next to overflow and of either sign; weights at their largest.  Against the CUDA-core kernel, row by row."""
    import torch
    M, N, K = 48, 128, 2048
    w = S.make_weight(qt, N, K, 3).reshape(N, K // 256, -1).copy()
    w[0, :, 4:] = 0xFF
    w[1, :, 0:4] = 0
    W = izb.Weight(qt, w.reshape(N, -1), N, K)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 4)).cuda())
    aq[0], aq[1] = 127, -128
    f = torch.ones_like(asc)
    for row, v in enumerate([1.0, 1.0, 0.0, 1e-45, 1e-40, 2.0 ** -126, 1e-36, 1e-30, 1e28, 1e31, -1.0]):
        f[:, row] = v
    f[5, 11], f[6, 12], f[7, 13], f[8, 14] = 0.0, 1e-20, -1.0, 1e20
    asc = torch.where(f.abs() < 1e-25, f, asc * f)
    got, core = izb.gemm(W, aq, asc, M=M)[:M].double(), izb.gemm(W, aq, asc, M=M, impl=izb.GEMM_CORE)[:M].double()
    assert torch.isfinite(core).all() and torch.isfinite(got).all()
    for row in range(M):
        big = core[row].abs().max()
        # (a sum of denormal terms is rounded to 2^-149 once per block in one kernel, once per superblock in the other)
        assert float((got[row] - core[row]).abs().max()) <= 1e-5 * float(big) + K / 32 * 2.0 ** -149, row
    assert float(core[3].abs().max()) > 0
    W.close()


def test_fold_scales_that_are_no_numbers(izb):
    """An infinite or undefined scale reaches what it reaches in the CUDA-core kernel's results, its own row, and no other row."""
    import torch
    M, N, K = 48, 128, 2048
    W = izb.Weight(12, S.make_weight(12, N, K, 5), N, K)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 6)).cuda())
    want = izb.gemm(W, aq, asc, M=M)[:M]
    asc[3, 2], asc[9, 20], asc[32, 33] = float("inf"), float("nan"), float("-inf")
    got, core = izb.gemm(W, aq, asc, M=M)[:M], izb.gemm(W, aq, asc, M=M, impl=izb.GEMM_CORE)[:M]
    assert torch.equal(torch.isfinite(got), torch.isfinite(core))
    keep = [r for r in range(M) if r not in (2, 20, 33)]
    assert torch.equal(got[keep], want[keep])
    W.close()


# Up to 4 : 1 two terms, up to 4096 : 1 three, beyond that block by block; 40 token rows, and tiles whose rows differ in kind
RATIOS = [1.0, 3.0, 5.0, 40.0, 2.0 ** 10, 2.0 ** 11.8, 2.0 ** 12.4, 2.0 ** 14, 2.0 ** 28, 2.0 ** 40]


@pytest.mark.parametrize("qt", [12, 13])
@pytest.mark.parametrize("K", [2048, 5120])
@pytest.mark.parametrize("zero", [False, True])
def test_fold_small_blocks_beside_a_large_one(izb, qt, K, zero):
    """One block of every superblock is many times the others; with `zero` its weights are zeros, and the small blocks' products are all there is.
    Bound: as in test_fold_against_64_bits, of the norm of every row."""
    import torch
    M, N = 40, 256
    w = S.make_weight(qt, N, K, K).copy()
    if zero:
        v = w.reshape(N, K // 256, -1)
        v[:, :, 4] &= 0xC0  # sub-scale and min of block 0
        v[:, :, 8] &= 0xC0
    W = izb.Weight(qt, w, N, K)
    w64 = weights64(qt, w, K)
    for ratio in RATIOS + [None]:
        x = S.make_act(M, K, K)
        f = np.float32(ratio) if ratio else np.array([RATIOS[m % len(RATIOS)] for m in range(M)], np.float32)[:, None, None]
        x.reshape(M, K // 256, 8, 32)[:, :, 0] *= f
        aq, asc, _ = izb.quantize_act(torch.from_numpy(x).cuda())
        got = izb.gemm(W, aq, asc, M=M).cpu().numpy()[:M]
        assert izb.device_status(0) == 0
        a = aq[:M].cpu().numpy().astype(np.float64).reshape(M, K // 32, 32) * asc[:, :M].cpu().numpy().T[:, :, None].astype(np.float64)
        ref = a.reshape(M, K) @ w64.T
        err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert err.max() < 4e-7, (ratio, err.max())
    W.close()


@pytest.mark.parametrize("qt,M,N,K", [(12, 130, 256, 2048), (13, 100, 144, 2304), (12, 40, 20000, 2048), (13, 40, 20000, 2048)])
def test_rows_do_not_depend_on_the_kinds_of_others(izb, qt, M, N, K):
    """Rows with two terms, with three and with blocks one by one, alone and beside each other in a superblock."""
    import torch
    W = izb.Weight(qt, np.tile(S.make_weight(qt, 16, K, 1), (N // 16, 1)), N, K)

    def run_with(kinds):
        x = S.make_act(M, K, 2)
        for sb in range(K // 256):
            for m in range(M):
                x[m, 256 * sb + 32 * (m % 8):256 * sb + 32 * (m % 8) + 32] *= np.float32(kinds(m, sb))
        aq, asc, _ = izb.quantize_act(torch.from_numpy(x).cuda())
        out = izb.gemm(W, aq, asc, M=M)[:M]
        assert izb.device_status(0) == 0
        return out
    plain, spread, wide = (run_with(lambda m, sb, f=f: f) for f in (1.0, 100.0, 2.0 ** 20))
    for a, b in ((1.0, 100.0), (1.0, 2.0 ** 20), (100.0, 2.0 ** 20)):
        of = {1.0: plain, 100.0: spread, 2.0 ** 20: wide}
        mixed = run_with(lambda m, sb: a if m % 3 else b)
        for m in range(M):
            assert torch.equal(mixed[m], of[a if m % 3 else b][m]), (a, b, m)
    W.close()


@pytest.mark.parametrize("M", [9, 40, 130])
def test_fold_rows_that_are_not_stored(izb, M):
    """What the padding rows hold (here no numbers, and scales far apart) reaches no result and is not written to."""
    import torch
    N, K = 256, 2048
    W = izb.Weight(12, S.make_weight(12, N, K, 3), N, K)
    Mp = izb.pad_rows(M) + 16
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 4)).cuda(), Mp=Mp)
    want = run(izb, W, aq, asc, M, N, Mp)
    aq[M:], asc[:, M:], asc[::3, M:], asc[::8, M + 1:] = 77, 1e30, 1e-20, float("nan")
    assert (run(izb, W, aq, asc, M, N, Mp) == want).all()
    W.close()


@pytest.mark.parametrize("qt,M,N,K", [(12, 40, 256, 2048), (13, 40, 256, 2048), (12, 40, 20000, 2048), (13, 40, 20000, 2048)])
@pytest.mark.parametrize("ratio", [1.0, 100.0, 2.0 ** 20])
def test_fold_waits_that_run_out(izb, qt, M, N, K, ratio):
    """Every element is the right one or was left alone, with K cut and not; the next call is whole again."""
    import torch
    W = izb.Weight(qt, np.tile(S.make_weight(qt, 16, K, 1), (N // 16, 1)), N, K)
    x = S.make_act(M, K, 2)
    x.reshape(M, K // 256, 8, 32)[M // 2:, :, 3] *= np.float32(ratio)
    Mp = izb.pad_rows(M)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(x).cuda(), Mp=Mp)
    want = izb.gemm(W, aq, asc, M=M)[:M]
    assert izb.device_status(0) == 0
    gave_up = 0
    for limit, skip in ((1, -1), (2, -1), (3, -1), (5, -1), (8, -1), (2000, 0), (2000, 5), (2000, 30)):  # (skip: a unit of the activations that is left out)
        izb.debug_wait_test(limit, skip)
        out = torch.full((Mp, N), float("nan"), device="cuda")
        izb.gemm(W, aq, asc, M=M, out=out)
        status = izb.device_status(0)
        kept = torch.isnan(out[:M])
        assert torch.equal(out[:M][~kept], want[~kept]), (limit, skip)
        assert status != 0 or not bool(kept.any())
        assert skip < 0 or status != 0
        gave_up += status != 0
    assert gave_up >= 3
    assert torch.equal(izb.gemm(W, aq, asc, M=M)[:M], want) and izb.device_status(0) == 0
    W.close()


# (256 tiles, and four, whose K is cut)
@pytest.mark.parametrize("qt,N,K,M,cut", [(12, 1024, 2048, 4096, False), (12, 128, 4096, 512, True), (13, 128, 4096, 512, True)])
def test_fold_in_a_capture_without_its_arena(izb, qt, N, K, M, cut):
    """Where the folded kernel's arena would have to grow inside a capture, the call goes to the other kernel, which may cut K as well."""
    import os
    import subprocess
    import sys
    body = f"""qt, N, K, M, cut = {qt}, {N}, {K}, {M}, {cut}
import torch, arcinferzero_b200 as izb
from arcinferzero_b200 import synth as S
W = izb.Weight(qt, S.make_weight(qt, N, K, 1), N, K)
aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 2)).cuda())
izb.gemm(W, aq, asc, out=torch.zeros(M, N, device="cuda"), acc=1)  # the arena of the other kernel
want = izb.gemm(W, aq, asc, out=torch.zeros(M, N, device="cuda"), acc=1)
core = izb.gemm(W, aq, asc, impl=izb.GEMM_CORE)
out = torch.zeros(M, N, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    izb.gemm(W, aq, asc, out=out)
g.replay()
torch.cuda.synchronize()
assert torch.equal(out, want) != cut and float((out - core).abs().max()) <= 1e-5 * float(core.abs().max())
got = out.clone()
izb.gemm(W, aq, asc, out=out)  # (the folded kernel)
assert not torch.equal(out, got) and izb.device_status(0) == 0
print("done")
"""
    r = subprocess.run([sys.executable, "-c", body], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr


def test_fold_without_memory_for_its_arena(izb):
    """On a full GPU a call whose folded arena cannot be had keeps the arena that is there, here one that a graph holds, and goes to the other kernel, as often as
    it is made; with memory again, the folded kernel has its own."""
    import os
    import subprocess
    import sys
    body = """
import torch, arcinferzero_b200 as izb
from arcinferzero_b200 import synth as S
N, K, M = 1024, 17408, 4096  # (arenas: 190 and 450 MB; K is not cut)
W = izb.Weight(12, S.make_weight(12, N, K, 1), N, K)
aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, 2)).cuda())
out = torch.zeros(M, N, device="cuda")
izb.gemm(W, aq, asc, out=out, acc=1)
want = izb.gemm(W, aq, asc, impl=izb.GEMM_TC)
q = (torch.empty((M, K), dtype=torch.int8, device="cuda"), torch.empty((K // 32, M), dtype=torch.float32, device="cuda"))
x = torch.zeros(M, K, device="cuda")
izb.quant_matmul(W, x[:64], 64)
again = torch.zeros(M, N, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    izb.gemm(W, aq, asc, out=again, acc=1)
g.replay()
assert torch.equal(again, want)
assert torch.equal(out, want) and out.any()  # (what torch allocates for these is there then)
torch.cuda.synchronize()
full = torch.empty(torch.cuda.mem_get_info()[0] - (96 << 20), dtype=torch.uint8, device="cuda")
free = torch.cuda.mem_get_info()[0]
for i in range(5):
    out.zero_()
    izb.gemm(W, aq, asc, out=out)
    torch.cuda.synchronize()
    assert torch.equal(out, want), float((out - want).abs().max())
    assert torch.cuda.mem_get_info()[0] == free, (i, torch.cuda.mem_get_info()[0] - free)
izb.quant_matmul(W, x, M, out=out, qout=q)
torch.cuda.synchronize()
assert not out.any() and torch.cuda.mem_get_info()[0] == free and izb.device_status(0) == 0
del full
torch.cuda.empty_cache()
for i in range(300):
    izb.gemm(W, aq, asc, out=out)
assert not torch.equal(out, want) and float((out - want).abs().max()) <= 1e-5 * float(want.abs().max())
again.zero_()
g.replay()
assert torch.equal(again, want) and izb.device_status(0) == 0
print("done")
"""
    r = subprocess.run([sys.executable, "-c", body], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr


# The quantiser that prepares the operands as it goes takes one row per warp up to one wave of such blocks (148 x 8), else four: the same bytes and products
# as the quantiser and the pre-pass one after the other.
@pytest.mark.parametrize("qt,N,K", [(12, 256, 2048), (13, 272, 2304), (8, 256, 2048), (14, 256, 2304)])
@pytest.mark.parametrize("M", [9, 37, 100, 129, 1000, 1180, 1300])
def test_quantising_pre_pass_equals_two_steps(izb, qt, N, K, M):
    import torch
    W = izb.Weight(qt, S.make_weight(qt, N, K, N + K), N, K)
    x = torch.from_numpy(S.make_act(M, K, M)).cuda()
    out, aq, asc = izb.quant_matmul(W, x, M)
    bq, bsc, _ = izb.quantize_act(x)
    assert torch.equal(aq, bq) and torch.equal(asc.view(torch.int32), bsc.view(torch.int32))
    assert torch.equal(out[:M], izb.matmul(W, bq, bsc, M)[:M])
    assert izb.device_status(0) == 0
    W.close()
