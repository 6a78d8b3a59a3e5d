"""The few-row kernels (1 .. 8 rows) at the sizes where their tiles, splits and rings end: rows that do not fill a 16-row tile, one
superblock, superblock counts that do not divide, activations that take one CTA per SM or two passes; dense and per-expert."""
import numpy as np
import pytest

from arcinferzero_b200 import synth as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


def rel(a, b):
    return float(np.abs(a.astype(np.float64) - b).max() / np.abs(b).max())


@pytest.mark.parametrize("qt", [12, 8, 14])
# (48, 17408) and (2400, 6144): Q4_K rows left over after whole rounds, dealt out by passes
@pytest.mark.parametrize("N,K", [(8, 256), (17, 512), (1000, 768), (4104, 2304), (48, 17408), (3000, 4096), (2400, 6144)])
def test_rows_match_oracle(izb, qt, N, K):
    import torch
    w = S.make_weight(qt, N, K, N + K + qt)
    W = izb.Weight(qt, w, N, K)
    for T in (1, 2, 3, 5, 8):
        aq, asc, _ = O.quantize_act(S.make_act(T, K, T + K), Mp=16)
        ref = O.matmul(qt, w, K, aq, asc, T, "f64")
        base = np.random.default_rng(T).standard_normal((T, N + 8)).astype(np.float32)
        for acc in (0, 1):
            out = torch.from_numpy(base).cuda()
            izb.matmul(W, torch.from_numpy(aq).cuda(), torch.from_numpy(asc).cuda(), T, out=out, c_off=4, acc=acc)
            got = out.cpu().numpy()
            assert rel(got[:, 4:N + 4] - (base[:, 4:N + 4] if acc else 0), ref) < (4 * TOL if acc else TOL), (T, acc)
            assert (got[:, :4] == base[:, :4]).all() and (got[:, N + 4:] == base[:, N + 4:]).all()
    assert izb.device_status(0) == 0
    W.close()


# Which kernel takes a call depends on its type, rows and sizes; a row's bits must not, since a decode step requantises them (Q4_K with
# K % 1024 == 0 and N >= 1024 has kernels of its own order up to four rows: there the few-row kernels are compared among themselves).
# Row tiles that fill no block of any split (16, 48, 96 rows), the borders of the dispatch in K and N, activations that take two passes.
@pytest.mark.parametrize("qt,N,K", [(14, 16, 512), (14, 48, 2048), (14, 96, 8192), (14, 112, 8448), (14, 144, 8192), (14, 1184, 17408), (14, 1200, 17408), (14, 4096, 1024),
                                    (12, 16, 4096), (12, 48, 1536), (12, 96, 4096), (12, 1008, 2048), (12, 2368, 18944), (12, 2384, 18944), (12, 16384, 2304), (12, 8192, 5376),
                                    (12, 4096, 8960), (12, 4096, 9472), (12, 12304, 5376), (12, 16384, 3840), (12, 1024, 2048), (8, 4096, 256), (8, 4096, 8192), (8, 16384, 1024), (8, 4112, 2304), (8, 6144, 512), (8, 16, 1024),
                                    (12, 5104, 5376), (12, 5120, 5376), (12, 4080, 6656), (12, 4096, 6656), (12, 12288, 3840), (12, 12288, 4352), (8, 24576, 2560), (8, 24592, 2560), (8, 65552, 1792),
                                    (8, 24576, 4352), (8, 24592, 4352),
                                    (13, 64, 768), (23, 64, 768), (2, 4096, 512)])
def test_rows_do_not_depend_on_their_number(izb, qt, N, K):
    import torch
    own_order = qt == 12 and K % 1024 == 0 and N >= 1024
    W = izb.Weight(qt, np.tile(S.make_weight(qt, 16, K, N + K + qt), (N // 16, 1)), N, K)
    x = torch.from_numpy(S.make_act(8, K, 5)).cuda()
    aq, asc, _ = izb.quantize_act(x)
    first = 5 if own_order else 1
    want = [izb.gemv(W, aq[j:].contiguous(), asc[:, j:].contiguous(), 1)[0] for j in range(8)] if not own_order else izb.gemv(W, aq, asc, 8)
    for T in range(first, 9):
        got = izb.gemv(W, aq, asc, T)
        for j in range(T):
            assert torch.equal(got[j], want[j]), (T, j)
    assert izb.device_status(0) == 0
    W.close()


# The matrix instruction's kernel for up to four rows (two pieces of a row per instruction) against the dot-product kernel: the first 16 weight
# rows alone make a matrix that is too small for the former.  Rows that do not fill a tile, fewer superblocks than warps share, odd counts of them,
# both sides of the K up to which the dot product's rings hold whole rows, and of the bounds in N.
@pytest.mark.parametrize("qt,N,K,Ts", [(14, 257, 4352, "1234"), (14, 1000, 8448, "1234"), (14, 4100, 4608, "1234"), (12, 12288, 256, "134"), (12, 12290, 3328, "1234"), (12, 2561, 768, "4"),
                                       (12, 4100, 2304, "34"), (12, 520, 10496, "1234"), (12, 520, 12288, "1234"), (12, 512, 17664, "1234"), (8, 5128, 2560, "134"), (8, 40968, 256, "1234"),
                                       (8, 6152, 1280, "1234"), (8, 3080, 768, "4"), (8, 520, 5888, "1234"), (8, 4104, 5120, "34"), (8, 1000, 8448, "1234"), (8, 512, 17152, "1234")])
def test_four_rows_equal_dot_products(izb, qt, N, K, Ts):
    import torch
    rows = S.make_weight(qt, 16, K, N + K + qt)
    W, head = izb.Weight(qt, np.tile(rows, ((N + 15) // 16, 1))[:N], N, K), izb.Weight(qt, rows, 16, K)
    x = S.make_act(4, K, 7)
    x[1] *= 1e4
    aq, asc, _ = izb.quantize_act(torch.from_numpy(x).cuda())
    for T in map(int, Ts):
        izb.profile_start()
        got = izb.gemv(W, aq, asc, T)
        ran = set(izb.profile_stop())
        izb.profile_start()
        want = izb.gemv(head, aq, asc, T)
        ran_head = set(izb.profile_stop())
        assert ran == {"gemv_rows"} and "gemv_rows" not in ran_head, (T, ran, ran_head)
        for n in range(0, N, 16):
            assert torch.equal(got[:T, n:n + 16], want[:T, :min(16, N - n)]), (T, n)
    assert izb.device_status(0) == 0
    W.close(), head.close()


@pytest.mark.parametrize("qt", [12, 8])
@pytest.mark.parametrize("T,TM,F,E", [(1, 8, 256, 512), (5, 4, 768, 1024), (40, 8, 256, 2304), (3, 1, 512, 256), (40, 8, 1024, 512), (4, 8, 3072, 256)])
def test_expert_rows_equal_dense_rows(izb, qt, T, TM, F, E):
    """Every slot's expert product against the same product as a dense call on that expert's matrix."""
    import torch
    NE, NU = 8, 2
    g, u, d = (S.make_weight(qt, NE * n, k, i) for i, (n, k) in enumerate(((F, E), (F, E), (E, F))))
    Wg, Wu, Wd = izb.Weight(qt, g, F, E, n_mats=NE), izb.Weight(qt, u, F, E, n_mats=NE), izb.Weight(qt, d, E, F, n_mats=NE)
    x = torch.from_numpy(S.make_act(T, E, 9)).cuda() * 0.02
    aq, asc, _ = izb.quantize_act(x)
    ids, wts, counts = izb.moe_route(torch.from_numpy(S.make_act(T, NE, 3)).cuda(), NU)
    offs, tiles, mt, stok, swt, inv = izb.moe_sort(ids, wts, counts, TM)
    h = izb.moe_gateup(Wg, Wu, aq, asc, tiles, mt, TM, stok, T * NU)
    hq, hsc, _ = izb.quantize_act(h)
    y = izb.moe_down(Wd, hq, hsc, tiles, mt, TM, swt, T * NU)
    for e in range(NE):
        for s in range(int(offs[e]), int(offs[e + 1])):
            t = int(stok[s])
            a, b = aq[t:t + 1].repeat(16, 1).contiguous(), asc[:, t:t + 1].repeat(1, 16).contiguous()
            gate, up = (izb.gemm(W, a, b, M=1, impl=izb.GEMM_CORE, mat=e)[0].double() for W in (Wg, Wu))
            want = gate / (1 + torch.exp(-gate)) * up
            assert float((h[s] - want).abs().max() / want.abs().max()) < TOL
            a, b = hq[s:s + 1].repeat(16, 1).contiguous(), hsc[:, s:s + 1].repeat(1, 16).contiguous()
            want = float(swt[s]) * izb.gemm(Wd, a, b, M=1, impl=izb.GEMM_CORE, mat=e)[0].double()
            assert float((y[s] - want).abs().max() / want.abs().max()) < TOL
    assert izb.device_status(0) == 0
    for W in (Wg, Wu, Wd):
        W.close()


@pytest.mark.parametrize("qt", [12, 8])
@pytest.mark.parametrize("F,E", [(256, 512), (272, 1024), (768, 2304), (1040, 256)])
def test_expert_rows_do_not_depend_on_the_other_tokens(izb, qt, F, E):
    """One token's expert products bit for bit in calls of 1 .. 96 tokens: few items and many, tiles of one or two slots and fuller ones,
    blocks of one row tile and of several."""
    import torch
    NE, NU = 8, 2
    g, u, d = (S.make_weight(qt, NE * n, k, i) for i, (n, k) in enumerate(((F, E), (F, E), (256, E))))
    Wg, Wu, Wd = izb.Weight(qt, g, F, E, n_mats=NE), izb.Weight(qt, u, F, E, n_mats=NE), izb.Weight(qt, d, 256, E, n_mats=NE)
    x = torch.from_numpy(S.make_act(96, E, 9)).cuda() * 0.02
    logits = torch.from_numpy(S.make_act(96, NE, 3)).cuda()
    def products(T, TM):
        aq, asc, _ = izb.quantize_act(x[:T])
        ids, wts, counts = izb.moe_route(logits[:T], NU)
        _, tiles, mt, stok, swt, inv = izb.moe_sort(ids, wts, counts, TM)
        h = izb.moe_gateup(Wg, Wu, aq, asc, tiles, mt, TM, stok, T * NU)
        aq2, asc2 = aq[stok.long()].contiguous(), asc[:, stok.long()].contiguous()  # (the down product's rows are slots)
        y = izb.moe_down(Wd, aq2, asc2, tiles, mt, TM, swt, T * NU)
        return h[inv.long()], y[inv.long()]  # by (token, choice)
    want = products(96, 8)
    for T, TM in ((1, 8), (2, 8), (3, 1), (5, 4), (9, 8), (24, 8), (48, 2), (96, 1)):
        for got, ref in zip(products(T, TM), want):
            assert torch.equal(got, ref[:T * NU]), (T, TM)
    assert izb.device_status(0) == 0
    for W in (Wg, Wu, Wd):
        W.close()


def test_rows_too_long_for_the_rings(izb):
    """Activations that leave no room for a ring go to the kernels that take them in pieces: expert rows of K = 20480, Q6_K rows of 65536."""
    import torch
    NE, NU, T, N, K = 2, 1, 5, 64, 20480
    for qt in (12, 8):
        g, u = S.make_weight(qt, NE * N, K, 1), S.make_weight(qt, NE * N, K, 2)
        Wg, Wu = izb.Weight(qt, g, N, K, n_mats=NE), izb.Weight(qt, u, N, K, n_mats=NE)
        aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(T, K, 9)).cuda() * 0.01)
        ids, wts, counts = izb.moe_route(torch.from_numpy(S.make_act(T, NE, 3)).cuda(), NU)
        _, tiles, mt, stok, swt, inv = izb.moe_sort(ids, wts, counts, 8)
        h = izb.moe_gateup(Wg, Wu, aq, asc, tiles, mt, 8, stok, T * NU)[inv.long()]
        y = izb.moe_down(Wg, aq[stok.long()].contiguous(), asc[:, stok.long()].contiguous(), tiles, mt, 8, swt, T * NU)[inv.long()]
        for t in range(T):
            e = int(ids[t, 0])
            gate, up = (izb.gemm(W, aq, asc, impl=izb.GEMM_CORE, mat=e)[t].double() for W in (Wg, Wu))
            for got, want in ((h[t], gate / (1 + torch.exp(-gate)) * up), (y[t], gate * float(wts[t, 0]))):
                assert float((got - want).abs().max() / want.abs().max()) < TOL
        Wg.close()
        Wu.close()
    W = izb.Weight(14, S.make_weight(14, N, 65536, 4), N, 65536)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(2, 65536, 5)).cuda())
    want = izb.gemm(W, aq, asc, impl=izb.GEMM_CORE)[:2].double()
    for t in (1, 2):
        got = izb.gemv(W, aq, asc, t)
        assert float((got - want[:t]).abs().max() / want.abs().max()) < TOL
    assert izb.device_status(0) == 0
    W.close()
