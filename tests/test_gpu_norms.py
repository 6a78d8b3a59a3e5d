"""The norm producers at the borders of their register plans: elements per thread, and numbers of long rows that change what a block
holds.  Bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


# (148 SMs: the number of long rows up to which a block holds both of its rows)
@pytest.mark.parametrize("M,K", [(3, 1024), (3, 1280), (3, 2304), (3, 4352), (3, 5376), (3, 8192), (3, 8448), (148, 8448), (149, 8448), (300, 16384)])
def test_add_norm_quant(izb, M, K):
    import torch
    rng = np.random.default_rng(M + K)
    x, t = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((M, K), dtype=np.float32) * 3
    w, w2 = ((1.0 + 0.2 * rng.standard_normal(K)).astype(np.float32) for _ in range(2))
    for second in (w2, None):
        xd = torch.from_numpy(x).cuda()
        aq, asc = izb.add_norm_quant(xd, torch.from_numpy(t).cuda(), torch.from_numpy(w).cuda(), 1e-6, 0.75, None if second is None else torch.from_numpy(second).cuda())
        rx, raq, rasc, _ = O.add_norm_quant(x, t, w, 1e-6, 0.75, second, Mp=asc.shape[1])
        assert (bits(xd.cpu().numpy()) == bits(rx)).all() and (aq.cpu().numpy() == raq).all() and (bits(asc.cpu().numpy()) == bits(rasc)).all()


# (148 SMs: two rows of more than 12288, or fourteen of more than 8192 values per SM are held in registers, more are read twice)
@pytest.mark.parametrize("M,K", [(3, 2304), (3, 4352), (3, 6400), (3, 8192), (3, 8448), (3, 12544), (3, 16640), (296, 12544), (297, 12544), (2072, 8448), (2073, 8448)])
def test_rmsnorm_quant(izb, M, K):
    import torch
    rng = np.random.default_rng(M + K)
    x, w = rng.standard_normal((M, K), dtype=np.float32), (1.0 + 0.2 * rng.standard_normal(K)).astype(np.float32)
    aq, asc, h = izb.rmsnorm_quant(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), 1e-6, want_h=True)
    ry, raq, rasc, _ = O.rmsnorm_quant(x, w, 1e-6, Mp=asc.shape[1])
    assert (bits(h.cpu().numpy()) == bits(ry)).all() and (aq.cpu().numpy() == raq).all() and (bits(asc.cpu().numpy()) == bits(rasc)).all()


# Few rows are shared by several CTAs (with the residual addition up to 3 x 148 CTAs in clusters of up to eight; without up to eight rows of 4096 and
# more): shares that do not divide, rows without a second norm, sums and padding, a step of a row that runs on from the one before.
@pytest.mark.parametrize("M,K", [(1, 1280), (1, 1536), (5, 2304), (2, 3840), (8, 4096), (48, 4096), (64, 4096), (3, 4352), (5, 4608), (1, 4864), (8, 5120), (63, 5120)])
def test_norms_of_few_rows(izb, M, K):
    import torch
    rng = np.random.default_rng(M + K)
    x, w, w2 = (rng.standard_normal(n, dtype=np.float32) for n in ((M, K), K, K))
    for second in (w2, None):
        xd, rx = torch.from_numpy(x).cuda(), x
        for step in range(3):
            t = rng.standard_normal((M, K), dtype=np.float32) * 3
            aq, asc = izb.add_norm_quant(xd, torch.from_numpy(t).cuda(), torch.from_numpy(w).cuda(), 1e-6, 0.75, None if second is None else torch.from_numpy(second).cuda())
            rx, raq, rasc, _ = O.add_norm_quant(rx, t, w, 1e-6, 0.75, second, Mp=asc.shape[1])
            assert (bits(xd.cpu().numpy()) == bits(rx)).all() and (aq.cpu().numpy() == raq).all() and (bits(asc.cpu().numpy()) == bits(rasc)).all(), step
    wide = torch.from_numpy(np.concatenate([x, x], 1)).cuda()  # (a row stride of its own)
    aq, asc, h = izb.rmsnorm_quant(wide[:, :K], torch.from_numpy(w).cuda(), 1e-6, want_h=True)
    ry, raq, rasc, _ = O.rmsnorm_quant(x, w, 1e-6, Mp=asc.shape[1])
    assert (bits(h.cpu().numpy()) == bits(ry)).all() and (aq.cpu().numpy() == raq).all() and (bits(asc.cpu().numpy()) == bits(rasc)).all()


# ... and the same bits as in many rows where values are no finite numbers: a row with one NaN is NaN throughout behind the norm.
@pytest.mark.parametrize("K", [1280, 2048, 4096, 5120])
def test_add_norm_quant_of_no_numbers(izb, K):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K)
    x, t = (torch.randn((600, K), generator=gen, device="cuda") for _ in range(2))
    w, w2 = (torch.randn(K, generator=gen, device="cuda") for _ in range(2))
    t[1, 5], t[2, 40], x[3, 700], x[4, 64:96], t[5, 0] = float("nan"), float("inf"), float("nan"), float("nan"), float("-inf")
    t[6], x[6] = 0.0, 0.0
    x[7, 32:64] = float("inf")
    same = lambda a, b: torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))
    for second in (w2, None):
        xm, xf = x.clone(), x[:8].clone()
        aqm, ascm = izb.add_norm_quant(xm, t, w, 1e-6, 0.75, second)
        aqf, ascf = izb.add_norm_quant(xf, t[:8].contiguous(), w, 1e-6, 0.75, second)
        assert same(xm[:8], xf) and same(aqm[:8], aqf[:8]) and same(ascm[:, :8], ascf[:, :8])
        assert bool(torch.isnan(ascf[:, 1]).all())


# The residual addition's outputs may lie anywhere (padding rows are zeroed 16 bytes at a time where they are aligned).
@pytest.mark.parametrize("M,K,off", [(1, 1024, 1), (3, 2048, 4), (3, 2048, 0), (5, 5376, 8)])
def test_add_norm_quant_unaligned_output(izb, M, K, off):
    import ctypes as C
    import torch
    rng = np.random.default_rng(M + K)
    x, t, w = (rng.standard_normal(n, dtype=np.float32) for n in ((M, K), (M, K), K))
    xd, td, wd = (torch.from_numpy(a).cuda() for a in (x, t, w))
    Mp = izb.pad_rows(M)
    buf, asc = torch.full((Mp * K + 32,), 7, dtype=torch.int8, device="cuda"), torch.full((K // 32, Mp), 7.0, device="cuda")
    p = lambda a, o=0: C.c_void_p(a.data_ptr() + o)
    rc = izb.lib().izb_add_norm_quant(p(xd), p(td), p(wd), C.c_float(1e-6), C.c_float(1.0), p(wd), M, Mp, K, p(buf, off), p(asc), None, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    _, raq, rasc, _ = O.add_norm_quant(x, t, w, 1e-6, 1.0, w, Mp=Mp)
    got = buf.cpu().numpy()
    assert (got[off:off + Mp * K].reshape(Mp, K) == raq).all() and (got[:off] == 7).all() and (got[off + Mp * K:] == 7).all()
    assert (bits(asc.cpu().numpy()) == bits(rasc)).all()


# The normalised rows may be written over the input (one block per row then), and a few rows may have any number of padding rows.
@pytest.mark.parametrize("M,K", [(1, 5120), (5, 4096), (8, 12288)])
def test_rmsnorm_quant_in_place(izb, M, K):
    import ctypes as C
    import torch
    rng = np.random.default_rng(M + K)
    x, w = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal(K, dtype=np.float32)
    p = lambda a: C.c_void_p(a.data_ptr())
    for Mp in (16, 1024):
        xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
        aq, asc = torch.full((Mp, K), 7, dtype=torch.int8, device="cuda"), torch.full((K // 32, Mp), 7.0, device="cuda")
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert izb.lib().izb_rmsnorm_quant(p(xd), K, p(wd), C.c_float(1e-6), M, Mp, K, p(xd), p(aq), p(asc), None, st) == 0
        ry, raq, rasc, _ = O.rmsnorm_quant(x, w, 1e-6, Mp=Mp)
        assert (bits(xd.cpu().numpy()) == bits(ry)).all() and (aq.cpu().numpy() == raq).all() and (bits(asc.cpu().numpy()) == bits(rasc)).all()
        assert izb.lib().izb_quantize_act(p(xd), K, M, Mp, K, p(aq), p(asc), None, st) == 0
        qaq, qasc, _ = O.quantize_act(ry, Mp=Mp)
        assert (aq.cpu().numpy() == qaq).all() and (bits(asc.cpu().numpy()) == bits(qasc)).all()


# Few rows go by a thread per value (148 x 8 blocks of one row and 256 columns, with the SwiGLU product four times as many), more by a thread per
# eight: the same bits, also for zeros, infinities, NaN and blocks whose 127 / amax overflows.
@pytest.mark.parametrize("M,K", [(1, 256), (16, 512), (17, 768), (147, 2048), (148, 2048), (591, 2048), (592, 2048)])
def test_quantisers_do_not_depend_on_the_number_of_rows(izb, M, K):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + K)
    x = torch.randn((2500, 2 * K), generator=gen, device="cuda")
    x[0, :32] = 0.0
    x[0, 40], x[0, 70], x[0, 100] = float("inf"), float("nan"), -0.0
    x[0, 128:160] = 1e-44
    x[0, 160:192] = float("nan")
    def same(a, b):
        return torch.equal(a.contiguous().view(torch.int8), b.contiguous().view(torch.int8))
    few, many = izb.quantize_act(x[:M, :K], want_absum=True), izb.quantize_act(x[:, :K], want_absum=True)
    hfew, hmany = izb.swiglu_quant(x[:M], K, want_h=True), izb.swiglu_quant(x, K, want_h=True)
    for f, m in ((few, many), (hfew, hmany)):
        assert same(f[0][:M], m[0][:M]) and not f[0][M:].any()
        assert same(f[1][:, :M], m[1][:, :M]) and f[1].shape[1] == izb.pad_rows(M) and not f[1][:, M:].any()
    assert same(few[2][:, :M], many[2][:, :M]) and not few[2][:, M:].any() and same(hfew[2][:M], hmany[2][:M])


# (a wave holds 148 x 8 blocks of 1024 logits, 148 x 16 blocks of 512 combined values)
@pytest.mark.parametrize("rows,N", [(1184, 1024), (1185, 1024), (600, 4100)])
def test_softcap_of_one_wave_and_more(izb, rows, N):
    import torch
    x = torch.randn(rows, N, generator=torch.Generator().manual_seed(N)) * 40
    got = izb.softcap_rows(x.cuda(), rows, N, 30.0).cpu().double()
    want = 30.0 * torch.tanh(x.double() / 30.0)
    # (x / cap, tanhf and the product: a few units in the last place of values up to 30)
    assert float((got - want).abs().max()) < 8 * 30 * 2.0 ** -24


@pytest.mark.parametrize("T,E", [(148, 8192), (149, 8192), (600, 8196)])
def test_combine_of_one_wave_and_more(izb, T, E):
    import torch
    rng = np.random.default_rng(T)
    x, y = rng.standard_normal((T, E), dtype=np.float32), rng.standard_normal((2 * T, E), dtype=np.float32)
    inv = rng.permutation(2 * T).astype(np.int32)
    out = izb.moe_combine(*(torch.from_numpy(a).cuda() for a in (x, y, inv)), 2)
    assert (bits(out.cpu().numpy()) == bits(O.moe_combine(x, y, inv, 2))).all()
