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
