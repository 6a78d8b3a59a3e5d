"""Bounded waits.  A wait that runs out must not split its warp: the lanes that leave would wait at a barrier of the CTA for lanes that
wait for them (or that issue an instruction which needs all 32), and the kernel would never return.  The sources are checked for
that on the CPU; on the GPU the tensor-core GEMM runs with limits so short that its waits give up at any moment."""
import os
import re

import numpy as np
import pytest

from arcinferzero_b200 import synth as S

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "arcinferzero_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return "\n".join(re.sub(r"//.*", "", line) for line in text.split("\n"))


def test_gemm_roles_wait_as_warps():
    """Producers, MMA issuers and combine warps take the voting wait; only the dequantisers' threads, which issue nothing warp-wide,
    wait one by one."""
    s = source("izb_gemm_tc.cu")
    kernel = s[s.index("gemm_tc_kernel(const __grid_constant__"):s.index("split_reduce_kernel(")]
    deq = kernel.index("} else if (warp < 8)"), kernel.index("setmaxnreg.inc")
    warp_wide = kernel[:deq[0]] + kernel[deq[1]:]
    assert len(re.findall(r"\bmbar_wait_warp\(", warp_wide)) >= 10 and not re.findall(r"\bmbar_wait\(", warp_wide)
    assert not re.findall(r"sync", kernel[deq[0]:deq[1]].replace("setmaxnreg.dec.sync", "").replace("fence_proxy_async", ""))
    assert re.search(r"bool mbar_wait_warp\([^{]*\{.*?__all_sync\(kAll, mbar_test.*?__all_sync\(kAll, mbar_try_wait", s, re.S)


def test_folded_gemm_waits_as_warps():
    """Every role of the folded GEMM issues something warp-wide: there is no wait but the voting ones."""
    s = source("izb_gemm_fold.cu")
    kernel = s[s.index("gemm_fold_kernel(const __grid_constant__"):s.index("int launch(const izb_weight")]
    assert len(re.findall(r"\bmbar_wait_warp\(", kernel)) >= 12 and not re.findall(r"\bmbar_(wait|test|try_wait)\(", kernel)
    assert re.search(r"bool mbar_wait_warp\([^{]*\{.*?__all_sync\(kAll, mbar_test.*?__all_sync\(kAll, mbar_try_wait", s, re.S)
    assert not re.findall(r"\bmbar_(test|try_wait)\(", re.sub(r"__all_sync\(kAll, mbar_(test|try_wait)\(", "", s[s.index("bool mbar_wait_warp("):]).replace("ok &= mbar_test(w[i]", ""))


@pytest.mark.parametrize("name", ["izb_rows.cu", "izb_gemv_stream.cu"])
def test_gemv_rings_wait_as_warps(name):
    """A look at a ring slot's barrier is only ever used through a vote."""
    s = source(name)
    looks = [line for line in s.split("\n") if re.search(r"\btry_wait\(", line) and "bool try_wait" not in line]
    looks += [line for line in s.split("\n") if re.search(r"\bif \(ok\) return base", line)]
    assert all("__all_sync(" in line for line in looks), looks
    assert s.count("__all_sync(") >= 1


@pytest.mark.gpu
@pytest.mark.parametrize("qt,M,N,K", [(12, 300, 272, 1024), (8, 300, 272, 1024), (13, 130, 128, 512), (14, 130, 128, 512), (23, 130, 128, 512), (12, 40, 128, 4096), (8, 40, 128, 4096), (14, 40, 128, 4096)])
def test_waits_that_run_out_at_any_moment(izb, qt, M, N, K):
    """Every element is the right one or was left alone; the next call is whole again."""
    import torch
    W = izb.Weight(qt, S.make_weight(qt, N, K, N + K + qt), N, K)
    Mp = izb.pad_rows(M)
    aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(M, K, M + K)).cuda(), Mp=Mp)
    want = izb.gemm(W, aq, asc, M=M)
    torch.cuda.synchronize()
    assert izb.device_status(0) == 0
    for limit in (1, 2, 3, 5, 8, 16):
        izb.debug_wait_test(limit, -1)
        out = torch.full((Mp, N), float("nan"), device="cuda")
        izb.gemm(W, aq, asc, M=M, out=out)
        torch.cuda.synchronize()
        status = izb.device_status(0)
        kept = torch.isnan(out[:M])
        assert torch.equal(out[:M][~kept], want[:M][~kept]), limit
        assert status != 0 or not bool(kept.any())
    assert torch.equal(izb.gemm(W, aq, asc, M=M)[:M], want[:M])
    assert izb.device_status(0) == 0
    W.close()
