"""Products inside a stream capture that are the first of their kind in the process: nothing may allocate there, and a replayed graph
may rely on no block that a later call gives back.  Each case is a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRELUDE = """
import numpy as np, torch
import arcinferzero_b200 as izb
from arcinferzero_b200 import synth as S

def captured(call):
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call()
    return graph

def rel(a, b):
    return float((a.double() - b.double()).abs().max() / b.double().abs().max())
"""


def run(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr


def test_first_call_is_a_captured_gemv():
    """Q6_K at three rows: a kernel with bounded waits whose first call in the process is in a capture."""
    run("""
N, K, T = 256, 768, 3
W = izb.Weight(14, S.make_weight(14, N, K, 1), N, K)
aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(T, K, 2)).cuda())
out = torch.zeros((T, N), device="cuda")
graph = captured(lambda: izb.gemv(W, aq, asc, T, out=out))
graph.replay()
torch.cuda.synchronize()
got = out.clone()
assert rel(got, izb.gemm(W, aq, asc, M=T, impl=izb.GEMM_CORE)[:T]) < 1e-5 and izb.device_status(0) == 0
print("done")
""")


@pytest.mark.parametrize("qt", [12, 14, 13])
def test_weights_are_whole_when_created(qt):
    """A product on another stream right behind the creation of a weight from pageable memory."""
    run(f"""
qt, N, K = {qt}, 4096, 4096
rows = S.make_weight(qt, N, K, 1)
aq, asc, _ = izb.quantize_act(torch.from_numpy(S.make_act(2, K, 2)).cuda())
torch.cuda.synchronize()
stream, got = torch.cuda.Stream(), []
with torch.cuda.stream(stream):
    for _ in range(4):
        W = izb.Weight(qt, rows, N, K)
        got.append(izb.gemv(W, aq, asc, 2))
        torch.cuda.synchronize()
assert all(torch.equal(g, got[-1]) for g in got)
assert rel(got[0], izb.gemm(W, aq, asc, M=2, impl=izb.GEMM_CORE)[:2]) < 1e-5
print("done")
""")


@pytest.mark.parametrize("qt,N", [(14, 128), (13, 128), (23, 128), (8, 144), (12, 144)])
def test_first_call_is_a_captured_gemm(qt, N):
    """Per-16-scale types and part columns: the tensor-core kernel's arena cannot be made in a capture, the CUDA-core kernel needs none."""
    run(f"""
qt, N, K, T = {qt}, {N}, 1024, 40
W = izb.Weight(qt, S.make_weight(qt, N, K, 1), N, K)
x = torch.from_numpy(S.make_act(T, K, 2)).cuda()
aq, asc, _ = izb.quantize_act(x)
a, b = torch.zeros((48, N), device="cuda"), torch.zeros((48, N), device="cuda")
q = (torch.empty_like(aq), torch.empty_like(asc))
def call():
    izb.matmul(W, aq, asc, T, out=a)
    izb.quant_matmul(W, x, T, out=b, qout=q)
graph = captured(call)
graph.replay()
torch.cuda.synchronize()
want = izb.gemm(W, aq, asc, impl=izb.GEMM_CORE)
assert torch.equal(a, want) and torch.equal(b, want) and torch.equal(q[0], aq)
assert rel(izb.matmul(W, aq, asc, T), want) < 1e-5 and izb.device_status(0) == 0  # (by itself: the arena is made, the tensor cores run)
print("done")
""")


def test_replays_outlive_the_growth_of_an_arena():
    run("""
qt, N, K = 14, 256, 1024
W = izb.Weight(qt, S.make_weight(qt, N, K, 1), N, K)
def operands(T):
    x = torch.from_numpy(S.make_act(T, K, T)).cuda()
    return izb.quantize_act(x)[:2]
aq, asc = operands(40)
out = torch.zeros((48, N), device="cuda")
izb.matmul(W, aq, asc, 40, out=out)
want = out.clone()
graph = captured(lambda: izb.matmul(W, aq, asc, 40, out=out))
for T in (3000, 9000, 20000):  # the arena grows past the graph's block
    big = operands(T)
    izb.matmul(W, *big, T)
    other = torch.full((64 << 20,), 0xFF, dtype=torch.uint8, device="cuda")  # whatever takes a block given back
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want), T
    assert int(other.min()) == 0xFF
assert izb.device_status(0) == 0
print("done")
""")
