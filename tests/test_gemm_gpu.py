"""The tcgen05 GEMM with NVFP4 epilogue: accumulators against an FP32 matmul, quantised rows bit for bit
against the host quantiser applied to the kernel's own accumulators, and the fused GEMM -> push -> AllReduce
path on emulated ranks against the host model fed with the kernel's NVFP4 partials."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from fp4_all_reduce_b200 import _native as N
from fp4_all_reduce_b200 import oracle as O
from fp4_all_reduce_b200.ops import gemm as G
from fp4_all_reduce_b200.parallel.context import EmulatedGroup, make_args
from fp4_all_reduce_b200.utils import data as D

pytestmark = pytest.mark.gpu


def _xw(M, K, Nn, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    wt = (torch.randn(Nn, K, generator=g) / K ** 0.5).to(torch.bfloat16).cuda()
    return x, wt


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("M,K,Nn", [(128, 64, 256), (300, 512, 512), (1024, 2048, 6144), (77, 4096, 6144)])
def test_gemm_accumulators_and_quantised_rows(M, K, Nn, pair, monkeypatch):
    monkeypatch.setenv("FP4AR_GEMM_PAIR", str(pair))      # 1: two CTAs per 256 x 256 tile (tcgen05 cta_group::2)
    x, wt = _xw(M, K, Nn, 1)
    gs = G.calibrate_gs(x, wt)
    q, acc = G.gemm_nvfp4(x, wt, gs, want_acc=True)
    torch.cuda.synchronize()
    assert G.gemm_status().code == 0
    ref = x.float() @ wt.float().t()
    err = (acc - ref).abs().max().item()
    assert err <= 2e-3 * ref.abs().max().item() + 1e-4, err
    want = O.encode_static_f32(acc.cpu().numpy(), gs)
    assert np.count_nonzero(q.cpu().numpy() != want) == 0


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("P", [2, 4])
def test_gemm_push_then_allreduce_on_emulated_ranks(P, pair, monkeypatch):
    monkeypatch.setenv("FP4AR_GEMM_PAIR", str(pair))
    _push_then_allreduce(P, 256, 512)


@pytest.mark.parametrize("P,M", [(2, 5), (2, 100), (4, 37), (8, 3), (8, 30)])
def test_gemm_push_of_few_rows(P, M):
    """Pushed rows finished by the narrow build of the AllReduce kernel (one or two rows per CTA)."""
    _push_then_allreduce(P, M, 512)


def _push_then_allreduce(P, M, K):
    g = EmulatedGroup(P, M)
    g.set_timeout_ms(500)
    xs, wts, gss, qs = [], [], [], []
    for r in range(P):
        x, wt = _xw(M, K, N.HIDDEN, 10 + r)
        xs.append(x); wts.append(wt)
        gss.append(G.calibrate_gs(x, wt))
    res = [D.residual(M).cuda() for _ in range(P)]
    res0 = res[0].clone()
    w = D.norm_weight().cuda()
    outs = [torch.zeros(M, N.HIDDEN, dtype=torch.bfloat16, device="cuda") for _ in range(P)]
    for call in range(3):                       # three calls: both window buffers and a reuse
        for r in range(P):
            res[r].copy_(res0)
            lq = torch.empty(M, N.QROW_BYTES, dtype=torch.uint8, device="cuda")
            G.gemm_push(g, xs[r], wts[r], gss[r], two_shot=P > 2, local_rank=r, local_q=lq)
            qs.append(lq)
        g.launch([make_args(x=None, out=outs[r], rows=M, input=N.IN_PUSHED, gs=gss, epilogue=N.EPI_NORM_BF16,
                            res_in=res[r], res_out=res[r], weight=w,
                            algo=N.ALGO_TWOSHOT if P > 2 else N.ALGO_ONESHOT) for r in range(P)])
        torch.cuda.synchronize()
        assert g.status(0).ok, g.status(0).describe()
        partials = [t.cpu().numpy() for t in qs[-P:]]
        exp = O.allreduce(partials, algo=1 if P > 2 else 0, input_kind=1, gs=gss, epi=1, res_in=O.bf16_bits(res0),
                          weight=O.bf16_bits(w))
        for r in range(P):
            assert np.array_equal(O.bf16_bits(outs[r]), exp["out"]), (call, r)
            assert np.array_equal(O.bf16_bits(res[r]), exp["res_out"]), (call, r)
    g.close()


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("M,K", [(1024, 2048), (2048, 512), (1000, 1024), (2300, 320)])
def test_gemm_stream_k_split(M, K, pair, monkeypatch):
    """Tile counts that do not fill the last wave of CTAs run with the K loop cut into equal ranges per CTA: a tile shared
    by two CTAs is summed from a partial accumulator.  Same checks as for whole tiles, over several calls (the partial
    slots and their flags are reused), inside a CUDA graph of back-to-back launches, and against the whole-tile walk."""
    Nn = N.HIDDEN
    x, wt = _xw(M, K, Nn, 3)
    gs = G.calibrate_gs(x, wt)
    ref = x.float() @ wt.float().t()
    tol = 2e-3 * ref.abs().max().item() + 1e-4
    monkeypatch.setenv("FP4AR_GEMM_PAIR", str(pair))
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "0")
    q_plain, acc_plain = G.gemm_nvfp4(x, wt, gs, want_acc=True)
    torch.cuda.synchronize()
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "1")
    for call in range(3):
        q, acc = G.gemm_nvfp4(x, wt, gs, want_acc=True)
        torch.cuda.synchronize()
        assert G.gemm_status().code == 0
        assert (acc - ref).abs().max().item() <= tol
        want = O.encode_static_f32(acc.cpu().numpy(), gs)
        assert np.count_nonzero(q.cpu().numpy() != want) == 0
        # the split changes the order of the FP32 additions, nothing else
        assert (acc - acc_plain).abs().max().item() <= 1e-5 * ref.abs().max().item() + 1e-6
    assert (q != q_plain).float().mean().item() < 0.01
    first = q.clone()
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    outs = [torch.empty_like(q) for _ in range(3)]
    with torch.cuda.stream(st):
        G.gemm_nvfp4(x, wt, gs, out=outs[0])
        st.synchronize()
        with torch.cuda.graph(g, stream=st):
            for o in outs:
                G.gemm_nvfp4(x, wt, gs, out=o)
    for _ in range(2):
        for o in outs:
            o.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert G.gemm_status().code == 0
        for o in outs:
            assert torch.equal(o, first)


def test_gemm_reset_keeps_the_kernel_usable():
    x, wt = _xw(1024, 2048, N.HIDDEN, 5)
    gs = G.calibrate_gs(x, wt)
    q0 = G.gemm_nvfp4(x, wt, gs)
    G.gemm_reset()
    assert G.gemm_status().code == 0
    q1 = G.gemm_nvfp4(x, wt, gs)
    torch.cuda.synchronize()
    assert G.gemm_status().code == 0 and torch.equal(q0, q1)


@pytest.mark.parametrize("M,K,Nn", [(1, 1024, 6144), (8, 64 * 17, 6144), (9, 512, 6144), (64, 2048, 6144), (65, 512, 6144), (127, 8192, 6144),
                                    (24, 64, 6144), (40, 64 * 5, 6144), (56, 64 * 6, 6144), (120, 64 * 3, 6144), (128, 256, 6144), (129, 576, 6144), (200, 128, 6144), (256, 4096, 6144), (257, 64, 6144), (384, 1024, 6144),
                                    (33, 512, 256), (100, 64, 512), (5, 192, 1024), (130, 320, 2048)])
def test_gemm_of_few_rows_equals_the_wide_tiles(M, K, Nn, monkeypatch):
    """Up to 384 rows a CTA takes a narrow tile with its whole K loop: the same chain of MMAs per accumulator as in the
    256-wide tiles that no two CTAs share, so sums and rows are the same bit for bit, and the rows equal the host quantiser on those sums."""
    assert G.gemm_plan(M, Nn, K, torch.cuda.get_device_properties(0).multi_processor_count)["tile_n"] <= 128
    x, wt = _xw(M, K, Nn, 7)
    gs = G.calibrate_gs(x, wt)
    q, acc = G.gemm_nvfp4(x, wt, gs, want_acc=True)
    q2 = G.gemm_nvfp4(x, wt, gs)
    monkeypatch.setenv("FP4AR_GEMM_TILE_N", "256")
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "0")
    wide, wide_acc = G.gemm_nvfp4(x, wt, gs, want_acc=True)
    torch.cuda.synchronize()
    assert G.gemm_status().code == 0
    ref = x.float() @ wt.float().t()
    assert (acc - ref).abs().max().item() <= 2e-3 * ref.abs().max().item() + 1e-4
    assert np.count_nonzero(q.cpu().numpy() != O.encode_static_f32(acc.cpu().numpy(), gs)) == 0
    assert torch.equal(q, q2)
    assert torch.equal(acc, wide_acc) and torch.equal(q, wide)


def _captured_gemm(x, wt, gs, out, stream):
    """A graph of one GEMM and the workspace that its launch took."""
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        G.gemm_nvfp4(x, wt, gs, out=out)
        space = G.gemm_workspace()
    return g, space


def test_split_gemms_that_may_overlap_have_a_workspace_each(monkeypatch):
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "1")
    torch.cuda.synchronize()
    G.gemm_reset()
    streams = [torch.cuda.Stream() for _ in range(11)]
    spaces = []
    for _ in range(2):
        for s in streams:
            with torch.cuda.stream(s):
                spaces.append(G.gemm_workspace())
    assert 0 not in spaces and spaces[:11] == spaces[11:]
    assert len(set(spaces[:8])) == 8 and len(set(spaces[8:11])) == 1 and spaces[8] not in spaces[:8]
    x, wt = _xw(1024, 512, N.HIDDEN, 0)
    gs = G.calibrate_gs(x, wt)
    out = torch.empty(1024, N.QROW_BYTES, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    kept = [_captured_gemm(x, wt, gs, out, streams[0]) for _ in range(3)]
    owned = [space for _, space in kept]
    assert len(set(owned)) == 3 and not set(owned) & set(spaces)
    with torch.cuda.stream(streams[0]):
        assert G.gemm_workspace() == spaces[0]
    seen = set()
    for _ in range(20):                                    # what a graph owned serves another one when it is gone
        g, space = _captured_gemm(x, wt, gs, out, streams[1])
        assert space not in owned
        seen.add(space)
        del g
        torch.cuda.synchronize()
    assert len(seen) < 20
    del kept
    torch.cuda.synchronize()
    G.gemm_reset()


def test_split_gemms_on_many_streams_at_once(monkeypatch):
    """Launches of different inputs on eleven streams (three of them take turns on one workspace) and in graphs replayed on
    others, nothing between them: every result equals the one computed alone."""
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "1")
    G.gemm_reset()
    M, K, n = 1024, 1024, 13
    data, alone, outs = [], [], []
    for i in range(n):
        x, wt = _xw(M, K, N.HIDDEN, 20 + i)
        gs = G.calibrate_gs(x, wt)
        data.append((x, wt, gs))
        alone.append(G.gemm_nvfp4(x, wt, gs).clone())
        outs.append([torch.zeros_like(alone[0]) for _ in range(3)])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(n)]
    graphs = {i: _captured_gemm(*data[i], outs[i][0], streams[i])[0] for i in (11, 12)}
    for rep in range(3):
        for i, (x, wt, gs) in enumerate(data):
            with torch.cuda.stream(streams[i]):
                if i in graphs:
                    outs[i][0].zero_()
                    graphs[i].replay()
                    outs[i][rep].copy_(outs[i][0])
                else:
                    G.gemm_nvfp4(x, wt, gs, out=outs[i][rep])
    torch.cuda.synchronize()
    assert G.gemm_status().code == 0
    for i in range(n):
        for o in outs[i]:
            assert torch.equal(o, alone[i]), i
    graphs.clear()
    torch.cuda.synchronize()
    G.gemm_reset()


@pytest.mark.parametrize("M", [16, 1024])
def test_first_gemm_of_a_process_may_be_captured(M):
    """Nothing that the first call sets up (status block, workspace, shared-memory limits) needs a call outside the capture."""
    code = f"""
import torch
from fp4_all_reduce_b200.ops import gemm as G
x = torch.randn({M}, 2048, device="cuda").to(torch.bfloat16)
wt = torch.randn(6144, 2048, device="cuda").to(torch.bfloat16)
out = torch.zeros({M}, 3456, dtype=torch.uint8, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    G.gemm_nvfp4(x, wt, 0.05, out=out)
g.replay()
torch.cuda.synchronize()
assert G.gemm_status().code == 0 and torch.equal(out, G.gemm_nvfp4(x, wt, 0.05)) and out.any()
"""
    env = dict(os.environ, FP4AR_GEMM_STREAM_K="1") if M > 384 else dict(os.environ)
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


class _Words:
    """`n` 32-bit words of device memory at an address, for torch.as_tensor."""

    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (address, False), "version": 3}


@pytest.mark.parametrize("pair", [0, 1])
def test_a_hand_off_that_never_comes_ends_with_a_status(pair, monkeypatch):
    """A flag that is neither "free" nor "written" lets the wait of its producer and of its consumer run out (2 s): the launch
    reports it and ends, and after a reset the same call gives the same rows as before."""
    monkeypatch.setenv("FP4AR_GEMM_STREAM_K", "1")
    monkeypatch.setenv("FP4AR_GEMM_PAIR", str(pair))
    x, wt = _xw(1024, 1024, N.HIDDEN, 4)
    gs = G.calibrate_gs(x, wt)
    good = G.gemm_nvfp4(x, wt, gs).clone()
    torch.cuda.synchronize()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    flags = torch.as_tensor(_Words(G.gemm_workspace() + sms * 128 * 256 * 4, 4 * sms), device="cuda")
    assert not flags.any()
    unit = 8                                  # an even CTA: the leader where CTAs work in pairs
    flags[4 * unit] = 2
    G.gemm_nvfp4(x, wt, gs)
    torch.cuda.synchronize()
    st = G.gemm_status()
    assert st.code == 2 and st.detail in (16 + 5, 16 + 6) and st.count >= 1
    del flags
    G.gemm_reset()
    for _ in range(2):
        assert torch.equal(G.gemm_nvfp4(x, wt, gs), good)
    torch.cuda.synchronize()
    assert G.gemm_status().code == 0
