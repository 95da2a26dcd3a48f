"""Argument checks of the native front end: an argument that the kernels could not trust raises by name before any launch."""
import pytest
import torch

from fp4_all_reduce_b200 import _native as N
from fp4_all_reduce_b200.ops import allreduce as A  # noqa: F401  (registers torch.ops.fp4ar)
from fp4_all_reduce_b200.ops import codec
from fp4_all_reduce_b200.ops import gemm as G
from fp4_all_reduce_b200.parallel.context import SoloRankContext

pytestmark = pytest.mark.gpu

ROWS = 8


def _bf16(rows=ROWS, cols=N.HIDDEN, device="cuda"):
    return torch.zeros(rows, cols, dtype=torch.bfloat16, device=device)


def test_norm_takes_only_memory_that_holds_its_rows():
    x, res, w = _bf16(), _bf16(), _bf16(1).view(-1)
    bad_out = {
        1: [_bf16(ROWS - 1), _bf16(device="cpu"), _bf16(ROWS, 2 * N.HIDDEN)[:, ::2]],
        2: [torch.zeros(ROWS, N.QROW_BYTES - 16, dtype=torch.uint8, device="cuda"), torch.zeros(ROWS, N.QROW_BYTES, dtype=torch.uint8)],
        3: [torch.zeros(ROWS, N.QROW_BYTES, dtype=torch.uint8, device="cuda")],
    }
    for epi, outs in bad_out.items():
        for out in outs:
            with pytest.raises(ValueError, match="out must be"):
                codec.add_rmsnorm(x, res, w, epilogue=epi, out=out)
    for bad_w in (_bf16(2).view(-1)[::2], torch.zeros(1, dtype=torch.bfloat16, device="cuda").expand(N.HIDDEN), w.cpu(), w[:100]):
        with pytest.raises(ValueError, match="weight must be"):
            codec.add_rmsnorm(x, res, bad_w)
    with pytest.raises(ValueError, match="residual must have"):
        codec.add_rmsnorm(x, res[:ROWS - 1], w)
    with pytest.raises(ValueError, match="residual"):
        codec.add_rmsnorm(x, res.cpu(), w)
    with pytest.raises(ValueError, match="epilogue"):
        codec.add_rmsnorm(x, res, w, epilogue=4)
    with pytest.raises(ValueError, match="residual must have"):
        torch.ops.fp4ar.add_rms_norm(x, res[:1], w, 1e-6, 1.0)
    out = _bf16(ROWS + 3)                                  # room for more rows than the call has: the rest is left alone
    out.fill_(7)
    y, _ = codec.add_rmsnorm(x + 1, res, w, out=out)
    assert y is out and torch.all(out[ROWS:] == 7) and torch.all(out[:ROWS] != 7)


def test_sources_of_a_sum_bring_enough_row_scales_on_the_same_device():
    q, rs = codec.encode(_bf16() + 1)
    for fn in (codec.decode_sum, codec.reduce_reencode, lambda a, b: torch.ops.fp4ar.decode_sum(a, b)):
        with pytest.raises(ValueError, match="row_scales must have 8 elements"):
            fn([q, q], [rs, rs[:ROWS - 1]])
        with pytest.raises((ValueError, NotImplementedError, RuntimeError)):
            fn([q, q], [rs, rs.cpu()])
        with pytest.raises((ValueError, NotImplementedError, RuntimeError)):
            fn([q, q.cpu()], [rs, rs])
        with pytest.raises(ValueError, match="one shape"):
            fn([q, q[:2]], [rs, rs])
        with pytest.raises(ValueError, match="3456"):
            fn([q[:, :3072].contiguous()], [rs])
    with pytest.raises(ValueError, match="static scale"):
        codec.decode_sum([q])
    with pytest.raises(ValueError, match="1..8"):
        codec.decode_sum([])


@pytest.mark.multigpu
def test_tensors_of_another_device_are_refused():
    x, res, w = _bf16(), _bf16(), _bf16(1).view(-1)
    there = "cuda:1"
    for args in ((x, res.to(there), w), (x, res, w.to(there))):
        with pytest.raises(ValueError, match="is on cuda:1"):
            codec.add_rmsnorm(*args)
    q, rs = codec.encode(x)
    with pytest.raises(ValueError, match="is on cuda:1"):
        codec.decode_sum([q, q.to(there)], [rs, rs])
    with pytest.raises(ValueError, match="is on cuda:1"):
        codec.decode_sum([q, q], [rs, rs.to(there)])
    with pytest.raises(ValueError, match="is on cuda:1"):
        G.gemm_nvfp4(_bf16(ROWS, 64), _bf16(N.HIDDEN, 64, there), 1.0)


def test_gemm_arguments():
    x, wt = _bf16(ROWS, 128), _bf16(N.HIDDEN, 128)
    for bad in ((x[:, :64], wt), (x, wt[:, :64]), (x, wt.cpu()), (x.float(), wt), (x, _bf16(100, 128))):
        with pytest.raises(ValueError):
            G.gemm_nvfp4(*bad, 1.0)
    for out in (torch.zeros(ROWS - 1, N.QROW_BYTES, dtype=torch.uint8, device="cuda"), torch.zeros(ROWS, N.QROW_BYTES, dtype=torch.uint8),
                torch.zeros(ROWS, N.QROW_BYTES, dtype=torch.int8, device="cuda")):
        with pytest.raises(ValueError, match="out must be"):
            G.gemm_nvfp4(x, wt, 1.0, out=out)


def test_a_number_beyond_a_double_is_an_overflow():
    ctx = SoloRankContext(2, ROWS)
    with pytest.raises(OverflowError):
        ctx.all_reduce_add_rms_norm(_bf16(), _bf16(), _bf16(1).view(-1), eps=10**400, mode=N.MODE_COMPUTE)
    ctx.close()


def test_fused_linear_checks_everything_before_it_pushes():
    """A refused call leaves the windows as they were: nothing was pushed that no launch would take."""
    ctx = SoloRankContext(2, ROWS)
    x, wt, res, w = _bf16(ROWS, 128), _bf16(N.HIDDEN, 128), _bf16(), _bf16(1).view(-1)
    window = ctx.window.clone()
    q8 = torch.zeros(ROWS, N.QROW_BYTES, dtype=torch.uint8, device="cuda")
    good = dict(x=x, wt=wt, gs=[1.0, 1.0], residual=res, weight=w)
    for bad in (dict(residual=res[:ROWS - 1]), dict(residual=res.cpu()), dict(weight=w[:64]), dict(weight=w.cpu()), dict(out=_bf16(ROWS - 1)),
                dict(epilogue=2, out=q8[:ROWS - 1]), dict(epilogue=3, out=q8), dict(epilogue=0), dict(gs=[1.0]), dict(gs=[1.0, 0.0]),
                dict(x=x.cpu()), dict(wt=_bf16(256, 128))):
        with pytest.raises(ValueError):
            G.gemm_all_reduce_add_rms_norm(ctx, **{**good, **bad})
    with pytest.raises(ValueError, match="local_q"):
        G.gemm_push(ctx, x, wt, 1.0, local_q=q8[:ROWS - 1])
    torch.cuda.synchronize()
    assert torch.equal(ctx.window, window)
    ctx.close()


def test_context_calls_name_what_is_wrong():
    """What the native front end does not take falls to the wrapper's checks, on CUDA tensors as well."""
    ctx = SoloRankContext(2, ROWS)
    x, res, w = _bf16(), _bf16(), _bf16(1).view(-1)
    q, rs = codec.encode(x + 1)
    kw = dict(mode=N.MODE_COMPUTE)

    def refused(match, fn, *a, **k):
        with pytest.raises(ValueError, match=match):
            fn(*a, **{**kw, **k})

    ar, block = ctx.all_reduce, ctx.all_reduce_add_rms_norm
    refused("must be bfloat16", ar, x.float())
    refused("shape", ar, _bf16(ROWS, 3072))
    refused("contiguous", ar, _bf16(ROWS, 2 * N.HIDDEN)[:, ::2])
    refused("is on cpu", ar, x.cpu())
    refused("max_rows", ar, _bf16(ROWS + 1))
    refused("out must have 8 rows", ar, x, _bf16(ROWS + 1))
    refused("out must be", ar, x, q)
    refused("out is on cpu", ar, x, _bf16(device="cpu"))
    for gs in (None, [1.0], [1.0, 0.0], [1.0, -1.0], [1.0, float("nan")]):
        refused("gs", ar, q, gs=gs)
    refused("residual must have 8 rows", block, x, res[:4], w)
    refused("residual is on cpu", block, x, res.cpu(), w)
    refused("residual_out", block, x, res, w, residual_out=_bf16(ROWS, 3072))
    refused("weight", block, x, res, w.float())
    refused("weight", block, x, res, _bf16(2).view(-1)[::2])
    refused("epilogue", block, x, res, w, epilogue=0)
    refused("out must be", block, x, res, w, epilogue=2, out=x)
    refused("out must have shape", block, x, res, w, epilogue=3, out=q)
    refused("mode=MODE_COMPUTE", ar, x, mode=N.MODE_FUSED)
    assert ctx.status().ok
    ctx.close()


def test_unusual_but_valid_context_calls_equal_the_plain_one():
    import numpy as np

    ctx = SoloRankContext(2, ROWS)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(ROWS, N.HIDDEN, generator=g, device="cuda").to(torch.bfloat16)
    res, w = x + 1, torch.randn(N.HIDDEN, generator=g, device="cuda").to(torch.bfloat16)
    q = codec.encode_static(x, 0.01)
    plain = ctx.all_reduce(q, gs=[0.01, 0.01], mode=N.MODE_COMPUTE)
    for gs in ((0.01, 0.01), np.array([0.01, 0.01]), torch.tensor([0.01, 0.01]), [np.float32(0.01), torch.tensor(0.01)]):
        assert torch.equal(ctx.all_reduce(q, gs=gs, mode=N.MODE_COMPUTE), plain)
    y, r = ctx.all_reduce_add_rms_norm(x, res.clone(), w, mode=N.MODE_COMPUTE)
    weight = torch.nn.Parameter(w.view(1, -1))
    out, res_out = torch.empty_like(x), torch.empty_like(x)
    kept = res.clone()
    y2, r2 = ctx.all_reduce_add_rms_norm(x, kept, weight, eps=np.float64(1e-6), weight_bias=1, out=out, residual_out=res_out, mode=N.MODE_COMPUTE)
    assert y2 is out and r2 is res_out and torch.equal(kept, res) and torch.equal(y, y2) and torch.equal(r, r2)
    empty = ctx.all_reduce(x[:0], mode=N.MODE_COMPUTE)
    assert empty.shape == (0, N.HIDDEN)
    ctx.close()
