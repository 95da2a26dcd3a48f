"""CPU tests of the op surface: schemas, fake (meta) implementations, argument validation, window sizes."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

from fp4_all_reduce_b200 import _native as N
from fp4_all_reduce_b200.ops import allreduce as A  # noqa: F401  (registers torch.ops.fp4ar)


def test_fake_impls_give_shapes_without_a_gpu():
    with torch._subclasses.FakeTensorMode():
        x = torch.empty(37, 6144, dtype=torch.bfloat16)
        res = torch.empty(37, 6144, dtype=torch.bfloat16)
        w = torch.empty(6144, dtype=torch.bfloat16)
        xq = torch.empty(37, 3456, dtype=torch.uint8)
        assert torch.ops.fp4ar.all_reduce(x, 1).shape == (37, 6144)
        assert torch.ops.fp4ar.all_reduce_nvfp4(xq, [1.0, 2.0], 1).dtype == torch.bfloat16
        assert torch.ops.fp4ar.all_reduce_add_rms_norm(x, res, w, 1e-6, 1.0, 1).shape == (37, 6144)
        assert torch.ops.fp4ar.all_reduce_add_rms_norm_nvfp4(xq, [1.0, 2.0], res, w, 1e-6, 1.0, 1).shape == (37, 6144)
        assert torch.ops.fp4ar.all_reduce_add_rms_norm_quant(x, res, w, 1e-6, 1.0, 2, 1.0, 1).shape == (37, 3456)
        assert torch.ops.fp4ar.all_reduce_add_rms_norm_quant(x, res, w, 1e-6, 1.0, 3, 1.0, 1).shape == (37, 6336)
        q, rs = torch.ops.fp4ar.encode(x)
        assert q.shape == (37, 3456) and rs.shape == (37,)
        assert torch.ops.fp4ar.decode_sum([q, q], [rs, rs]).shape == (37, 6144)
        xk = torch.empty(37, 2048, dtype=torch.bfloat16)
        wt = torch.empty(6144, 2048, dtype=torch.bfloat16)
        assert torch.ops.fp4ar.linear_nvfp4(xk, wt, 0.5).shape == (37, 3456)
        y = torch.ops.fp4ar.linear_all_reduce_add_rms_norm(xk, wt, [0.5, 0.5], res, w, 1e-6, 1.0, 1)
        assert y.shape == (37, 6144) and y.dtype == torch.bfloat16


def test_unknown_context_id_is_an_error():
    with pytest.raises(RuntimeError):
        A._ctx(987654)


def test_window_bytes_and_argument_validation_without_a_gpu(cuda_lib):
    lib = cuda_lib
    assert lib.fp4ar_window_bytes(16384, 6144, 2) == 2 * 2 * 16384 * 3584   # 2 buffers x 2 sources x rows x slot
    assert lib.fp4ar_window_bytes(16384, 6144, 8) % (2 << 20) == 0
    assert lib.fp4ar_window_bytes(16384, 4096, 2) == 0      # only hidden 6144
    assert lib.fp4ar_window_bytes(16384, 6144, 3) == 0      # 1, 2, 4, 8 ranks
    assert lib.fp4ar_window_bytes(0, 6144, 2) == 0
    # a window that is too small or a null pointer is rejected before any CUDA call
    ctx = C.c_void_p()
    ptrs = (C.c_void_p * 2)(0x1000, 0x2000)
    assert lib.fp4ar_create(C.byref(ctx), 0, 2, 0, 1024, 6144, ptrs, 4096) == 1
    ptrs = (C.c_void_p * 2)(None, None)
    assert lib.fp4ar_create(C.byref(ctx), 0, 2, 0, 1024, 6144, ptrs, 1 << 30) == 1
    assert lib.fp4ar_launch(None, None, None) == 1
    assert b"sm_100a" in lib.fp4ar_build_info()


def test_kernel_table_holds_every_product_shape(cuda_lib):
    """Host-side check of the compiled-shape table (no GPU): three-warp teams for every shape, six-warp teams for the
    two-shot shapes of four and eight ranks (their default), nothing else."""
    lib = cuda_lib
    has = lambda *a: int(lib.fp4ar_has_kernel(*a))
    for P, algos in ((1, (0,)), (2, (0, 1)), (4, (0, 1)), (8, (0, 1))):
        for algo in algos:
            assert has(P, algo, 0, 0, 3) > 0, (P, algo)
    for P in (2, 4, 8):
        algo = 0 if P == 2 else 1
        for inp in (0, 1, 2):
            for epi in (0, 1, 2, 3):
                assert has(P, algo, inp, epi, 3) > 0, (P, algo, inp, epi)
                assert has(P, algo, inp, epi, 6) == (3 if P >= 4 else 0), (P, algo, inp, epi)
                assert has(P, algo, inp, epi, 2) == 0
    assert has(4, 0, 0, 0, 6) == 0 and has(1, 0, 0, 1, 6) == 0
    assert lib.fp4ar_default_team_warps(8, 1) == 6 and lib.fp4ar_default_team_warps(2, 0) == 3


def _unbound_context(nranks=2, max_rows=64):
    """A context object with only the fields the argument checks read (no GPU, no native context)."""
    from fp4_all_reduce_b200.parallel.context import Fp4ArContext

    ctx = Fp4ArContext.__new__(Fp4ArContext)
    ctx.nranks, ctx.max_rows, ctx.device, ctx._ctx = nranks, max_rows, torch.device("cuda", 0), None
    return ctx


def test_all_reduce_wrappers_reject_bad_tensors_before_any_launch():
    """Wrong dtype, width, strides, row count, scales or device never reach the kernel, which trusts its pointers."""
    ctx = _unbound_context()
    good = torch.zeros(8, 6144, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="bfloat16"):
        ctx.all_reduce(good.float())
    with pytest.raises(ValueError, match="shape"):
        ctx.all_reduce(torch.zeros(8, 4096, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="contiguous"):
        ctx.all_reduce(torch.zeros(8, 2 * 6144, dtype=torch.bfloat16)[:, ::2])
    with pytest.raises(ValueError, match="is on cpu"):
        ctx.all_reduce(good)                                        # a host tensor, context on cuda:0
    with pytest.raises(ValueError, match="shape"):
        ctx.all_reduce(torch.zeros(8, 3000, dtype=torch.uint8), gs=[1.0, 1.0])
    xq = torch.zeros(8, 3456, dtype=torch.uint8)
    with pytest.raises(ValueError, match="gs"):
        ctx.all_reduce(xq)                                          # NVFP4 rows without scales
    with pytest.raises(ValueError, match="gs"):
        ctx.all_reduce(xq, gs=[1.0])                                # one scale per rank
    with pytest.raises(ValueError, match="gs"):
        ctx.all_reduce(xq, gs=[1.0, 0.0])
    with pytest.raises(ValueError, match="max_rows"):
        ctx.all_reduce(torch.zeros(65, 6144, dtype=torch.bfloat16))


def test_companion_tensors_of_the_norm_call_are_checked():
    ctx = _unbound_context()
    ctx.device = torch.device("cpu")            # host tensors pass the device test, so every later check is reached
    x = torch.zeros(8, 6144, dtype=torch.bfloat16)
    res = torch.zeros(8, 6144, dtype=torch.bfloat16)
    w = torch.zeros(6144, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="epilogue"):
        ctx.all_reduce_add_rms_norm(x, res, w, epilogue=7)
    with pytest.raises(ValueError, match="residual must have 8 rows"):
        ctx.all_reduce_add_rms_norm(x, res[:7], w)
    with pytest.raises(ValueError, match="residual_out"):
        ctx.all_reduce_add_rms_norm(x, res, w, residual_out=torch.zeros(8, 6000, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="weight"):
        ctx.all_reduce_add_rms_norm(x, res, w[:100])
    with pytest.raises(ValueError, match="weight"):
        ctx.all_reduce_add_rms_norm(x, res, w.float())
    with pytest.raises(ValueError, match="out must be"):
        ctx.all_reduce_add_rms_norm(x, res, w, epilogue=2, out=torch.zeros(8, 3456, dtype=torch.int8))
    with pytest.raises(ValueError, match="out must have shape"):
        ctx.all_reduce_add_rms_norm(x, res, w, epilogue=3, out=torch.zeros(8, 3456, dtype=torch.uint8))
    with pytest.raises(ValueError, match="out must have 8 rows"):
        ctx.all_reduce(x, out=torch.zeros(9, 6144, dtype=torch.bfloat16))


def test_zero_row_call_and_poisoned_code_have_names():
    assert N.ERROR_NAMES[4] == "context poisoned"
    with pytest.raises(N.ContextPoisoned):
        N.check(4, "fp4ar_launch")


@pytest.fixture(scope="module")
def front(cuda_lib):
    """The native front end on host tensors: what it does before its device checks needs no GPU."""
    try:
        return N.front()
    except (RuntimeError, OSError, ImportError) as e:
        pytest.skip(str(e))


def test_static_scales_are_read_only_for_sources_without_row_scales(front):
    """A list of scales may hold anything in the places of sources that bring row scales, as in `gs[i]` of plain Python."""
    q, rs = torch.zeros(3, 3456, dtype=torch.uint8), torch.ones(3)
    for gs in ([None, 0.5], ("unused", 0.5), {1: 0.5}, torch.tensor([float("nan"), 0.5])):
        for fn in (front.decode_sum, front.reduce_reencode):
            with pytest.raises(ValueError, match="CUDA"):          # the first complaint is that these are host tensors
                fn([q, q], [rs, None], gs)
    with pytest.raises(IndexError):
        front.decode_sum([q, q], None, [0.5])
    with pytest.raises(TypeError):
        front.decode_sum([q, q], [None, rs], [None, 0.5])


def test_a_flag_without_a_truth_value_raises_its_own_error(front):
    x, w = torch.zeros(3, 6144, dtype=torch.bfloat16), torch.zeros(6144, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="ambiguous"):
        front.add_rmsnorm(x, x, w, 1e-6, 1.0, 1, 1.0, torch.ones(2), None)
    with pytest.raises(RuntimeError, match="ambiguous"):
        front.gemm(x, x, 1.0, torch.ones(2), None)


def test_every_shape_runs_with_the_teams_it_is_built_for(cuda_lib):
    """The registers of a build are shared out over `max_teams` teams, so that many must fit into a CTA's shared memory."""
    from fp4_all_reduce_b200.parallel.context import launch_plan

    shapes = 0
    for P in (1, 2, 4, 8):
        for algo in (0, 1):
            for inp in (0, 1, 2):
                for epi in (0, 1, 2, 3):
                    for width in (3, 6):
                        teams = int(cuda_lib.fp4ar_has_kernel(P, algo, inp, epi, width))
                        if teams == 0:
                            continue
                        shapes += 1
                        pl = launch_plan(P, 100000, algo=algo, input=inp, epilogue=epi, team_warps=width)
                        assert pl["teams"] == teams and pl["team_warps"] == width and not pl["narrow"], (P, algo, inp, epi, width)
                        assert pl["smem"] <= 227 * 1024
    assert shapes > 60
    assert int(cuda_lib.fp4ar_has_kernel(4, 1, 0, 2, 3)) == 4 and int(cuda_lib.fp4ar_has_kernel(8, 1, 0, 2, 3)) == 3


def test_calls_of_few_rows_take_the_narrow_build(cuda_lib):
    """Two teams of the narrow build need no more trips than the teams of the wide one: up to two rows per CTA, and four where
    the wide build has three teams.  Whoever names a width or a team count gets it."""
    from fp4_all_reduce_b200.parallel.context import launch_plan

    for P, wide in ((1, 3), (2, 3), (4, 6), (8, 6)):
        for rows in (1, 148, 149, 296, 297, 444, 445, 592, 593, 888, 16384):
            for inp, epi in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 3)):
                pl = launch_plan(P, rows, input=inp, epilogue=epi)
                per_cta = -(-rows // 148)
                narrow = per_cta <= 2 or (P >= 4 and per_cta == 4)
                assert bool(pl["narrow"]) == narrow and pl["team_warps"] == (6 if narrow else wide), (P, rows, inp, epi, pl)
                assert pl["teams"] <= per_cta
                if per_cta <= pl["teams"]:
                    assert (pl["lag_owner"], pl["lag_finish"]) == (1, 2)
                assert not launch_plan(P, rows, input=inp, epilogue=epi, team_warps=wide)["narrow"]
                assert not launch_plan(P, rows, input=inp, epilogue=epi, teams=1)["narrow"]


@pytest.mark.parametrize("width", [3, 6])
def test_a_team_width_from_the_environment_holds_for_calls_of_few_rows(cuda_lib, width):
    code = """
from fp4_all_reduce_b200.parallel.context import launch_plan
print([(p["team_warps"], p["narrow"]) for p in (launch_plan(P, r, epilogue=1) for P in (2, 4) for r in (1, 16384))])
"""
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, FP4AR_TEAM_WARPS=str(width)), capture_output=True, text=True,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), timeout=300)
    assert r.returncode == 0, r.stderr
    few = (6, 1) if width == 6 else (3, 0)                    # the narrow build is one of six-warp teams
    assert eval(r.stdout) == [few, (3, 0), few, (width, 0)]   # the wide build of two ranks exists at three warps only
