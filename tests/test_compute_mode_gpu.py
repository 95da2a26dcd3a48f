"""Compute mode: one rank's whole work with every push looped back into its own window (`SoloRankContext`), against the
host model.  Every "peer" contributes this rank's own rows, so a one-shot sum and the rows that the rank owns are those of a
group whose ranks all hold x, and a two-shot row of another owner is the plain decode of x."""
import numpy as np
import pytest
import torch

from fp4_all_reduce_b200 import _native as N
from fp4_all_reduce_b200 import oracle as O
from fp4_all_reduce_b200.parallel.context import SoloRankContext, launch_plan
from fp4_all_reduce_b200.utils import data as D

pytestmark = pytest.mark.gpu

GS = 0.02
QSCALE = 168.0


def _model(x, ranks, inp, epi, res, w):
    """The outputs of every row: those of the sum, and in the two-shot rows of other owners those of x alone."""
    kw = dict(input_kind=inp, epi=epi, res_in=res, weight=w, qscale=QSCALE)
    both = O.allreduce([x] * ranks, algo=1 if ranks > 2 else 0, gs=[GS] * ranks, **kw)
    if ranks > 2:
        alone = O.allreduce([x], algo=0, gs=[GS], **kw)
        for k, v in both.items():
            if v is not None:
                theirs = np.arange(v.shape[0]) % ranks != 0
                v[theirs] = alone[k][theirs]
    return both


@pytest.mark.parametrize("ranks", [2, 4, 8])
@pytest.mark.parametrize("inp", [N.IN_BF16, N.IN_NVFP4])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_one_rank_alone_equals_the_host_model(ranks, inp, epi):
    """Row counts on both sides of the narrow build's limits; at each four calls of changing inputs in one context, so both
    window buffers are armed again and used again."""
    dev = torch.device("cuda", torch.cuda.current_device())
    ctas = torch.cuda.get_device_properties(dev).multi_processor_count
    counts = [1, 7, ctas, ctas + 1, 2 * ctas, 2 * ctas + 1, 4 * ctas, 4 * ctas + 3]
    narrow = {launch_plan(ranks, r, ctas_per_rank=ctas, input=inp, epilogue=epi)["narrow"] for r in counts}
    assert narrow == {0, 1}
    most = max(counts)
    w = D.norm_weight()
    sets = []
    for seed in (1, 2, 3):
        bits = O.bf16_bits(D.partial(most, seed))
        x = bits if inp == N.IN_BF16 else O.encode_static(bits, GS)
        res = D.residual(most, seed=seed)
        want = _model(x, ranks, inp, epi, O.bf16_bits(res), O.bf16_bits(w))
        xd = D.partial(most, seed).to(dev) if inp == N.IN_BF16 else torch.from_numpy(x).to(dev)
        sets.append((xd, res.to(dev), {k: torch.from_numpy(v.view(np.int16) if v.dtype == np.uint16 else v).to(dev)
                                       for k, v in want.items() if v is not None}))
    ctx = SoloRankContext(ranks, most)
    ctx.set_timeout_ms(2000)
    wd = w.to(dev)
    for rows in counts:
        for call in range(4):
            x, res, want = sets[call % 3]
            kw = dict(gs=[GS] * ranks if inp == N.IN_NVFP4 else None, mode=N.MODE_COMPUTE)
            if epi == 0:
                got = {"out": ctx.all_reduce(x[:rows], **kw)}
            else:
                r = res[:rows].clone()
                y, ro = ctx.all_reduce_add_rms_norm(x[:rows], r, wd, epilogue=epi, qscale=QSCALE, **kw)
                assert ro is r
                got = {"out" if epi == 1 else "outq": y, "res_out": ro}
            torch.cuda.synchronize()
            assert ctx.status().ok, (rows, call, ctx.status().describe())
            for k, t in got.items():
                t = t.view(torch.int16) if t.dtype == torch.bfloat16 else t
                assert torch.equal(t, want[k][:rows]), (rows, call, k)
    ctx.close()
