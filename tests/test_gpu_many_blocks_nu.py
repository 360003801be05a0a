"""Non-uniform methods on device rows over several blocks per call (level by
level in one launch sequence): the output equals that of one-block calls bit for
bit -- at every block size, for calls that start and end anywhere within the
levels' periods, through IR swaps and flushes, for explicit schedules (several
levels with work items, single-partition levels, sizes that grow by more than
two), off the 8-byte grid, with null rows, in place and with rows that overlap."""
import numpy as np
import pytest

from tan_b200 import convolution as cv
from tests import helpers as H

pytestmark = pytest.mark.gpu

FLUSH = cv.TAN_CONVOLUTION_CHANNEL_FLAG_FLUSH_STREAM
STOP = cv.TAN_CONVOLUTION_CHANNEL_FLAG_STOP_INPUT
METHOD = cv.TAN_CONVOLUTION_METHOD_FFT_PARTITIONED_NONUNIFORM


def make(ctx, L, B, C, levels=None):
    conv = cv.TANConvolution(ctx)
    rc = conv.InitNonUniform(METHOD, L, B, C, levels) if levels else conv.Init(METHOD, L, B, C)
    assert rc == cv.AMF_OK, cv.last_error()
    return conv


def stream(conv, x, B, plan, events, flags, place="apart", nulls=False):
    import torch

    C, T = x.shape
    wide = torch.zeros((C, T + B + 1), device="cuda")
    wide[:, 1:1 + T] = torch.from_numpy(x).cuda()
    out = torch.zeros_like(wide)
    size = wide.stride(0) * 4
    xi = wide.data_ptr() + (4 if place != "aligned" else 8)
    yo = {"apart": out.data_ptr() + 4, "aligned": out.data_ptr() + 8, "same": xi, "shifted": xi + 4 * B}[place]
    k = 0
    for n in plan:
        if k in events:
            assert conv.UpdateResponseTD(events[k], events[k].shape[1]) == 0
        ins = [None if nulls and c == 1 else xi + c * size + 4 * k * B for c in range(C)]
        outs = [None if nulls and c == 0 else yo + c * size + 4 * k * B for c in range(C)]
        rc, done = conv.ProcessDevice(ins, outs, n * B, flags.get(k))
        assert rc == 0 and done == n * B, cv.last_error()
        k += n
    assert conv.Synchronize() == 0
    return (out if place in ("apart", "aligned") else wide).cpu().numpy()


CASES = [
    (128, 40000, 3, None, [1, 70, 3, 4, 37, 64, 2, 128, 9]),
    (128, 1 << 19, 2, None, [130, 7, 128, 261]),
    (256, 60000, 2, None, [5, 33, 20, 4, 64]),
    (512, 90000, 2, None, [4, 9, 30, 1, 8]),
    (1024, 90000, 1, None, [4, 6, 13]),
    (2048, 150000, 1, None, [5, 4, 7]),
    (128, 30000, 2, [(128, 2), (256, 9), (1024, 12), (4096, 4)], [9, 8, 40, 33]),  # items in periods of 2, 8 blocks
    (128, 30000, 2, [(128, 2), (256, 1), (512, 14), (2048, 11)], [9, 50, 4, 33]),  # and of 4 and 16
    (128, 40000, 2, [(128, 8), (1024, 1), (2048, 20)], [9, 40, 33]),               # work items in the base level
    (256, 70000, 2, [(256, 2), (512, 3), (2048, 1), (4096, 17)], [21, 40, 16, 3]),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_many_blocks_equal_one_block_calls(tan_ctx, case):
    B, L, C, levels, plan = CASES[case]
    g = H.rng(700 + case)
    n = sum(plan)
    x = H.noise(g, C, n * B)
    events = {0: H.irs(g, C, L), plan[0]: H.irs(g, C, L), sum(plan[:3]): H.irs(g, C, L)}
    one, many = make(tan_ctx, L, B, C, levels), make(tan_ctx, L, B, C, levels)
    y1 = stream(one, x, B, [1] * n, events, {})
    assert np.array_equal(stream(many, x, B, plan, events, {}), y1)
    one.Release()
    many.Release()


@pytest.mark.parametrize("place,nulls", [("apart", True), ("aligned", False), ("same", False), ("shifted", False)])
def test_many_blocks_rows_and_flags(tan_ctx, place, nulls):
    g = H.rng(750)
    B, L, C, plan = 128, 40000, 3, [40, 30, 6, 50, 21]
    starts = np.cumsum([0] + plan)
    x = H.noise(g, C, int(starts[-1]) * B)
    per_call = {1: [FLUSH, 0, 0], 2: [0, 0, STOP], 3: [0, FLUSH, 0]}
    f_many = {int(starts[i]): np.array(f, np.uint32) for i, f in per_call.items()}
    f_one = {int(starts[i]) + b: np.array(f, np.uint32) for i, f in per_call.items() for b in range(plan[i])}
    events = {0: H.irs(g, C, L), int(starts[3]): H.irs(g, C, L)}
    one, many = make(tan_ctx, L, B, C), make(tan_ctx, L, B, C)
    y1 = stream(one, x, B, [1] * int(starts[-1]), events, f_one, "apart" if place == "same" else place, nulls)
    if place == "same":
        y1[:, 1 + x.shape[1]:] = 0
    assert np.array_equal(stream(many, x, B, plan, events, f_many, place, nulls), y1)
    one.Release()
    many.Release()


@pytest.mark.parametrize("B,levels", [(128, [(128, 2), (256, 1), (512, 1), (1024, 7), (2048, 1), (8192, 3)]),
                                      (256, [(256, 2), (512, 1), (1024, 1), (2048, 7), (4096, 1), (16384, 2)])])
def test_levels_that_grow_by_more_than_two(tan_ctx, B, levels):
    """Calls that start where a small level's next output lies behind a larger
    one's: the larger one's rings hold samples that the smaller one's heads of the
    same call also add to."""
    g = H.rng(780 + levels[-1][0])
    C, L = 2, sum(b * k for b, k in levels)
    plan = [9, 14, 6, 17, 5, 30, 11, 8, 23, 7, 13, 64, 19, 12]
    n = sum(plan)
    x = H.noise(g, C, n * B)
    events = {0: H.irs(g, C, L), plan[0] + plan[1]: H.irs(g, C, L)}
    one, many = make(tan_ctx, L, B, C, levels), make(tan_ctx, L, B, C, levels)
    y1 = stream(one, x, B, [1] * n, events, {})
    assert np.array_equal(stream(many, x, B, plan, events, {}), y1)
    one.Release()
    many.Release()
