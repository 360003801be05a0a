"""Calls over several blocks run as one launch sequence (forward transforms of
every new block, the products of every output block, inverse transforms): the
output and the state left behind equal those of one-block calls bit for bit,
at every block size, at partition counts around the chunks of the sum, at block
counts around a launch's groups, for each kind of row, through swaps and
flushes, and for calls that keep to the one-block path."""
import numpy as np
import pytest

from tan_b200 import convolution as cv
from tests import helpers as H

pytestmark = pytest.mark.gpu

FLUSH = cv.TAN_CONVOLUTION_CHANNEL_FLAG_FLUSH_STREAM
STOP = cv.TAN_CONVOLUTION_CHANNEL_FLAG_STOP_INPUT


def make(ctx, L, B, C, tiling=None):
    conv = cv.TANConvolution(ctx)
    assert conv.Init(cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, L, B, C) == cv.AMF_OK
    if tiling is not None:
        assert conv.tiling(tiling)[0] == cv.AMF_OK
    return conv


def stream(conv, x, B, plan, events, flags):
    """One host-row call per entry of `plan` (blocks per call), with the IR
    updates of `events` and the flags of `flags` at their blocks."""
    y = np.zeros_like(x)
    k = 0
    for n in plan:
        if k in events:
            assert conv.UpdateResponseTD(events[k], events[k].shape[1]) == 0
        xs = np.ascontiguousarray(x[:, k * B:(k + n) * B])
        ys = np.zeros_like(xs)
        rc, done = conv.Process(xs, ys, n * B, flags.get(k))
        assert rc == 0 and done == n * B, cv.last_error()
        y[:, k * B:(k + n) * B] = ys
        k += n
    return y


@pytest.mark.parametrize("B,L,C", [(32, 32, 1), (32, 3000, 3), (64, 200, 2), (128, 128 * 3, 5), (128, 5000, 130),
                                   (256, 256 * 10, 1), (512, 512 * 11 + 1, 2), (1024, 1024 * 20, 3), (2048, 30000, 2),
                                   (4096, 50000, 1), (8192, 100000, 2)])
def test_many_blocks_equal_one_block_calls(tan_ctx, B, L, C):
    g = H.rng(B + L)
    plan = [2, 3, 12, 1, 13, 9] if B <= 1024 else [2, 1, 5, 4]
    n = sum(plan)
    x = H.noise(g, C, n * B)
    events = {0: H.irs(g, C, L), plan[0] + plan[1]: H.irs(g, C, L)}  # at a call's first block
    one, many = make(tan_ctx, L, B, C), make(tan_ctx, L, B, C)
    y1 = stream(one, x, B, [1] * n, events, {})
    y = stream(many, x, B, plan, events, {})
    assert np.array_equal(y, y1)
    one.Release()
    many.Release()


@pytest.mark.parametrize("tiling", [0, 1, 3, 5, 9, 12])  # 8, 16, 32 chunks; 4 chunks and the bulk pipeline: one-block path
def test_many_blocks_with_each_chunking(tan_ctx, tiling):
    g = H.rng(900 + tiling)
    B, L, C, plan = 256, 256 * 70 + 9, 2, [40, 30, 1, 66]
    n = sum(plan)
    x = H.noise(g, C, n * B)
    events = {0: H.irs(g, C, L)}
    one, many = make(tan_ctx, L, B, C, tiling), make(tan_ctx, L, B, C, tiling)
    y1 = stream(one, x, B, [1] * n, events, {})
    y = stream(many, x, B, plan, events, {})
    assert np.array_equal(y, y1)
    one.Release()
    many.Release()


def test_many_blocks_flags_and_snapshot(tan_ctx):
    """Flushes at a call's first block, a ring-out (one-block path) and a channel
    that starts again from silence; then both objects hold the same state."""
    g = H.rng(31)
    B, L, C, plan = 128, 128 * 12 + 5, 3, [6, 4, 8, 30, 5, 20]
    starts = np.cumsum([0] + plan)
    x = H.noise(g, C, starts[-1] * B)
    per_call = {1: [FLUSH, 0, 0], 3: [0, STOP, 0]}
    f_many = {int(starts[i]): np.array(f, np.uint32) for i, f in per_call.items()}
    f_one = {int(starts[i]) + b: np.array(f, np.uint32) for i, f in per_call.items() for b in range(plan[i])}
    one, many = make(tan_ctx, L, B, C), make(tan_ctx, L, B, C)
    events = {0: H.irs(g, C, L), int(starts[4]): H.irs(g, C, L)}
    y1 = stream(one, x, B, [1] * int(starts[-1]), events, f_one)
    y = stream(many, x, B, plan, events, f_many)
    assert np.array_equal(y, y1)
    rc, snap = many.Snapshot()
    assert rc == 0
    third = make(tan_ctx, L, B, C)
    assert third.Restore(snap) == 0
    x2 = H.noise(g, C, 4 * B)
    y2 = stream(one, x2, B, [1] * 4, {}, {})
    assert np.array_equal(stream(third, x2, B, [1, 3], {}, {}), y2)
    assert np.array_equal(stream(many, x2, B, [4], {}, {}), y2)
    for o in (one, many, third):
        o.Release()


@pytest.mark.parametrize("C", [2, 129])
def test_many_blocks_device_rows(tan_ctx, C):
    """Device rows off the 8-byte grid, null rows, in place, and output rows
    that overlap other input rows (one-block path)."""
    import torch

    g = H.rng(77)
    B, L, n = 256, 256 * 9, 19
    x = H.noise(g, C, n * B)
    h = H.irs(g, C, L)

    def run(step, place, null_in=False):
        conv = make(tan_ctx, L, B, C)
        assert conv.UpdateResponseTD(h, L) == 0
        wide = torch.zeros((C, n * B + 2 * B + 1), device="cuda")
        wide[:, 1:1 + n * B] = torch.from_numpy(x).cuda()
        out = torch.zeros_like(wide)
        base, size = wide.data_ptr(), wide.stride(0) * 4
        obase = {"apart": out.data_ptr() + 4, "same": base + 4, "shifted": base + 4 + 4 * B}[place]
        for k in range(0, n, step):
            m = min(step, n - k)
            xi = [base + 4 + c * size + 4 * k * B if not (null_in and c == 1) else None for c in range(C)]
            yo = [obase + c * size + 4 * k * B if not (null_in and c == 0) else None for c in range(C)]
            rc, done = conv.ProcessDevice(xi, yo, m * B)
            assert rc == 0 and done == m * B
        assert conv.Synchronize() == 0
        conv.Release()
        return (out if place == "apart" else wide).cpu().numpy()

    for place, null_in in (("apart", False), ("apart", True), ("same", False), ("shifted", False)):
        assert np.array_equal(run(n, place, null_in), run(1, place, null_in)), (place, null_in)
