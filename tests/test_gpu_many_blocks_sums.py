"""The product kernels of calls over several blocks against one-block calls, bit
for bit, with the route checked by the launch count: every tail tiling; the form
for many channels (a warp per 64 bins and all partitions) where a chunk of the
sum ends inside a stage of eight partitions, where its rings of 64 input and 32
IR rows wrap, over one and several CTAs of output groups (36 outputs each), in
both its widths, with parameter and table descriptors, device and host rows; and
staged host rows of 256 KB a block, which take the sequence from eight blocks on."""
import numpy as np
import pytest

from tan_b200 import convolution as cv
from tests import helpers as H

pytestmark = pytest.mark.gpu


def make(ctx, L, B, C, tiling=None):
    conv = cv.TANConvolution(ctx)
    assert conv.Init(cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, L, B, C) == cv.AMF_OK
    if tiling is not None:
        assert conv.tiling(tiling)[0] == cv.AMF_OK
    return conv


def responses(g, C, L):
    return (g.standard_normal((C, L)) * np.exp(-3.0 * np.arange(L) / L) / np.sqrt(L)).astype(np.float32)


def play(conv, xd, B, plan):
    """Device rows; the output and the head launches of the calls."""
    import torch

    C = xd.shape[0]
    y = torch.zeros_like(xd)
    conv.profile_read()
    k = 0
    for n in plan:
        rows = slice(k * B, (k + n) * B)
        rc, done = conv.ProcessDevice([xd[c, rows] for c in range(C)], [y[c, rows] for c in range(C)], n * B)
        assert rc == 0 and done == n * B, cv.last_error()
        k += n
    assert conv.Synchronize() == 0
    return y.cpu().numpy(), conv.profile_read()["head"]["launches"]


def compare(ctx, L, B, C, plan, tiling=None, seed=1):
    """`plan` starts with the block that the responses fade in on."""
    import torch

    g = H.rng(seed)
    assert plan[0] == 1
    n = sum(plan)
    xd = torch.from_numpy(H.noise(g, C, n * B)).cuda()
    h = torch.from_numpy(responses(g, C, L)).cuda()
    torch.cuda.synchronize()
    one, many = make(ctx, L, B, C, tiling), make(ctx, L, B, C, tiling)
    for o in (one, many):
        assert o.UpdateResponseTDDevice(h, L, None, cv.TAN_CONVOLUTION_OPERATION_FLAG_BLOCK_UNTIL_READY) == 0
    y1, heads1 = play(one, xd, B, [1] * n)
    y, heads = play(many, xd, B, plan)
    one.Release()
    many.Release()
    assert np.array_equal(y, y1)
    # two transform launches a sequence, whose workspace holds eight blocks at least
    assert heads1 == n and heads <= 1 + sum(2 * -(-m // 8) for m in plan[1:])


@pytest.mark.parametrize("tiling", range(18))
def test_every_tiling(tan_ctx, tiling):
    compare(tan_ctx, 512 * 29 + 7, 512, 3, [1, 3, 30, 9], tiling, 40 + tiling)   # run_mac_kernel
    compare(tan_ctx, 512 * 29 + 7, 512, 112, [1, 3, 14], tiling, 60 + tiling)    # run_mac_line_kernel


# 126 and 129 partitions in the sum: chunks of 16 and 17 (tiling 0), 8 and 9 (tiling 1)
@pytest.mark.parametrize("tiling", [0, 1])
@pytest.mark.parametrize("L", [512 * 128, 512 * 130 + 1])
def test_many_channels_long_responses(tan_ctx, L, tiling):
    compare(tan_ctx, L, 512, 64, [1, 12, 33, 32], tiling, 80)


# three blocks: the narrow width; 64: two CTAs of output groups
@pytest.mark.parametrize("B,L,C,plan", [(512, 512 * 70 + 3, 112, [1, 3, 3, 5]), (1024, 1024 * 260, 56, [1, 3, 35, 64]),
                                        (256, 256 * 41, 240, [1, 3, 15, 36])])
def test_widths_and_groups(tan_ctx, B, L, C, plan):
    compare(tan_ctx, L, B, C, plan, None, 90)


@pytest.mark.parametrize("C,B,L", [(128, 512, 512 * 37 + 1), (130, 512, 512 * 37 + 1)])
def test_staged_host_rows(tan_ctx, C, B, L):
    """256 KB a block and more: seven blocks go one by one, eight and more as
    launch sequences of what the staging rows hold."""
    g = H.rng(95)
    plan = [1, 8, 7, 21]
    n = sum(plan)
    x, h = H.noise(g, C, n * B), responses(g, C, L)
    got = []
    for calls in ([1] * n, plan):
        conv = make(tan_ctx, L, B, C)
        assert conv.UpdateResponseTD(h, L) == 0
        conv.profile_read()
        y = np.zeros_like(x)
        heads, k = [], 0
        for m in calls:
            xs = np.ascontiguousarray(x[:, k * B:(k + m) * B])
            ys = np.zeros_like(xs)
            rc, done = conv.Process(xs, ys, m * B)
            assert rc == 0 and done == m * B, cv.last_error()
            y[:, k * B:(k + m) * B] = ys
            heads.append(conv.profile_read()["head"]["launches"])
            k += m
        got.append((y, heads))
        conv.Release()
    assert np.array_equal(got[0][0], got[1][0])
    assert got[1][1][2] == 7 and got[1][1][1] < 8 and got[1][1][3] < 21
