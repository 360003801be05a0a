"""TIME_DOMAIN at the edges of the FIR kernel's tiles (128 outputs, chunks of
256 taps, steps of 32): ProcessDirect against the restatement within 1e-5 of
output RMS (the bound of test_gpu_time_domain.py), and Process on device rows
in place against the same stream with rows apart, bit for bit; and Process with
blocks longer than the history (the response's length rounded up to a power of
two), which go through it in pieces, against a float64 statement of the circular
history within the same bound."""
import numpy as np
import pytest

from oracle import ref
from tan_b200 import convolution as cv
from tests import helpers as H

pytestmark = pytest.mark.gpu


def make(ctx, L, B, C):
    conv = cv.TANConvolution(ctx)
    assert conv.Init(cv.TAN_CONVOLUTION_METHOD_TIME_DOMAIN, L, B, C) == cv.AMF_OK, cv.last_error()
    return conv


@pytest.mark.parametrize("L", [1, 2, 31, 32, 33, 255, 256, 257, 512, 1000])
def test_direct_tile_edges(tan_ctx, L):
    g = H.rng(400 + L)
    C = 5
    length = 1 << (L - 1).bit_length()
    gpu, oracle = make(tan_ctx, L, 128, C), ref.RefTimeDomain(L, C)
    for i, n in enumerate([1, 31, 127, 128, 129, length, 300, 2]):
        n = min(n, length)
        ir = np.zeros((C, length), np.float32)
        ir[:, :L] = H.irs(g, C, L)
        x = H.noise(g, C, n)
        # whole rows, or ranges that are empty, one tap, and off the grid of four
        nz = None if i % 2 == 0 else np.array(
            [[0, 0], [L // 2, min(L // 2 + 1, L)], [L // 3, L], [0, min(33, L)], [min(5, L), L]], np.int32).reshape(-1)
        y = np.zeros_like(x)
        rc, done = gpu.ProcessDirect(ir, x, y, n, nz)
        rcr, yr, doner = oracle.process_direct(ir, x, nz)
        assert rc == rcr == 0 and done == doner == n, cv.last_error()
        scale = np.sqrt(np.mean(yr.astype(np.float64) ** 2)) + 1e-30
        assert np.max(np.abs(y - yr)) <= 1e-5 * scale
    gpu.Release()


def test_process_in_place_on_device_rows(tan_ctx):
    import torch

    g = H.rng(9)
    C, B, L, nb = 3, 256, 700, 9
    x = H.noise(g, C, nb * B)
    irs = {0: H.irs(g, C, L), 4: H.irs(g, C, L)}
    outs = []
    for place in ("apart", "same"):
        conv = make(tan_ctx, L, B, C)
        xd = torch.from_numpy(x).cuda()
        yd = torch.zeros_like(xd) if place == "apart" else xd
        for k in range(nb):
            if k in irs:
                assert conv.UpdateResponseTD(irs[k], L) == 0
            rc, done = conv.ProcessDevice([xd[c, k * B:(k + 1) * B] for c in range(C)],
                                          [yd[c, k * B:(k + 1) * B] for c in range(C)], B)
            assert rc == 0 and done == B
        assert conv.Synchronize() == 0
        outs.append(yd.cpu().numpy())
        conv.Release()
    assert np.array_equal(outs[0], outs[1])


def long_block_statement(x, calls, B, L, irs):
    """Process calls of `calls` samples over a circular history of N = nextpow2(L)
    that takes N samples at a time; irs: {call: (C, L) response}, crossfaded in
    over the B samples from that call on."""
    C, N = x.shape[0], 1 << (L - 1).bit_length()
    hist, h, new = np.zeros((C, N)), np.zeros((C, N)), None
    y = np.zeros(x.shape)
    fade = pos = 0
    for i, n in enumerate(calls):
        if i in irs:
            new, fade = np.zeros((C, N)), 0
            new[:, :L] = irs[i]
        for at in range(0, n, N):
            m = min(N, n - at)
            hist[:, (pos + np.arange(m)) % N] = x[:, pos:pos + m]
            for j in range(m):
                w = hist[:, (pos + j - np.arange(N)) % N]
                o = np.sum(w * h, axis=1)
                if new is not None:
                    b = np.sum(w * new, axis=1)
                    o = b if fade >= B else b * (fade / B) + o * ((B - fade) / B)
                    fade += 1
                y[:, pos + j] = o
            pos += m
        if new is not None and fade >= B:
            h, new = new, None
    return y


@pytest.mark.parametrize("L", [1, 33, 100, 128])
def test_process_blocks_longer_than_the_history(tan_ctx, L):
    import torch

    g = H.rng(600 + L)
    C, B = 3, 256
    N = 1 << (L - 1).bit_length()
    calls = [B, B, N + 1, B - 3, 2 * N if 2 * N <= B else B, B]
    x = H.noise(g, C, sum(calls))
    irs = {0: H.irs(g, C, L), 2: H.irs(g, C, L)}  # the second one's fade runs over several calls
    exp = long_block_statement(x, calls, B, L, irs)
    bound = 1e-5 * np.sqrt(np.mean(exp ** 2))
    got = {}
    for place in ("host", "apart", "same"):
        conv = make(tan_ctx, L, B, C)
        xd = torch.from_numpy(x).cuda()
        yd = xd if place == "same" else torch.zeros_like(xd)
        y = np.zeros_like(x)
        at = 0
        for i, n in enumerate(calls):
            if i in irs:
                assert conv.UpdateResponseTD(irs[i], L) == 0
            if place == "host":
                ys = np.zeros((C, n), np.float32)
                rc, done = conv.Process(np.ascontiguousarray(x[:, at:at + n]), ys, n)
                y[:, at:at + n] = ys
            else:
                rc, done = conv.ProcessDevice([xd[c, at:at + n] for c in range(C)],
                                              [yd[c, at:at + n] for c in range(C)], n)
            assert rc == 0 and done == n, cv.last_error()
            at += n
        assert conv.Synchronize() == 0
        got[place] = y if place == "host" else yd.cpu().numpy()
        conv.Release()
        assert np.max(np.abs(got[place] - exp)) <= bound, place
    assert np.array_equal(got["host"], got["apart"]) and np.array_equal(got["host"], got["same"])
