"""Device rows whose outputs lie between the inputs of one buffer (in, out, in,
out, ...) are apart: same samples as separate buffers bit for bit, and a call
over several blocks runs as one launch sequence. An output that is another
channel's input row keeps to the one-block path."""
import numpy as np
import pytest

from tan_b200 import convolution as cv
from tan_b200 import engine as eng
from tests import helpers as H

pytestmark = pytest.mark.gpu


def place_rows(x, where):
    """(buffer, input pointers, output pointers, rows of the outputs in it)."""
    import torch

    C, T = x.shape
    buf = torch.zeros((2 * C, T), device="cuda")
    rows = {"apart": (range(C), range(C, 2 * C)), "between": (range(0, 2 * C, 2), range(1, 2 * C, 2)),
            "crossed": (range(C), [(c + 1) % C for c in range(C)])}[where]
    ri, ro = list(rows[0]), list(rows[1])
    buf[ri] = torch.from_numpy(x).cuda()
    return buf, [buf.data_ptr() + r * T * 4 for r in ri], [buf.data_ptr() + r * T * 4 for r in ro], ro


def call(conv, x, where, B, plan):
    buf, xi, yo, ro = place_rows(x, where)
    k = 0
    for n in plan:
        at = 4 * k * B
        rc, done = conv.ProcessDevice([p + at for p in xi], [p + at for p in yo], n * B)
        assert rc == 0 and done == n * B, cv.last_error()
        k += n
    assert conv.Synchronize() == 0
    return buf[ro].cpu().numpy()


@pytest.mark.parametrize("method,B,L", [(cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, 256, 3000),
                                        (cv.TAN_CONVOLUTION_METHOD_FFT_PARTITIONED_NONUNIFORM, 128, 40000),
                                        (cv.TAN_CONVOLUTION_METHOD_TIME_DOMAIN, 256, 700)])
def test_output_rows_between_input_rows(tan_ctx, method, B, L):
    g = H.rng(800 + L)
    C, nb = 3, 66
    direct = method == cv.TAN_CONVOLUTION_METHOD_TIME_DOMAIN
    x, h = H.noise(g, C, nb * B), H.irs(g, C, L)
    out, launches = {}, {}
    for name, where, plan in (("one", "apart", [1] * nb), ("one between", "between", [1] * nb),
                              ("many between", "between", [1] * nb if direct else [nb])):
        conv = cv.TANConvolution(tan_ctx)
        assert conv.Init(method, L, B, C) == 0 and conv.UpdateResponseTD(h, L) == 0
        first = H.noise(H.rng(1), C, B)  # the response's crossfade, in a block of its own
        call(conv, first, where, B, [1])
        conv.profile_read()
        out[name] = call(conv, x, where, B, plan)
        launches[name] = conv.profile_read()["head"]["launches"]
        conv.Release()
    assert np.array_equal(out["one between"], out["one"]) and np.array_equal(out["many between"], out["one"])
    if method == cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED:
        assert launches["one"] == nb and launches["many between"] < nb // 3


def test_crossed_rows_go_block_by_block(tan_ctx):
    """Channel c's output over channel c + 1's input: what one-block calls give."""
    g = H.rng(830)
    B, L, C, nb = 256, 3000, 3, 12
    x, h = H.noise(g, C, nb * B), H.irs(g, C, L)
    launches = {}
    for plan in ([1] * nb, [nb]):
        conv = cv.TANConvolution(tan_ctx)
        assert conv.Init(cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, L, B, C) == 0
        assert conv.UpdateResponseTD(h, L) == 0
        call(conv, H.noise(H.rng(1), C, B), "apart", B, [1])
        conv.profile_read()
        call(conv, x, "crossed", B, plan)
        launches[len(plan)] = conv.profile_read()["head"]["launches"]
        conv.Release()
    assert launches[1] == launches[nb] == nb


def test_engine_rows_between_input_rows(tan_ctx):
    """Level heads and base heads in either order: 2^15 taps, levels due at many blocks."""
    import torch

    g = H.rng(840)
    B, C, L, nb = 128, 2, 1 << 15, 40
    x, h = H.noise(g, C, nb * B), H.irs(g, C, L)
    levels = [(128, 2), (256, 1), (512, 1), (1024, 31)]
    outs = []
    for between in (False, True):
        e = eng.Engine(tan_ctx, B, eng.SPECTRUM_FP32, eng.session_bytes(B, C, L, levels, eng.SPECTRUM_FP32),
                       max_channels=C)
        rc, s = e.open_session_nu(C, L, levels)
        assert rc == 0 and s.update_response_td(h, block_until_ready=True) == 0
        T = nb * B
        buf = torch.zeros((2 * C, T), device="cuda")
        buf[0::2] = torch.from_numpy(x).cuda()
        y = torch.zeros_like(buf)
        dst, at = (buf, 1) if between else (y, 0)
        torch.cuda.synchronize()
        for k in range(nb):
            assert e.process_device(buf.data_ptr() + k * B * 4, dst.data_ptr() + (at * T + k * B) * 4, 2 * T) == 0
        e.synchronize()
        outs.append(dst[at::2].cpu().numpy())
        s.close()
        e.release()
    assert np.array_equal(outs[0], outs[1])
