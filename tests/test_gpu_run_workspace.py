"""The workspace of calls over several blocks is allocated by Init and counted in
the object's device bytes: no call allocates device memory, whatever its length."""
import numpy as np
import pytest

from tan_b200 import convolution as cv
from tests import helpers as H

pytestmark = pytest.mark.gpu


# workspaces well above the 2 MB granularity of the free-memory figure: 32 blocks
# (8 MB), 16 blocks (20 MB) and a non-uniform object's
@pytest.mark.parametrize("method,B,L,C", [(cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, 256, 3000, 64),
                                          (cv.TAN_CONVOLUTION_METHOD_FFT_UNIFORM_PARTITIONED, 1024, 9000, 80),
                                          (cv.TAN_CONVOLUTION_METHOD_FFT_PARTITIONED_NONUNIFORM, 128, 60000, 64)])
def test_calls_allocate_nothing(tan_ctx, method, B, L, C):
    import torch

    x = torch.from_numpy(H.noise(H.rng(5), C, 80 * B)).cuda()
    y = torch.zeros_like(x)
    h = H.irs(H.rng(6), C, L)

    def play(conv, step):
        for k in range(0, 80, step):
            rows = slice(k * B, min(80, k + step) * B)
            rc, done = conv.ProcessDevice([x[c, rows] for c in range(C)], [y[c, rows] for c in range(C)],
                                          rows.stop - rows.start)
            assert rc == 0 and done == rows.stop - rows.start, cv.last_error()
        assert conv.Synchronize() == 0

    outs = []
    for turn in range(2):  # the first object also loads the kernels
        conv = cv.TANConvolution(tan_ctx)
        assert conv.Init(method, L, B, C) == 0 and conv.UpdateResponseTD(h, L) == 0
        play(conv, 1)
        free, held = torch.cuda.mem_get_info()[0], conv.info()["device_bytes"]
        for step in (8, 20, 80):
            play(conv, step)
            if turn:
                assert torch.cuda.mem_get_info()[0] == free
                assert conv.info()["device_bytes"] == held
        outs.append(y.cpu().numpy())
        conv.Release()
    assert np.array_equal(*outs)
