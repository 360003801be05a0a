"""Room responses whose longest image axis is each of the three in turn, whose
tables do not fit in shared memory (every image from its indices alone), and
whose two rows are one buffer: bit for bit the restatement's."""
import numpy as np
import pytest

from oracle import ref
from tan_b200 import convolution as cv
from tan_b200 import roomgen as rg

pytestmark = pytest.mark.gpu

DAMP = (0.6, 0.2, 0.7, 0.1, 0.5, 0.3)


@pytest.mark.parametrize("size,length", [((3.0, 8.0, 9.0), 9000), ((8.0, 3.0, 9.0), 9001), ((8.0, 9.0, 3.0), 9002),
                                         ((0.03, 40.0, 45.0), 6000), ((5.0, 5.0, 5.0), 40)])
def test_room_paths(tan_ctx, size, length):
    import torch

    src, ears, rate = (size[0] / 3, size[1] / 2, size[2] / 4), (size[0] / 2, size[1] / 3, size[2] / 2, 0.16, 20.0, 5.0, 0.0), 48000
    lp, hp = ref.simple_head_filters(ear_spacing=ears[3])
    el, er, n = ref.room_response(size + DAMP, src, ears, rate, length, lp, hp, 0, 0)
    gen = rg.RoomGenerator(tan_ctx, length + 5)
    L = rg.listener(ears[:3], ears[3], *ears[4:], lp, hp)
    left, right = torch.full((length,), 7.0, device="cuda"), torch.full((length,), 7.0, device="cuda")
    for _ in range(2):
        assert gen.response(rg.Room(*size, *DAMP), rg.Source(*src), L, rate, length, left, right) == 0, cv.last_error()
        assert gen.synchronize() == 0
        assert gen.images() == n
        assert np.array_equal(left.cpu().numpy(), el) and np.array_equal(right.cpu().numpy(), er)
    assert gen.response(rg.Room(*size, *DAMP), rg.Source(*src), L, rate, length, left, left) == 0
    assert gen.synchronize() == 0
    assert np.array_equal(left.cpu().numpy(), er)  # the right ear is written last
    gen.release()
