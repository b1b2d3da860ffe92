"""GPU parity of convolutions at the edges of the tile choice: map widths around full rows of pixels, channel blocks that do
and do not fill a K block, several images per tile, wide filters, strides and dilation, many tiles per CTA; bit for bit
against the oracle."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
import cases  # noqa: E402
from bolt_b200 import synth  # noqa: E402
from test_conv_gpu import conv_gpu, oracle_conv  # noqa: E402

pytestmark = pytest.mark.gpu
SCALES = [31.75, -1.0, 640.0]


def check(n, ic, ih, iw, oc, fh, fw, st, pad, dilation=1, u8=False):
    shape = (n, ic, ih, iw, oc, fh, fw, st, pad)
    seed = hash(shape) % 100000
    x = synth.u8(seed, (n, ic, ih, iw))
    w = synth.s8(seed + 1, (oc, ic, fh, fw))
    bias = synth.normal(seed + 2, (oc,))
    xin = cases.to_blocked(x, 16)
    got, sc, _ = conv_gpu(shape, xin, w, bias, 16, u8, True, SCALES, dilation=dilation)
    ref, rsc = oracle_conv(shape, xin, w, bias, 16, u8, True, SCALES, dilation=dilation)
    assert got.tobytes() == ref.tobytes() and np.array(sc, np.float32).tobytes() == rsc.tobytes()


@pytest.mark.parametrize("iw", [3, 7, 13, 14, 15, 16, 28, 29])
@pytest.mark.parametrize("ic", [16, 32, 48, 64, 96, 128, 160])
def test_widths_and_channels(iw, ic):
    check(2, ic, 7, iw, 40, 3, 3, 1, 1)


@pytest.mark.parametrize("n", [1, 3, 5])
@pytest.mark.parametrize("hw", [4, 7, 14])
def test_several_images_per_tile(n, hw):
    check(n, 64, hw, hw, 136, 3, 3, 1, 1, u8=True)
    check(n, 288, hw, hw, 264, 3, 3, 1, 1)


@pytest.mark.parametrize("fh,fw,pad", [(1, 3, 1), (3, 1, 1), (2, 2, 0), (5, 5, 2), (3, 7, 1), (1, 15, 0), (1, 16, 0), (7, 7, 3)])
def test_filter_shapes(fh, fw, pad):
    check(2, 64, 17, 33, 72, fh, fw, 1, pad)
    check(1, 160, 17, 20, 24, fh, fw, 1, pad)


def test_strides_and_dilation():
    for st, dil in ((2, 1), (3, 1), (1, 2), (2, 2)):
        check(2, 96, 19, 21, 48, 3, 3, st, 1, dil)


@pytest.mark.parametrize("batch", [1, 40])
def test_more_tiles_than_ctas(batch):
    """several tiles per CTA, several column blocks"""
    check(batch, 64, 30, 30, 64, 3, 3, 1, 1)
    check(batch, 32, 15, 31, 520, 3, 3, 1, 1, u8=True)
