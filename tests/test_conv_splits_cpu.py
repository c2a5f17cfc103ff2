"""How a convolution's weight gradient is split over the SMs."""
import pytest

from oxidized_neural_orchestra_b200.models.conv_engine import wgrad_split

SMS = 148


@pytest.mark.parametrize("F,ckk", [(64, 288), (64, 576), (129, 900), (200, 1200), (255, 1152), (256, 1152), (384, 900), (512, 2304), (1024, 9216)])
@pytest.mark.parametrize("rows", [100352, 1 << 20])
def test_long_weight_gradients_use_the_chip(F, ckk, rows):
    tiles = -(-F // 128) * -(-ckk // 128)
    for bf16 in (False, True):
        kw = wgrad_split(bf16, F, ckk, rows, SMS)
        split = kw.get("split_k", 0)
        if not split:           # left to the library: two passes up to an eighth as many tiles as SMs, clusters of 4 above a quarter are few
            assert not bf16 and (8 * tiles <= SMS or 4 * tiles > SMS)
            continue
        width = 256 if kw.get("bn") == 256 else 128
        units = -(-F // 128) * -(-ckk // width) * split
        assert units <= SMS or split <= 3
        assert 2 * units > SMS
        assert F * ckk * split <= 8 << 20 or split == 1      # slabs that fit the workspace


@pytest.mark.parametrize("rows", [64, 640, 6272])
def test_short_weight_gradients_are_the_librarys(rows):
    assert wgrad_split(False, 200, 1200, rows, SMS) == {}
    kw = wgrad_split(True, 200, 1200, rows, SMS)
    assert 1 <= kw["split_k"] <= -(-rows // 64)
