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


#        bf16   B     C   H   F    K  S  P  one kernel pays: measured us, one / two
@pytest.mark.parametrize("bf16,B,C,H,F,K,S,P,pays", [
    (False, 128, 64, 4, 256, 3, 1, 1, False), (False, 128, 96, 7, 96, 5, 1, 2, False), (True, 128, 96, 7, 96, 5, 1, 2, False),     # 32.0 / 10.7, 37.0 / 22.3, 24.9 / 17.0
    (True, 113, 128, 6, 32, 3, 2, 1, False), (False, 548, 96, 4, 96, 3, 2, 1, False),                                              # 11.8 / 7.3, 15.6 / 10.2
    (False, 342, 32, 28, 64, 3, 2, 1, True), (True, 2048, 64, 14, 64, 3, 2, 1, True), (False, 64, 64, 14, 64, 3, 2, 1, True),      # 40.4 / 53.7, 58.9 / 72.5, 8.0 / 9.5
    (False, 8, 64, 4, 256, 3, 1, 1, True), (False, 227, 17, 5, 40, 5, 1, 0, True)])                                                # small; channels that end inside a piece
def test_input_gradient_form(bf16, B, C, H, F, K, S, P, pays):
    import torch

    from oxidized_neural_orchestra_b200.ops import _lib
    from oxidized_neural_orchestra_b200.ops import conv as cv

    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    assert cv.dgrad_pays(cv.geom(B, C, H, H, K, S, P), F, torch.bfloat16 if bf16 else torch.float32) is pays


@pytest.mark.parametrize("bf16,B,C,H,F,K,S,P,pays", [
    (False, 16, 20, 12, 40, 5, 1, 0, False), (False, 8, 64, 14, 64, 3, 2, 1, False), (False, 6, 64, 12, 256, 1, 2, 0, False),      # 16.3 / 14.2, 15.7 / 14.9, 11.1 / 8.0
    (True, 16, 20, 12, 40, 5, 1, 0, True), (False, 8, 16, 28, 32, 3, 2, 1, True), (False, 342, 64, 14, 64, 3, 2, 1, True)])        # -, 8.0 / 9.3, 16.9 / 22.5
def test_forward_form(bf16, B, C, H, F, K, S, P, pays):
    import torch

    from oxidized_neural_orchestra_b200.ops import _lib
    from oxidized_neural_orchestra_b200.ops import conv as cv

    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    assert cv.fprop_pays(cv.geom(B, C, H, H, K, S, P), F, torch.bfloat16 if bf16 else torch.float32) is pays
