"""The tensor-core kernels' tile widths, the training step's one launch for every layer
(sums of the weight-gradient CTAs, Adam, the two BF16 copies) and the input packing where x
starts off a 16-byte boundary."""
import numpy as np
import pytest

import cnn_oracle as N
import test_cnn

LR = 1e-3


def _batch(shape, seed):
    import torch

    rng = np.random.default_rng(seed)
    x = torch.from_numpy(rng.standard_normal(shape + (N.IN_REAL,)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal(shape + (3,)).astype(np.float32)).cuda()
    return x, t


def _weights():
    """Mask of the vector's weights (the biases are not trained)."""
    out = []
    for ci, co, _ in N.LAYERS:
        out += [np.ones(co * 9 * ci, bool), np.zeros(co, bool)]
    return np.concatenate(out)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 8, 16), (1, 304, 16), (3, 104, 16), (2, 130, 257)],
                         ids=["1-tile", "38-tiles", "39-tiles", "every-sm"])
def test_gpu_step_is_adam_on_the_gradients(sbp, shape):
    """One partial sum, the 38 loaded at a time, one more, and as many as the chip has SMs.
    Two steps against FP64 Adam on the gradients that `gradients` returns for the same weights.
    Tolerance: an update is at most lr in size and takes fewer than 16 FP32 roundings from the
    gradient; the weight itself is rounded once more."""
    B, H, W = shape
    x, t = _batch(shape, 11)
    mask = _weights()
    with sbp.Cnn(H, W, B) as net, sbp.Cnn(H, W, B) as fresh:
        net.set_params(test_cnn._small_params(5).astype(np.float32))
        m = v = 0.0
        for k in (1, 2):
            p = net.get_params().astype(np.float64)
            loss, g = net.gradients(x.data_ptr(), t.data_ptr(), B)
            assert np.any(g[mask])
            assert net.train_step(x.data_ptr(), t.data_ptr(), B, LR) == pytest.approx(loss, rel=1e-5)
            g = np.where(mask, g.astype(np.float64), 0.0)
            b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
            m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
            want = p - LR * (m / (1 - b1**k)) / (np.sqrt(v / (1 - b2**k)) + 1e-8)
            got = net.get_params().astype(np.float64)
            # 1 - b2^k is itself a difference of FP32 values near one: relative error 2^-24 / (k 1e-3)
            tol = 2 * LR * (16 * 2.0**-24 + 2.0**-23 / 1e-3) + np.abs(p) * 2.0**-23
            assert np.all(np.abs(got - want) <= tol), k
        # the copies the kernels read are those of the new weights: same bits as when they are set
        fresh.set_params(net.get_params())
        assert np.array_equal(net.gradients(x.data_ptr(), t.data_ptr(), B)[1][mask],
                              fresh.gradients(x.data_ptr(), t.data_ptr(), B)[1][mask])


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_gpu_unaligned_input_gives_the_same_bits(sbp, offset):
    import torch

    B, H, W = 2, 7, 19
    x, t = _batch((B, H, W), 4)
    shifted = torch.zeros(x.numel() + 4, dtype=torch.float32, device="cuda")
    shifted[offset:offset + x.numel()] = x.reshape(-1)
    out = torch.empty((2, B, H, W, 3), dtype=torch.float32, device="cuda")
    with sbp.Cnn(H, W, B) as net:
        net.set_params(test_cnn._small_params(3).astype(np.float32))
        net.forward(x.data_ptr(), B, out[0].data_ptr())
        net.forward(shifted.data_ptr() + 4 * offset, B, out[1].data_ptr())
    assert torch.any(out[0] != 0) and torch.equal(out[0], out[1])


# 8, 16 and 32 pixels wide; every SM's weight-gradient CTA with a second tile at width 16;
# an image smaller than a tile
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 10, 8), (1, 8, 48), (1, 4, 33), (9, 8, 272), (1, 1, 1)],
                         ids=["8-wide", "16-wide", "32-wide", "153-tiles", "1-pixel"])
def test_gpu_tile_widths_match_oracle(sbp, shape):
    test_cnn.test_gpu_forward_and_gradients_match_oracle(sbp, shape)
