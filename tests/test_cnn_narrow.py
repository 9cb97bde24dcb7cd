"""Images of few columns or rows: the tensor-core kernels' tiles of 64 x 2 pixels (one or two
pixels high), and tiles whose rows run down the image (up to four pixels wide), with sizes one
below, at and above a tile and several tiles per CTA. The oracle test's own tolerances."""
import pytest

import test_cnn


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 64), (2, 1, 65), (1, 2, 63), (3, 1, 7000), (1, 64, 1), (2, 65, 1), (1, 63, 2),
                                   (3, 7000, 1), (1, 32, 3), (2, 33, 4), (1, 31, 4), (40, 513, 3), (2, 3, 40), (2, 9, 5)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gpu_narrow_images_match_oracle(sbp, shape):
    test_cnn.test_gpu_forward_and_gradients_match_oracle(sbp, shape)
