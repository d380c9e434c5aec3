"""The autotuner times block-aligned chunks whatever block sizes a batch mixes."""
import numpy as np
import pytest

import binary2d as b2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32_comp", "fp32_state64"])
def test_mixed_blocks_have_a_height(precision):
    """Blocks of 32^2 beside 128^2 blocks of a mesh on which chunks of 128 rows
    still fill the GPU: the heights end at the small blocks'.  The height that was
    set, chunks of single rows, is not what remains."""
    shapes = [(8, 32), (32, 128)]
    runs = [b2.Run(m, h, p) for m, h, p, _ in (b2.presets.iso_disk(nb, bs, seed=90) for nb, bs in shapes)]
    with b2.Runtime(runs, precision=precision) as rt:
        for k, (nb, bs) in enumerate(shapes):
            cons = np.zeros((nb, nb, bs, bs, 3))
            cons[..., 0], cons[..., 1] = 1.0, 0.1
            rt.upload(k, cons)
        rt.set_tile(0, 1)
        _, h, ms = rt.autotune(fold=1, reps=1)
        assert h in (8, 16, 32)
        assert 0.0 < ms < 1e3
