"""What a box world takes of the device's memory. A box has 27 grid entries of 20 bytes and up to 4 x 27 hash slots of 4, 49
candidates of 12, 8 manifold slots of 2 x 672 (records and keys), 528 (the columns, whose room the contact geometry
shares) and 28, and some 350 of its own: 16.8 KB and a fifth of its hash slots' spare."""
import numpy as np
import pytest
import torch

from shatterforge_b200 import boxes as X

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes,boxes", [(1, 200000), (100, 2000)])
def test_device_bytes_a_box(sf, scenes, boxes):
    first = X.BoxWorld([X.pile(40)], X.box_params())      # (the kernels' code is loaded with their first launch)
    first.step(np.float32(1 / 60))
    piles = [np.tile(X.pile(100), (boxes // 100, 1))] * scenes
    free = torch.cuda.mem_get_info()[0]
    w = X.BoxWorld(piles, X.box_params())
    took = free - torch.cuda.mem_get_info()[0]
    assert took <= 17800 * scenes * boxes, took / (scenes * boxes)
    w.close()
    first.close()
