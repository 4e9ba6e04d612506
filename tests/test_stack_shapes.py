"""A stack prepares a block's weights while the block before runs only where a fault in them would have shown in the first block."""
import copy

import numpy as np

from localfold_b200 import EncodedTensor
from localfold_b200.stack import _same_shapes


def _block(**change):
    b = {"heads": np.int64(4), "gate": None, "bias": [0.0, 1.0], "linear": np.zeros((4, 8), np.float32),
         "coded": EncodedTensor(bytes(64), 41, 43, 32, (4, 8)), "norm": {"scale": np.ones(8, np.float32)}}
    b.update(change)
    return b


def test_blocks_of_one_layout():
    assert _same_shapes([_block()])
    assert _same_shapes([_block(), copy.deepcopy(_block()), _block(linear=np.ones((4, 8), np.float32), bias=np.zeros(2))])


def test_blocks_of_different_layouts():
    for change in ({"heads": np.int64(8)}, {"heads": 4.5}, {"gate": np.zeros(8, np.float32)}, {"bias": [0.0]}, {"linear": np.zeros((8, 4), np.float32)},
                   {"coded": EncodedTensor(bytes(60), 41, 43, 32, (4, 8))}, {"coded": EncodedTensor(bytes(64), 40, 43, 32, (4, 8))},
                   {"coded": EncodedTensor(bytes(64), 41, 43, 32, (4, 8), block=64)}, {"norm": {"scale": np.ones(4, np.float32)}}, {"extra": 1}):
        assert not _same_shapes([_block(), _block(**change)]), change
