"""unpack_int4_split on both sides of the size from which it takes 128-row tiles
(40 tiles of 128 rows x 32 channels, 592 for float32), with ragged rows and
channels: the comparison is that of the tile tests."""

import pytest
import test_copy_tiles as tiles
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,npkt,nant,nchan", [
    (torch.int8, 312, 16, 32), (torch.int8, 314, 16, 31), (torch.float16, 20, 64, 97),
    (torch.float16, 43, 12, 321), (torch.float16, 130, 4, 255), (torch.float32, 147, 64, 255),
    (torch.float32, 148, 64, 255), (torch.float32, 149, 68, 250)])
def test_unpack(dtype, npkt, nant, nchan):
    tiles.test_unpack(dtype, npkt, nant, nchan)
