"""The register-resident recurrence kernels at the edges of their rule: every width bound they are compiled for (k tiles of
a warp, one CTA per head or a cluster), a ragged and a single batch row, one step, more 8-row groups than the GPU holds
clusters (where the tcgen05 kernels take over). Oracle and tolerance are those of test_gpu_parity.py."""

import pytest

from tests import test_gpu_parity

pytestmark = pytest.mark.gpu

WIDTHS = (16, 32, 48, 64, 96, 128, 160, 192, 224, 256)
CELLS = ("lstm", "slstm", "gru", "elman")
SHAPES = [(CELLS[(i + j) % 4], (1, 9, 13, 8)[(i + 2 * j) % 4], (7, 1, 6, 3)[(i + j) % 4], 1 + (i + j) % 3, D, 60 + 4 * i + j, j == 0)
          for i, D in enumerate(WIDTHS) for j in range(4)]
SHAPES += [("lstm", 3, 5, 2, 80, 113, False), ("gru", 2, 4, 1, 200, 114, False)]   # a half-filled last CTA; a width that is padded to 208
# more groups than the GPU holds clusters; 16-unit slices on the tcgen05 side (112)
OVERFLOW = [("lstm", 152, 3, 3, 256, 110, False), ("elman", 2600, 2, 1, 64, 111, False), ("gru", 700, 2, 2, 96, 112, False),
            ("lstm", 200, 4, 6, 112, 115, False)]


@pytest.mark.parametrize("shape", SHAPES + OVERFLOW, ids=lambda s: f"{s[0]}-B{s[1]}-T{s[2]}-N{s[3]}-D{s[4]}")
def test_every_width_bound(shape, cuda_device):
    from flashrnn_b200 import _lib

    cell, B, _, N, D = shape[:5]
    taken = shape not in OVERFLOW
    assert _lib.register_kernels(cell, False, B, N, D + -D % 16) == (taken, taken)
    test_gpu_parity.test_cuda_matches_oracle(shape, cuda_device)
