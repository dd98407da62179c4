"""Single-component record transfers on both sides of the sizes from which host threads take part (16 MiB
of 1,024-byte records for downloads, 64 MiB for uploads), with pageable memory: the exact round trips of
test_gpu_transfers."""
import pytest

import test_gpu_transfers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(23, 23, 24), (24, 23, 24), (38, 39, 38), (40, 39, 38)])
def test_single_component(shape):
    test_gpu_transfers.test_single_component(shape)
