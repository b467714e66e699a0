"""What a draw asks of the ring that it is given, on the host: everything the kernel reads or writes has to be there."""
import pytest
import torch

from mynah_slm_b200.ops.kernels import _check_ring
from mynah_slm_b200.ops.lib import KernelError


def _ring(rows=4, stride=8, counts=4, heads=4, dtype=torch.int32):
    return torch.zeros((rows, stride), dtype=torch.int32), torch.zeros(counts, dtype=dtype), torch.zeros(heads, dtype=torch.int32)


def test_a_ring_that_fits_is_taken():
    _check_ring(_ring(), torch.zeros(8), 4, False)
    _check_ring(_ring(), torch.zeros(8), 9, True)                    # rows go by slot: more rows than slots is the caller's business


@pytest.mark.parametrize("ring,params,rows", [(_ring(counts=3), 8, 4), (_ring(heads=3), 8, 4), (_ring(heads=1, counts=1), 8, 1),
                                              (_ring(dtype=torch.int64), 8, 4), (_ring(), 7, 4), (_ring(), 8, 5), (_ring()[:2], 8, 4)])
def test_a_ring_that_does_not_fit_is_refused(ring, params, rows):
    with pytest.raises(KernelError):
        _check_ring(ring, torch.zeros(params), rows, False)
