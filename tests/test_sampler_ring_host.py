"""What a draw asks of the ring that it is given, on the host: everything the kernel reads or writes has to be there."""
import pytest
import torch

from mynah_slm_b200.ops.kernels import Ring
from mynah_slm_b200.ops.lib import KernelError


def _ring(rows=4, stride=8, counts=4, heads=4, dtype=torch.int32):
    return torch.zeros((rows, stride), dtype=torch.int32), torch.zeros(counts, dtype=dtype), torch.zeros(heads, dtype=torch.int32)


def test_a_ring_that_fits_is_taken():
    Ring(*_ring()).check(torch.zeros(8), 4, False)
    Ring(*_ring()).check(torch.zeros(8), 9, True)                    # rows go by slot: more rows than slots is the caller's business


@pytest.mark.parametrize("parts", [_ring(counts=3), _ring(heads=3), _ring(heads=1, counts=1), _ring(dtype=torch.int64),
                                   (torch.zeros((8, 4), dtype=torch.int32).t(),) + _ring()[1:]])
def test_parts_that_do_not_fit_are_refused(parts):
    with pytest.raises(KernelError):
        Ring(*parts)


@pytest.mark.parametrize("params,rows", [(7, 4), (8, 5)])
def test_a_draw_that_does_not_fit_is_refused(params, rows):
    with pytest.raises(KernelError):
        Ring(*_ring()).check(torch.zeros(params), rows, False)
