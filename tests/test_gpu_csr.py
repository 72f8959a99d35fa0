"""Row pointers of a receiver index (csrc/csr.cu) against a search: empty lists, empty first, middle and last rows, one row,
both index types, ascending or not, on either side of what one thread block sorts."""
import pytest
import torch

from cuequivariance_b200.channelwise import _CsrCache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n,rows,lo,hi", [(0, 5, 0, 5), (1, 1, 0, 1), (1, 9, 4, 5), (255, 7, 2, 5), (256, 300, 0, 300), (257, 3, 0, 3), (4096, 1999, 10, 1500),
                                          (4097, 1999, 10, 1500), (4000, 65537, 0, 65537)])
@pytest.mark.parametrize("ascending", [True, False])
def test_rows(n, rows, lo, hi, ascending, dtype):
    gen = torch.Generator().manual_seed(n)
    idx = torch.randint(lo, hi, (n,), generator=gen)
    idx = torch.sort(idx).values if ascending else idx
    order, rowptr = _CsrCache().get(idx.to("cuda", dtype), rows)
    ref, perm = torch.sort(idx, stable=True)
    assert torch.equal(rowptr.cpu().long(), torch.searchsorted(ref, torch.arange(rows + 1)))
    assert rowptr.dtype == torch.int32
    if order is None:
        assert bool((idx[1:] >= idx[:-1]).all())
    else:
        assert order.dtype == torch.int32 and torch.equal(order.cpu().long(), perm)
