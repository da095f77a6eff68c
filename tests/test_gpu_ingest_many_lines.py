"""An edge list of more than 2^32 lines, nearly all of weight zero: the lines that
drop out need no device memory and no number.  (The arrays are zero pages but for
a few lines.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_lines_than_entries_are_numbered(rfmf, ctx):
    n = 2**32 + 77
    try:
        a, b = np.zeros(n, np.int64), np.zeros(n, np.int64)
    except MemoryError:
        pytest.skip("no address space for the list")
    lines = [3, 10**9, 2**32 + 5, 2**32 + 70]
    a[lines] = [7, 1, 30, 7]          # vertex and weight of the line (a, 0)
    g = rfmf.DeviceGraph.from_edges(ctx, a, b, a)
    off, col, w = g.csr()
    assert g.orig_ids().tolist() == [0, 1, 7, 30]
    assert off.tolist() == [0, 3, 4, 5, 6] and col.tolist() == [1, 2, 3, 0, 0, 0] and w.tolist() == [1, 7, 30, 1, 7, 30]
    g.close()
    a[2**31] = 2**31
    with pytest.raises(rfmf.RfmfError, match="weight at edge 2147483648 does not fit int32"):
        rfmf.DeviceGraph.from_edges(ctx, a, b, a)
