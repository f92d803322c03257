"""Predictions written over the records that they are made from, at any
overlap: the same as with buffers of their own."""
import pytest
import torch

from kiraray_gb300 import _lib
from kiraray_gb300.nrc import RECORD_FLOATS, NeuralRadianceCache
from tests.test_nrc_gpu import _records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor_cores", [1, 0])
@pytest.mark.parametrize("n", [1, 127, 129, 5000, 400003])
def test_in_place(krr_lib, cuda, n, tensor_cores):
    cache = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), log2_table_size=14, tensor_cores=tensor_cores)
    rec = torch.from_numpy(_records(n, n)).cuda()
    want = cache.query(rec)
    ends = n * RECORD_FLOATS - 3 * n
    # predictions before the records, over them at the front, in the middle
    # and at the end, and behind them
    for at in (-3 * n, -3 * n + 1, -1, 0, 1, ends // 2, ends, ends + 3 * n - 1, ends + 3 * n):
        buf = torch.zeros(n * RECORD_FLOATS + 6 * n, device="cuda")
        records = buf[3 * n:3 * n + n * RECORD_FLOATS]
        records.copy_(rec.reshape(-1))
        out = buf[3 * n + at:6 * n + at]
        _lib.check(cache.lib.krr_nrc_query(cache._h, records.data_ptr(), n, out.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), "krr_nrc_query")
        assert torch.equal(out.reshape(n, 3), want), at
    assert cache.status() == (0, False)
