"""The self-test of the bounded waits at limits of the order of the clock's units: it has to report that both ran out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit_ns", [1, 1000, 1024, 3000, 10_000, 40_000, 100_000])
def test_short_limits_run_out(limit_ns):
    from compactattention_b200 import _lib, ops
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    waited = torch.zeros(8, dtype=torch.int64, device="cuda")
    for i in range(8):
        assert _lib.load().ca_selftest_bounded_wait(limit_ns, status[i:].data_ptr(), waited[i:].data_ptr(), ops._stream()) == 0
    assert (status == _lib.CA_STATUS_TIMEOUT).all()
    assert (waited >= limit_ns).all()
