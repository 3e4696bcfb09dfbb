"""The table rows of the cooperative kernels when they stop coming: the waits give up, in all lanes and
warps of the block (none goes on while another waits), and the kernel ends with its status."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("feed", [False, True])
@pytest.mark.parametrize("chunks", [0, 1, 2, 3, 6])
def test_rows_that_stop_coming(feed, chunks):
    from cmaq_gb300 import _lib
    assert _lib.starved_rows(feed, chunks) == [chunks == 6] * (32 if feed else 96)   # four chunks are taken
