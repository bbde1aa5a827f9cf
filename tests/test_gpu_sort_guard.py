"""A node sort whose bounded wait ran out leaves keys in no order.  The kernels
queued behind it form no work items, empty lists and no entries (in bounds for
any keys), so that the host can report the time-out."""
import pytest

import _device_check

pytestmark = pytest.mark.gpu


def test_no_lists_from_unsorted_keys(native_lib, tmp_path):
    assert _device_check.run("sort_guard_check", tmp_path).strip() == "ok"
