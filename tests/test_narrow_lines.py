"""The amounts of work from which "auto" calls on narrow frames leave the exact
kernel, which needs no workspace: later where the call prepares its centers."""
import pytest

AUTO = 2


@pytest.mark.parametrize("n,d,k,narrow", [
    (7048, 19, 986, False), (73734, 5, 980, False), (150_000, 3, 500, False), (14_000, 30, 980, False),
    (75_000, 5, 1400, True), (2_000_003, 4, 500, True), (20_000, 30, 980, True)])
def test_single_calls(kmlib, n, d, k, narrow):
    assert (kmlib.km_assign_workspace_size(n, d, k, AUTO) > 0) == narrow


@pytest.mark.parametrize("n,d,k,narrow", [
    (7048, 19, 986, False), (40_000, 3, 980, False), (20_000, 19, 980, True), (20_000, 15, 980, True),
    (14_000, 19, 980, False)])
def test_lloyd_runs(kmlib, n, d, k, narrow):
    # the changed labels of a narrow run take 12 bytes per frame
    size = kmlib.km_lloyd_workspace_size(n, d, k, AUTO) - kmlib.km_lloyd_workspace_size(n, d, k, 0)
    assert (size >= 12 * n) == narrow
