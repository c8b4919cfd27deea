"""The training step at batches whose row tiles take 3, 5 and 6 rows a thread on a GPU of
152 SMs (one wave of 48, 80 and 96 rows a CTA; full, one row more than the height
below, ragged), loss and gradients against the CPU oracle with the 512-row check's bounds."""
import pytest

from test_gpu_surrogate_training import test_gradients_match_oracle as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [6001, 7296, 9729, 12160, 12161, 14592, 24320])
def test_gradients_match_oracle_at_every_height(rows):
    _check(rows)
