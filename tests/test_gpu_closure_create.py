"""Creating a closure does not wait for the work queued on the device."""

import pytest
import torch

import symcode as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", (lambda d, g: S.create_bardina(2.0, d, g), S.create_dynamic_smagorinsky))
def test_the_test_filter_table_is_not_queued_behind_the_caller(make):
    g = S.Grid(3, 32, dtype=torch.float32, device="cuda:0")
    keep = [make(4 * g.spacing, g)]  # loads the kernel
    torch.cuda.synchronize()
    queued = torch.cuda.Event()
    torch.cuda._sleep(2_000_000_000)  # about a second
    queued.record()
    keep.append(make(4 * g.spacing, g))
    assert not queued.query()
    torch.cuda.synchronize()
    for c in keep:
        c.close()
    g.close()
