"""Inputs that the one-launch set-up and the one-call evaluation leave to the compositions
of tensor operations: equal to the composition's own values, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("categories", [4.0, np.int64(4), 3.5])
def test_category_counts_that_are_no_ints(categories):
    from torchtree_gb300 import site_models

    shape = torch.tensor([[0.3], [0.7]], dtype=torch.float64, device="cuda")
    rates, props = site_models.weibull_rates(shape, categories)
    want, want_p = site_models._weibull(shape, categories)
    for a, b in ((rates, want), (props, want_p)):  # (3.5 has no mean rate of one: NaN either way)
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    assert rates.shape == (2, 4)
