"""The device's Gamma quantiles, their shape derivatives and the category rates made of
them, to the last bit: FP32 transition matrices are rounded from the rates, so a rate
that moves by 1e-16 moves FP32 gradients by more than 1e-9.

``golden/gamma_quantiles.json``: ``gamma_quantile`` (csrc/tt_gamma.cuh) by one thread per
quantile on a GB300, hexadecimal.  Shapes 0.001 to 200 (among them ones whose iteration
stops, wanders among neighbouring values to its last step, and fails: NaN), 1 to 32
categories.  Equality, no tolerance."""
import json
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SETS = json.loads((Path(__file__).parent / "golden" / "gamma_quantiles.json").read_text())["sets"]


def _numbers(x):
    return np.array([_numbers(v) if isinstance(v, list) else float.fromhex(v) for v in x])


@pytest.mark.parametrize("case", SETS, ids=lambda s: f"k{s['categories']}")
def test_quantiles_keep_their_bits(case):
    from torchtree_gb300 import _native

    k, shapes = case["categories"], _numbers(case["shapes"])
    a = torch.tensor(shapes, device="cuda")
    x = torch.empty(len(shapes), k, dtype=torch.float64, device="cuda")
    d = torch.empty_like(x)
    _native.check(_native.load().tt_gamma_quantiles(
        len(shapes), k, _native.ptr(a), _native.ptr(x), _native.ptr(d),
        _native.ptr_value(torch.cuda.current_stream().cuda_stream)))
    np.testing.assert_array_equal(x.cpu().numpy(), _numbers(case["quantiles"]))
    np.testing.assert_array_equal(d.cpu().numpy(), _numbers(case["derivatives"]))


@pytest.mark.parametrize("case", SETS, ids=lambda s: f"k{s['categories']}")
def test_rates_keep_the_bits_of_the_composition(case):
    from torchtree_gb300 import site_models

    shape = torch.tensor(_numbers(case["shapes"]), device="cuda").unsqueeze(-1)
    rates, _ = site_models.gamma_rates(shape, case["categories"])
    want, _ = site_models._gamma(shape, case["categories"])
    np.testing.assert_array_equal(rates.cpu().numpy(), want.cpu().numpy())
