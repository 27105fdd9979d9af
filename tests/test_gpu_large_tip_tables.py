"""FP32 codon plans of 65 and 128 codes with enough patterns for the large table of tip
products (12 tiles of 128 patterns, 8,192 products), beside 64 and 129 codes: against the
CPU oracle as in test_gpu_wide_tips, at the repository's parity bounds (lnL 1e-6, gradients
1e-4), and a captured pass that meets the other counts."""
import pytest

from test_gpu_captured_code_counts import test_captured_pass_follows_other_code_counts as _captured

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(65, 128, 64, 129), (128, 140, 61), (64, 100)])
def test_large_tables(counts):
    _captured(61, "f32", 20, 1409, 4, 9, counts)
