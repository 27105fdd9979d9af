"""FP64 codon passes whose levels choose between tiles of 32 and 16 patterns: pattern
counts around both tiles (1, 16, 17, 33, 301, 512) and past the rule (513), one and
several samples and categories (tall and flat levels), with the internal children's
products kept and with the gradient budget that leaves no room for them.  lnL, dlnL/dP,
dlnL/dpi and dlnL/dw against the CPU oracle's autograd, at the repository's FP64 bound
of 1e-10 of the largest entry."""
import pytest

from test_gpu_wide_tips import test_tip_lookups_match_oracle as _against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [None, "1"])
@pytest.mark.parametrize("N,K,b,extra", [(1, 1, 1, 0), (16, 4, 1, 1), (17, 2, 3, 2), (33, 1, 1, 5), (301, 4, 1, 1),
                                         (512, 2, 1, 1), (513, 2, 1, 0)])
def test_fine_tiles_match_oracle(budget, N, K, b, extra, monkeypatch):
    if budget:  # bytes: no room for products (and slabs of the smallest size)
        monkeypatch.setenv("TT_GRADIENT_BUDGET_BYTES", budget)
    _against_oracle("f64", 61, N, K, b, extra)


@pytest.mark.parametrize("budget", [None, "1"])
@pytest.mark.parametrize("S,N,K,b,extra", [(20, 1, 1, 1, 0), (20, 129, 4, 2, 1), (20, 300, 2, 1, 5), (7, 257, 3, 1, 2),
                                           (20, 200, 2, 1, 60), (33, 130, 2, 1, 1)])
def test_kept_products_match_oracle(budget, S, N, K, b, extra, monkeypatch):
    """The same with 20 and other state counts."""
    if budget:
        monkeypatch.setenv("TT_GRADIENT_BUDGET_BYTES", budget)
    _against_oracle("f64", S, N, K, b, extra)
