"""Forms of the models' inputs beside the usual ones."""
import torch


def test_codon_tables_as_sequences():
    from torchtree_gb300 import substitution as sub

    want = sub.codon_pair_masks()
    for table in (list(sub.UNIVERSAL_CODE), tuple(sub.UNIVERSAL_CODE)):
        got = sub.codon_pair_masks(table)
        assert got[3] == want[3] and all(torch.equal(a, b) for a, b in zip(got[:3], want[:3]))
        one = torch.ones(1, dtype=torch.float64)
        pi = torch.full((61,), 1.0 / 61, dtype=torch.float64)
        assert torch.equal(sub.mg94_q(one, 2.0 * one, 3.0 * one, pi, table), sub.mg94_q(one, 2.0 * one, 3.0 * one, pi))


def test_mg94_with_one_frequency_for_all_codons():
    from torchtree_gb300 import substitution as sub

    one = torch.ones(1, dtype=torch.float64)
    pi = torch.tensor(1.0 / 61, dtype=torch.float64)
    assert torch.equal(sub.mg94_q(one, 2.0 * one, 3.0 * one, pi), sub.mg94_q(one, 2.0 * one, 3.0 * one, pi.expand(61)))
