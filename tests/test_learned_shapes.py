"""LearnedProposal.train refuses arrays that its kernel would read beyond, before any device work."""
import numpy as np
import pytest

from feynsimul_gb300.learned import LearnedProposal


@pytest.mark.parametrize("feats,targets", [((50, 16), (40, 8)), ((50, 12), (50, 8)), ((50, 16), (50, 6)),
                                           ((800,), (50, 8)), ((50, 16), (400,))])
def test_train_checks_shapes(feats, targets):
    m = LearnedProposal(6, 0.25, 5.0)
    before = m.params.copy()
    for kw in ({}, {"reproducible": True}):
        with pytest.raises(ValueError, match="targets"):
            m.train(np.zeros(feats, np.float32), np.zeros(targets, np.float32), steps=1, batch=10, **kw)
    assert np.array_equal(m.params, before) and m.history == []
