"""GPU: several handles, streams and host threads at a time -- what one of them
sets, keeps or gives back does not reach the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def functional(mdf, k):
    return mdf.optibasis.HermiteLossFunc(2.0, 4, 0.95, [k] * 3, 20736.0, 20736, [30.0] * 3)


def test_functionals_of_two_meshes_in_turn(mdf):
    import torch
    c = torch.from_numpy(mdf.optibasis.bspline_initial_basis(2.0, 4, 4)[None]).cuda()
    big = functional(mdf, 256)
    want = mdf.optibasis.ik_error_loss(c, big)
    small = functional(mdf, 224)
    other = mdf.optibasis.ik_error_loss(c, small)
    for _ in range(2):
        assert torch.equal(mdf.optibasis.ik_error_loss(c, big), want)
        assert torch.equal(mdf.optibasis.ik_error_loss(c, small), other)
