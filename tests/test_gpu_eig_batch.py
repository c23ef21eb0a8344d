"""The r largest eigenpairs of batches around the number of SMs, where the launch for orders of 33 to 64
changes: the same matrices give the same pairs to rounding, checked against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 33, 50, 64, 65])
@pytest.mark.parametrize("batch", [148, 149, 300])
def test_batches_around_the_sms(cuda, n, batch):
    import torch
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(n * batch)
    x = rng.standard_normal((batch, n, 3 * n)) + 3.0
    a, r = x @ x.transpose(0, 2, 1), 4
    ev, V, info = pl.eigh_top(torch.from_numpy(a).to(cuda), r)
    assert torch.count_nonzero(info).item() == 0
    ev, V = ev.cpu().numpy(), V.cpu().numpy()
    scale = np.abs(a).max((1, 2))
    w = np.linalg.eigvalsh(a)[:, n - r:]
    # the bounds of the other eigensolver tests
    assert (np.abs(ev - w).max(1) < 1e-12 * n * scale).all()
    assert np.abs(V.transpose(0, 2, 1) @ V - np.eye(r)).max() < 1e-12
    assert (np.abs(a @ V - V * ev[:, None, :]).max((1, 2)) < 1e-12 * n * scale).all()
