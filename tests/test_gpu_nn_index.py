"""A mini-batch's sample numbers: one that lies beyond the samples' memory is
refused before anything is launched, and the network goes on; repeated numbers
and those of the last sample give what the samples themselves give."""
import numpy as np
import pytest

from mplb_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


def test_index_beyond_the_samples_is_refused(gpu_lib):
    import torch
    net = ws.Network(2)
    net.init(3)
    rng = np.random.default_rng(1)
    cond = torch.from_numpy(rng.uniform(0, 1, (5, 3)).astype(np.float32)).cuda()
    target = torch.from_numpy(rng.normal(0, 1, (5, 128, 128, 3)).astype(
        np.float32)).cuda()
    torch.cuda.synchronize()

    def loss(index):
        return net.loss_grad(cond, target, index=index, want_loss=True)

    before = loss([4, 0])
    for index in ([2**31 - 1], [0, 2**31 - 1], [2**30, 1], [-1]):
        with pytest.raises(Exception, match="index"):
            loss(index)
    # the loss is one double sum in an order that may differ
    assert abs(loss([4, 0]) - before) <= 1e-12 * before
    rows = torch.tensor([4, 4], device="cuda")
    want = net.loss_grad(cond[rows].contiguous(), target[rows].contiguous(),
                         want_loss=True)
    torch.cuda.synchronize()
    assert abs(loss([4, 4]) - want) <= 1e-12 * want
    net.close()
