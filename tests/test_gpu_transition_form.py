"""The form of a block's pair transition: with few rows and many hidden channels the three launches, which spread the hidden channels over
the chip, otherwise the one that keeps them in the SM; bit for bit the operators one by one, whose transition is the one launch throughout."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,n,batch,one", [(256, 24, 1, False), (256, 33, 1, False), (256, 64, 1, False), (256, 45, 2, False), (256, 80, 1, False), (256, 102, 1, True),
                                           (256, 103, 1, True), (256, 129, 1, True), (128, 24, 1, True), (128, 64, 1, True)])
def test_blocks_take_the_faster_form(c, n, batch, one):
    from kfold_b200 import _lib as L, modules as M
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(1000 * c + n)
    blk = M.TriangularBlock(c).to(dev)
    with torch.no_grad():
        for p in blk.parameters():
            p.normal_(0.0, p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1, generator=gen).add_(1.0 if p.dim() == 1 else 0.0)
        z = torch.randn(batch, n, n, c, generator=gen, device=dev).bfloat16()
        mask = torch.rand(batch, n, n, generator=gen, device=dev) > 0.1
        got = blk(z, mask)
        L.profile_enable(True)
        again = blk(z, mask)
        torch.cuda.synchronize()
        tags = L.profile_report()
        L.profile_enable(False)
        ref = blk.transition_z(blk.tri_mul_in(blk.tri_mul_out(z, mask, residual=True), mask, residual=True), residual=True)
    assert ("transition_pair" in tags) == one and torch.equal(got, again)
    assert torch.equal(got, ref)
    assert L.device_status() == 0
