"""The flow's pass with two groups of warps gives the bits of the pass with one.

Both run the same BF16 products with FP32 accumulation along the hidden units, the same
FP32 order of the first layer's sums, and splines whose two forms (packed, and with the
shorter latency) differ only in how a bin is found.  Rows are independent, so the bits
of a row do not depend on how many there are."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K', [16, 32])
@pytest.mark.parametrize('dim', [2, 3, 5, 8, 9, 16])
def test_pass_of_many_rows_has_the_bits_of_few(dim, K):
    from vegas_gb300.flow import Flow
    import flow_oracle as F
    fl = Flow(dim, K=K)
    fl.set_theta(F.init_theta(dim, 6, K, 128, seed=4, out_scale=1.0))
    many = torch.cuda.get_device_properties(0).multi_processor_count * 128
    g = torch.Generator(device='cuda').manual_seed(dim + K)
    u = torch.rand((3 * many + 77, dim), generator=g, device='cuda')
    u[:2 * dim:2] = 0.0        # at the ends and at quarters, where a bin may start
    u[1:2 * dim:2] = 1.0 - 2.0 ** -24
    u[2 * dim:4 * dim] = torch.arange(2 * dim, device='cuda').remainder(5)[:, None] / 4.0
    for run in (fl.sample, fl.density):
        parts = [run(c.contiguous()) for c in u.split(5000)]
        zr, lr = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        for n in (many + 1, 2 * many - 127, u.shape[0]):
            z, ld = run(u[:n].contiguous())
            assert torch.equal(z, zr[:n]) and torch.equal(ld, lr[:n])
