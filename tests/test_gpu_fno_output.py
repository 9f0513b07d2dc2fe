"""ehd_fno_forward into output memory that the projection kernel cannot store to:
an array of floats at an odd address is reached by a copy, with the same bits.
"""
import pytest

from conftest import ehd, fno

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_forward_into_any_alignment(offset):
    import torch
    net = fno.FNO(12, 10, 8, 3, 2, width=16, layers=2, modes=(3, 2, 2), hidden=32, max_batch=2, seed=3)
    with net:
        g = torch.Generator(device="cuda").manual_seed(5)
        a = torch.randn(2, 8, 10, 12, 3, generator=g, device="cuda")
        ref = net.forward(a)
        raw = torch.zeros(4 * ref.numel() + 16, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ehd._check(fno.lib().ehd_fno_forward(net.h, 2, a.data_ptr(), raw.data_ptr() + offset))
        net.synchronize()
        got = raw[offset:offset + 4 * ref.numel()].clone().view(torch.float32)
        assert torch.equal(got, ref.flatten())
        assert int(raw[:offset].sum()) == 0 and int(raw[offset + 4 * ref.numel():].sum()) == 0
