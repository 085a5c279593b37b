"""The norm of many rows by CTAs that walk them: the same bits as a CTA per row, around the number of rows at which the
one takes over from the other, and with rows left over for some CTAs."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
# multiples of the rows that run at once with a CTA each, and a few more: a vector a thread and two, last vectors of which
# some threads have none
@pytest.mark.parametrize("d, rounds", [(64, 1), (1024, 1), (1536, 2), (2048, 1), (2052, 1), (2052, 2), (2052, 4), (3072, 3),
                                       (4096, 1), (4096, 2), (4096, 3)])
def test_rows_in_one_launch_and_a_few_at_a_time(d, rounds, dtype):
    from llmoxide_b200 import kernels
    vectors = 1 if d <= 2048 else 2
    threads = max(64, -(-d // 4 // vectors // 32) * 32)
    n = rounds * torch.cuda.get_device_properties(0).multi_processor_count * (1536 // threads) + 5
    torch.manual_seed(d + n)
    h, gain = torch.randn(n + 1, d, device=DEV), torch.randn(d, device=DEV)
    out = torch.full((n + 1, d), 7.0, device=DEV, dtype=dtype)
    kernels.add_rms_norm(h[:n], None, gain, 1e-6, out[:n])
    assert (out[n] == 7.0).all()
    few = torch.empty_like(out[:n])
    for i in range(0, n, 300):
        kernels.add_rms_norm(h[i : min(n, i + 300)], None, gain, 1e-6, few[i : min(n, i + 300)])
    assert torch.equal(out[:n], few)
    want = h[:n].double() / torch.sqrt((h[:n].double() ** 2).mean(1, keepdim=True) + 1e-6) * gain.double()
    # a root mean square of at most 4096 values in chains of eight and butterflies: 1e-6; one rounding to bfloat16: 2^-9
    assert ((out[:n].double() - want).abs() / (want.abs() + 1e-3)).max().item() < (2e-6 if dtype == torch.float32 else 4.1e-3)
