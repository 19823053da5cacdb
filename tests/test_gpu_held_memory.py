"""The device blocks that destroyed handles leave for later ones are given back
when something else of the library needs the memory: an allocation that fails
(of a batch that is larger than any GPU, which is refused as it always was), the
start of a server, whose budget is a share of the free memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HELD = 40 << 20     # of the eight blocks of 6 MB below


def hold(gpu):
    """Eight blocks of about 6 MB in the library's hands; the memory that is free then."""
    import torch

    many = [gpu.Stepper(gpu.make_desc((500, 500), 1, np.float64, "ch", dt=0.002)) for _ in range(8)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for s in many:
        s.close()
    assert torch.cuda.mem_get_info()[0] < before + HELD     # they are held
    return before


def test_failed_allocation_frees_them(gpu):
    import torch

    before = hold(gpu)
    with pytest.raises(gpu.GpuError) as ei:
        gpu.Batch([gpu.make_desc((64, 1 << 15, 1 << 15), 1, np.float64, "ch", dt=0.002)])
    assert ei.value.code == gpu.ENOMEM
    assert torch.cuda.mem_get_info()[0] >= before + HELD
    d = gpu.make_desc((500, 500), 1, np.float64, "ch", dt=0.002)
    with gpu.Stepper(d) as s:              # and handles go on working
        x = 0.4 + 0.05 * np.random.default_rng(1).random((500, 500))
        s.upload(x)
        s.step(3)
        first = s.download()
    with gpu.Stepper(d) as s:
        s.upload(x)
        s.step(3)
        assert np.array_equal(s.download(), first)


def test_server_start_frees_them(gpu):
    import torch

    with gpu.Server(budget_bytes=1 << 30):                  # what the driver keeps of a first one
        pass
    before = hold(gpu)
    with gpu.Server(budget_bytes=1 << 30):
        pass
    assert torch.cuda.mem_get_info()[0] >= before + HELD
