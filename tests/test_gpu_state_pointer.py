"""A state that the program reads through mmsp_gpu_state on a stream of its own:
destroying the handle waits for that work, and the next handle of the same size
does not get the memory under it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3)


@pytest.mark.parametrize("steps", [0, 3])
def test_read_of_a_state_outlives_its_handle(gpu, steps):
    import torch

    shape = (96, 80)
    d = gpu.make_desc(shape, 1, np.float64, "ch", dt=0.002)
    x, other = [0.4 + 0.05 * np.random.default_rng(k).random(shape) for k in (1, 2)]
    side = torch.cuda.Stream()
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        s = gpu.Stepper(d)
        s.upload(x)
        if steps:
            s.step(steps)
        want = s.download()
        view = torch.as_tensor(View(s.state_ptr(), shape), device="cuda")
        with torch.cuda.stream(side):
            torch.cuda._sleep(4 * 10 ** 8)         # a fifth of a second before the copy
            out.copy_(view, non_blocking=True)
        s.close()
        with gpu.Stepper(d) as t:
            t.upload(other)
            t.step(5)
            t.synchronize()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
