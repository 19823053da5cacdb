"""Step calls that a caller captures, on 2D FP32 grids of few rows: their tile
kernel takes its work from two counters in turn, whose state a replay must not
depend on.  Odd and even numbers of launches, replayed several times, between
direct calls, and captured without ever being run.

The same steps as direct calls, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lead", [0, 4, 8], ids=lambda n: "after%d" % n)
@pytest.mark.parametrize("steps", [4, 8, 12, 20, 23])
@pytest.mark.parametrize("shape", [(9, 33), (23, 500)], ids=["9x33", "23x500"])
def test_replays_of_captured_tile_steps(gpu, shape, steps, lead):
    import torch

    d = gpu.make_desc(shape, 1, np.float32, "ch", dt=0.002)
    rng = np.random.default_rng(steps)
    xs = [(0.4 + 0.05 * rng.random(shape)).astype(np.float32) for _ in range(4)]
    stream = torch.cuda.Stream()
    with gpu.Stepper(d) as s, gpu.Stepper(d) as direct:
        def steps_of(x):
            direct.upload(x)
            direct.step(steps)
            return direct.download()

        s.set_stream(stream.cuda_stream)
        inp, out = torch.zeros(shape, device="cuda"), torch.zeros(shape, device="cuda")
        torch.cuda.synchronize()
        s.upload(xs[0])
        if lead:
            s.step(lead)
        graphs = []
        for _ in range(2):                     # the first is never run
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                s.upload_device(inp.data_ptr(), 4 * inp.numel())
                s.step(steps)
                s.download_device(out.data_ptr(), 4 * out.numel())
            graphs.append(g)
        for x in xs[1:]:
            s.upload(xs[0])                    # a direct call between the replays
            s.step(steps)
            assert np.array_equal(s.download(), steps_of(xs[0]))
            for _ in range(3):
                inp.copy_(torch.from_numpy(x))
                out.zero_()
                torch.cuda.synchronize()
                graphs[1].replay()
                torch.cuda.synchronize()
                assert np.array_equal(out.cpu().numpy(), steps_of(x))
