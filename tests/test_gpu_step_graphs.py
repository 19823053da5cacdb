"""Step calls around the lengths where the handle goes over to graph replays
(run_launches in mmsp_gpu.cu): one launch under and over each threshold and
each multiple, starting from either buffer, blocked grids (strips and tiles,
whose launches are four steps) and plain ones, a stream that the caller
captures.  One call equals many short ones bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [((20, 24, 28), 1, np.float32, "ch", 1), ((12, 14, 16), 3, np.float64, "gg", 1), ((40, 48), 1, np.float32, "ch", 4),
         ((9, 33), 1, np.float32, "ch", 4)]


def state(shape, fields, dtype):
    x = 0.4 + 0.05 * np.random.default_rng(3).random(shape + ((fields,) if fields > 1 else ()))
    return x.astype(dtype)


@pytest.mark.parametrize("lead", [0, 1, 2])
@pytest.mark.parametrize("shape,fields,dtype,model,per", GRIDS, ids=["x".join(map(str, g[0])) for g in GRIDS])
def test_one_call_equals_short_calls(gpu, shape, fields, dtype, model, per, lead):
    d = gpu.make_desc(shape, fields, dtype, model, dt=0.002)
    x = state(shape, fields, dtype)
    with gpu.Stepper(d) as a, gpu.Stepper(d) as b:
        for n in (31, 32, 33, 47, 48, 65, 191, 192, 193, 225, 300):
            for s in (a, b):
                s.upload(x)
                for _ in range(lead):      # the state is in the other buffer after an odd number
                    s.step(per)
            a.step(n * per + (n % per if per > 1 else 0))
            for _ in range(n):
                b.step(per)
            if per > 1 and n % per:
                b.step(n % per)
            assert np.array_equal(a.download(), b.download()), n


@pytest.mark.parametrize("shape,dtype", [((20, 24, 28), np.float32), ((48, 50), np.float64), ((48, 50), np.float32)],
                         ids=["3d-f32", "2d-f64", "2d-f32"])
def test_steps_on_a_captured_stream(gpu, shape, dtype):
    import torch

    d = gpu.make_desc(shape, 1, dtype, "ch", dt=0.002)
    x = state(shape, 1, dtype)
    stream = torch.cuda.Stream()
    with gpu.Stepper(d) as s:
        s.upload(x)
        s.step(120)
        want = s.download()
        s.set_stream(stream.cuda_stream)
        s.upload(x)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            s.step(40)
        for _ in range(3):                 # 40 steps end in the buffer that they began in
            g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.download(), want)
