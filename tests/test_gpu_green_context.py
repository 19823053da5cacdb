"""Handles on a stream that has only a part of the GPU's SMs (a green context):
the launches whose blocks wait for one another want a block per SM there, and
the steps have to be taken all the same, with the results of any other stream.

2D FP64 Cahn-Hilliard bit for bit (its two passes); the convex-splitting solve
within 1e-10 of the oracle, its other tests' bound (its residual is added up in
another order, so a stop can fall one check apart)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def part_stream(gpu):
    """A stream on 16 or so of the SMs."""
    import torch

    torch.zeros(1, device="cuda")          # the primary context is there
    cu = ctypes.CDLL("libcuda.so.1")
    SM, DEFAULT_STREAM, NON_BLOCKING = 1, 1, 1

    class Resource(ctypes.Structure):      # CUdevResource
        _fields_ = [("type", ctypes.c_uint), ("pad", ctypes.c_ubyte * 92), ("sms", ctypes.c_uint),
                    ("rest", ctypes.c_ubyte * 44)]

    def ok(rc):
        if rc:
            pytest.skip("no green contexts here: %d" % rc)

    dev, whole, part, rest = ctypes.c_int(), Resource(), Resource(), Resource()
    ok(cu.cuCtxGetDevice(ctypes.byref(dev)))
    ok(cu.cuDeviceGetDevResource(dev, ctypes.byref(whole), SM))
    n = ctypes.c_uint(1)
    ok(cu.cuDevSmResourceSplitByCount(ctypes.byref(part), ctypes.byref(n), ctypes.byref(whole), ctypes.byref(rest), 0, 16))
    assert 1 <= part.sms < whole.sms
    desc, green, stream = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    ok(cu.cuDevResourceGenerateDesc(ctypes.byref(desc), ctypes.byref(part), 1))
    ok(cu.cuGreenCtxCreate(ctypes.byref(green), desc, dev, DEFAULT_STREAM))
    ok(cu.cuGreenCtxStreamCreate(ctypes.byref(stream), green, NON_BLOCKING, 0))
    yield stream.value
    torch.cuda.synchronize()
    cu.cuStreamDestroy_v2(stream)
    cu.cuGreenCtxDestroy(green)


@pytest.mark.parametrize("contract", [False, True])
@pytest.mark.parametrize("shape", [(70, 90), (640, 640), (5, 7)], ids=lambda s: "x".join(map(str, s)))
def test_many_steps_on_a_part_of_the_sms(gpu, part_stream, shape, contract):
    from mmsp_gb300 import inputs

    x = inputs.noisy_composition(shape, 0.45, 0.05, 5)
    out = []
    for stream in (None, part_stream):
        with gpu.Stepper(gpu.make_desc(shape, 1, np.float64, "ch", dt=0.004, contract=contract)) as s:
            if stream:
                s.set_stream(stream)
            s.upload(x)
            s.step(7)
            s.step(300)
            out.append(s.download())
            s.set_stream(None)             # back on a stream with all of them
            s.upload(x)
            s.step(307)
            out.append(s.download())
    assert all(np.array_equal(v, out[0]) for v in out)


@pytest.mark.parametrize("shape", [(40, 24), (400, 200), (20, 18, 22)], ids=lambda s: "x".join(map(str, s)))
def test_convex_solve_on_a_part_of_the_sms(gpu, oracle, part_stream, shape):
    from mmsp_gb300 import inputs

    x = inputs.convex_start(shape, 17)
    want, iters = oracle.ch_convex(x, 2, return_iters=True)
    with gpu.Stepper(gpu.make_desc(shape, 2, np.float64, "ch_convex")) as s:
        s.set_stream(part_stream)
        s.upload(x)
        s.step(2)
        got = s.download()
        assert abs(s.reduce().solver_iterations - iters) <= 5
    assert np.abs(got - want).max() <= 1e-10 * max(1.0, np.abs(want).max())
