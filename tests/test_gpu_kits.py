"""Handles from used device blocks (the held sets in mmsp_gpu.cu): whatever a
block was used for before -- another model, type, size, a caller's stream --
a new handle's results are those of a fresh one, one after another, more at
once than are held, and from several threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [((64, 64), 1, np.float64, "ch"), ((33, 29), 1, np.float32, "ch"), ((20, 18), 2, np.float64, "ch_convex"),
         ((12, 10, 11), 3, np.float32, "gg"), ((9, 50), 1, np.float32, "ch_poly"), ((40, 24), 4, np.float64, "ac"),
         ((17, 13, 15), 1, np.float64, "ch"), ((700, 800), 1, np.float64, "ch")]   # the last: too large to be held


def run(gpu, k, stream=None):
    shape, fields, dtype, model = KINDS[k % len(KINDS)]
    rng = np.random.default_rng(k % len(KINDS))
    x = (0.4 + 0.05 * rng.random(shape + ((fields,) if fields > 1 else ()))).astype(dtype)
    p = dict(r=1.0, u=1.0) if model == "ch_poly" else {}
    if model != "ch_convex":
        p["dt"] = 0.002
    with gpu.Stepper(gpu.make_desc(shape, fields, dtype, model, **p)) as s:
        if stream is not None:
            s.set_stream(stream)
        s.upload(x)
        s.step(2 if model == "ch_convex" else 9)
        st = s.reduce()
        return s.download(), st.mass, st.energy


def same(a, b):
    return np.array_equal(a[0], b[0]) and a[1:] == b[1:]


def test_handles_one_after_another(gpu):
    import torch

    first = [run(gpu, k) for k in range(len(KINDS))]
    order = np.random.default_rng(5).integers(0, len(KINDS), 60)
    side = torch.cuda.Stream()
    for i, k in enumerate(order):
        assert same(run(gpu, int(k), side.cuda_stream if i % 3 == 0 else None), first[k])


def test_more_handles_than_are_held(gpu):
    d = gpu.make_desc((32, 32), 1, np.float64, "ch", dt=0.002)
    x = 0.4 + 0.05 * np.random.default_rng(1).random((32, 32))
    want = None
    for _ in range(3):
        many = [gpu.Stepper(d) for _ in range(20)]
        for i, s in enumerate(many):
            s.upload(x + 0.001 * i)
        for s in many:
            s.step(5)
        got = [s.download() for s in many]
        for s in many:
            s.close()
        assert len({g.tobytes() for g in got}) == 20
        assert want is None or all(np.array_equal(a, b) for a, b in zip(got, want))
        want = got


def test_handles_from_threads(gpu):
    first = [run(gpu, k) for k in range(len(KINDS))]
    bad = []

    def work(seed):
        try:
            for k in np.random.default_rng(seed).integers(0, len(KINDS), 25):
                if not same(run(gpu, int(k)), first[k]):
                    bad.append(int(k))
        except Exception as e:
            bad.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
