"""Every kernel of a call reads what the operation before it on the stream has
written: inputs are refreshed by asynchronous copies from pinned memory right
before each call, rectangle clips bring a new table with each call, and every
result equals that of a call on settled inputs, bit for bit (the engine is
deterministic)."""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


def _engine(n):
    return HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, 1.0),
                               max_kernels=6)


def _stream(own):
    import torch
    return torch.cuda.Stream() if own else torch.cuda.current_stream()


@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("n,dtype,form", [(128, "uint8", "auto"), (512, "complex64", "auto"), (1024, "uint8", "auto"),
                                          (512, "float32", "auto"), (1024, "uint8", "fft"), (1024, "uint8", "tc")])
def test_copies_before_a_call(n, dtype, form, own_stream):
    import torch
    eng, st = _engine(n), _stream(own_stream)
    src = [(torch.rand(1, n, n) > 0.5).to(getattr(torch, dtype)).pin_memory() for _ in range(3)]
    dev = torch.empty((1, n, n), dtype=src[0].dtype, device="cuda")
    with torch.cuda.stream(st):
        ref = []
        for s in src:
            dev.copy_(s)
            torch.cuda.synchronize()
            ref.append(eng.compute_batch(dev, form=form, stream=st).clone())
            torch.cuda.synchronize()
        for i in np.random.default_rng(n).integers(3, size=40):
            dev.copy_(src[i], non_blocking=True)
            assert torch.equal(eng.compute_batch(dev, form=form, stream=st), ref[i])


@pytest.mark.parametrize("own_stream", [False, True])
def test_copies_before_a_gradient(own_stream):
    import torch
    from highuvlith_b200 import ilt
    n = 256
    eng, st = _engine(n), _stream(own_stream)
    src = [torch.rand(2, n, n).pin_memory() for _ in range(3)]
    target = (torch.rand(2, n, n, device="cuda") > 0.5).float()
    dev = torch.empty((2, n, n), device="cuda")
    with torch.cuda.stream(st):
        ref = []
        for s in src:
            dev.copy_(s)
            torch.cuda.synchronize()
            cost, grad = ilt.cost_and_gradient(eng, dev, target, ilt.IltSettings(), stream=st)
            torch.cuda.synchronize()
            ref.append((np.array(cost), grad.clone()))
        for i in np.random.default_rng(1).integers(3, size=40):
            dev.copy_(src[i], non_blocking=True)
            cost, grad = ilt.cost_and_gradient(eng, dev, target, ilt.IltSettings(), stream=st)
            assert np.array_equal(np.array(cost), ref[i][0]) and torch.equal(grad, ref[i][1])


@pytest.mark.parametrize("form", ["fft", "auto"])
@pytest.mark.parametrize("n,clips,count", [(128, 3, 15), (512, 8, 60)])
def test_rectangle_tables(n, clips, count, form):
    import torch
    rng = np.random.default_rng(n)
    sets = [[[tuple(v) for v in np.concatenate([rng.uniform(-n / 2, n / 2, (count, 2)), rng.uniform(4, 30, (count, 2))], 1)]
             for _ in range(clips)] for _ in range(3)]
    eng = _engine(n)
    first = eng.compute_batch_rects(sets[0], form=form).clone()  # a new table's first copy
    ref = []
    for s in sets:
        torch.cuda.synchronize()
        eng.compute_batch_rects(s, form=form)
        torch.cuda.synchronize()
        ref.append(eng.compute_batch_rects(s, form=form).clone())
    assert torch.equal(first, ref[0])
    for i in rng.integers(3, size=40):
        assert torch.equal(eng.compute_batch_rects(sets[i], form=form), ref[i])
