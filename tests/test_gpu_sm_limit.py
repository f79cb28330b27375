"""`sm_limit`: the multiprocessors a step leaves are empty all the way through it, for the kernels of another stream, and the step's
results are those of a step that has the whole machine."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _make(name, kw, shapes, limit, seed=3):
    import kaon_b200
    gen = torch.Generator(device="cuda").manual_seed(seed)
    params = []
    for s in shapes:
        p = torch.nn.Parameter((torch.randn(s, device="cuda", generator=gen) * 0.02).bfloat16())
        p.grad = (torch.randn(s, device="cuda", generator=gen) * 1e-3).bfloat16()
        params.append(p)
    opt = getattr(kaon_b200, name)(params, **kw)
    opt.sr_seed = 7
    getattr(opt, "base_optimizer", opt).sm_limit = limit
    return params, opt


@pytest.mark.parametrize("name,kw", [
    ("Adakaon", dict(lr=1e-3, momentum_dtype="int8")),
    ("Nekaon", dict(lr=1e-3, weight_decay=0.1)),
    ("AdaPNM", dict(lr=1e-3, momentum_dtype="4bit")),
    ("KProdigy", dict(second_moment="factored", cautious=True)),
    ("Lion", dict(lr=1e-3, momentum_dtype="4bit")),
])
def test_same_bits_on_half_the_machine(name, kw):
    shapes = [(257, 264), (1025, 512), (13, 4096), (300,), (64, 256), (333, 77), (1280, 1280)]
    runs = []
    for limit in (None, 74):
        params, opt = _make(name, kw, shapes, limit)
        for _ in range(2):
            opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        runs.append([p.detach().clone() for p in params])
    for a, b in zip(*runs):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16)), a.shape


@pytest.mark.parametrize("name,kw", [
    ("Adakaon", dict(lr=1e-3, momentum_dtype="int8")),
    ("Nekaon", dict(lr=1e-3, weight_decay=0.1)),
])
def test_another_stream_finds_room_throughout(name, kw):
    """A chain of one-block kernels beside a step of about 1.5 ms: none of them waits for a kernel of the step to end (a COUNT,
    a quarter of the step, where blocks of the next launch sit on the multiprocessors that are to be left).  Everything
    is queued before either begins."""
    params, opt = _make(name, kw, [(1280, 1280)] * 48 + [(10240, 1280), (1280, 5120)] * 8, 128)
    for _ in range(2):
        opt.step()
    side, x = torch.cuda.Stream(), torch.zeros(64, device="cuda")
    n = 300
    marks = [torch.cuda.Event(enable_timing=True) for _ in range(n + 1)]
    go, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for again in range(2):   # (the first time round the side stream's kernels are loaded)
        torch.cuda.synchronize()
        torch.cuda._sleep(40_000_000)
        go.record()
        opt.step()
        end.record()
        with torch.cuda.stream(side):
            side.wait_event(go)
            marks[0].record()
            for m in marks[1:]:
                x.add_(1.0)
                m.record()
        torch.cuda.synchronize()
    step = go.elapsed_time(end)
    inside = [a.elapsed_time(b) for a, b in zip(marks, marks[1:]) if go.elapsed_time(a) < step]
    assert go.elapsed_time(marks[-1]) > 0.6 * step, "the chain ended before the step's sweeps"
    assert max(inside) < 0.08 * step, (step, sorted(inside)[-5:])
