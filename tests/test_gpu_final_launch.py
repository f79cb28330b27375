"""FINAL as launches of its own, at the edges of its strips (128 columns) and of the row table's runs (256 rows): one strip
exactly two wide, a last strip of eight columns, one row beyond a run, fewer runs of rows than warps; int8 momentum over rows
that are whole trips of a warp (their maxima wait for the row's end) and over rows that are not.  Two steps against the CPU
oracle: statistics, scales and codes, weights."""
import sys

import numpy as np
import pytest
import torch

import kaon_oracle as ko

pytestmark = pytest.mark.gpu

EDGES = [(65, 256), (257, 264), (40, 1032), (1025, 512), (13, 4096), (300,)]


@pytest.mark.parametrize("name,kw", [
    ("Adakaon", dict(momentum_dtype="int8")),
    ("Adakaon", dict(momentum_dtype="int8", cautious=False, weight_decay=0.1)),
    ("Adakaon", dict(momentum_dtype="4bit", weight_decay=0.1, bf16_method="none")),
    ("Adakaon", dict(bf16_method="kahan", weight_decay=0.1)),
    ("Nekaon", dict(momentum_dtype="int8")),
    ("AdaPNM", dict(momentum_dtype="4bit")),
    ("KProdigy", dict(second_moment="factored", cautious=True)),
])
def test_final_edges_vs_oracle(name, kw):
    import kaon_b200
    from _gpu import state_np, to_bits
    kw = dict(kw) if name == "KProdigy" else dict(kw, lr=1e-3)
    gen = torch.Generator().manual_seed(47)
    host = [(torch.randn(s, generator=gen) * 0.02).bfloat16() for s in EDGES]
    params = [torch.nn.Parameter(h.clone().cuda()) for h in host]
    opt = getattr(kaon_b200, name)(params, **kw)
    opt.sr_seed = 5
    inner = getattr(opt, "base_optimizer", opt)
    orc = getattr(ko, "Oracle" + name)([to_bits(h) for h in host], EDGES, seed=5, **kw)
    for step in range(2):
        grads = [(torch.randn(s, generator=gen) * 1e-3).bfloat16() for s in EDGES]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        orc.step([to_bits(g) for g in grads])
        bad = total = bad_codes = codes = 0
        for i, p in enumerate(params):
            at = (step, EDGES[i])
            for key, want in orc.tensors[i].state.items():
                got = state_np(inner.state[p], key)
                if not isinstance(want, np.ndarray) or got is None or want.size == 0 or key == "shift":
                    continue
                got, want = got.reshape(-1), want.reshape(-1)
                if got.dtype.kind == "f":       # sums in another order: an ulp or two of a statistic
                    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max(), (at, key)
                else:                           # codes, packed codes, bf16 bits: a neighbour where the quotient lies on a boundary
                    diff = np.nonzero(got != want)[0]
                    bad_codes += diff.size
                    codes += got.size
                    if got.dtype == np.uint16 or got.dtype == np.int16:
                        # bf16 momentum: a neighbour of the update (2^-7 of it at most) enters by w1 < 1; in steps of the momentum
                        # itself that can be several, where it is small
                        val = lambda b: (b.view(np.uint16).astype(np.uint32) << 16).view(np.float32)  # noqa: E731
                        assert np.abs(val(got) - val(want)).max() <= 2.0 ** -7 * np.abs(val(want)).max(), (at, key)
                        continue
                    for x, y in zip(got[diff].tolist(), want[diff].tolist()):
                        step_of = max(abs((x & 15) - (y & 15)), abs((x >> 4) - (y >> 4))) if got.dtype == np.uint8 else abs(x - y)
                        assert step_of == 1, (at, key)
            diff = np.abs(to_bits(p).astype(np.int32) - orc.tensors[i].p.reshape(-1).astype(np.int32))
            assert diff.max() <= (2 if name == "Nekaon" else 1), at   # the other bf16 neighbour at most; Nekaon rounds twice (update, climb)
            bad += int((diff != 0).sum())
            total += diff.size
        assert bad <= 1e-3 * total, (step, bad, total)
        assert bad_codes <= 2 + 1e-4 * codes, (step, bad_codes, codes)


@pytest.mark.parametrize("name", ["Adakaon", "AdaPNM"])
def test_a_row_whose_squares_overflow_has_an_infinite_statistic(name):
    """Gradients of 1e20 in one row, of either sign in turn (so that the row's mean is zero whatever the order of its sum): its
    statistic, and those of the columns, are infinite, as the oracle's are, and not NaN; other rows keep theirs."""
    import kaon_b200
    from _gpu import state_np, to_bits
    shape = (65, 512)
    gen = torch.Generator().manual_seed(3)
    host = (torch.randn(shape, generator=gen) * 0.02).bfloat16()
    grad = (torch.randn(shape, generator=gen) * 1e-3).bfloat16()
    grad[7] = 1e20
    grad[7, 1::2] = -1e20
    p = torch.nn.Parameter(host.clone().cuda())
    opt = getattr(kaon_b200, name)([p], lr=1e-3)
    orc = getattr(ko, "Oracle" + name)([to_bits(host)], [shape], lr=1e-3)
    p.grad = grad.cuda()
    opt.step()
    torch.cuda.synchronize()
    opt.check_device_status()
    orc.step([to_bits(grad)])
    want = orc.tensors[0].state
    assert np.isinf(want["row"]).sum() == 1 and np.isinf(want["col"]).all()
    for key in ("row", "col"):
        got = state_np(opt.state[p], key)
        assert np.array_equal(np.isinf(got), np.isinf(want[key])) and not np.isnan(got).any(), key
        fine = np.isfinite(want[key])
        assert np.abs(got[fine] - want[key][fine]).max(initial=0.0) <= 2e-6 * np.abs(want[key][fine]).max(initial=1e-30), key


@pytest.mark.parametrize("name,kw", [
    ("Adakaon", dict(momentum_dtype="int8")),
    ("AdaPNM", dict(momentum_dtype="4bit")),
    ("KProdigy", dict(second_moment="factored", cautious=True)),
])
def test_odd_tensors_beside_the_statistics_of_others(name, kw, monkeypatch):
    """Rows that are no multiple of eight keep their stages in the persistent kernel, which runs at the same time as the STATS
    launch of the other tensors."""
    monkeypatch.setattr(sys.modules[__name__], "EDGES", [(333, 77), (640, 512), (160, 100), (257, 264), (300,)])
    test_final_edges_vs_oracle(name, kw)


@pytest.mark.parametrize("name,kw", [
    ("Adakaon", dict(momentum_dtype="int8")),
    ("Adakaon", dict(bf16_method="kahan", weight_decay=0.1)),
    ("AdaPNM", dict(momentum_dtype="4bit")),
])
def test_final_gives_the_same_bits_wherever_it_runs(name, kw):
    """Three tensors by themselves, whose FINAL is a launch, and at the head of a list that keeps FINAL in the persistent kernel
    (thirty tall matrices, whose stages stay there, beside STATS of twenty wide ones): statistics and weights of the three are the same."""
    import kaon_b200
    gen = torch.Generator(device="cuda").manual_seed(3)
    shapes = [(40, 1032), (640, 512), (1300, 264)] + [(1280, 32)] * 30 + [(32, 1280)] * 20
    values = [((torch.randn(s, device="cuda", generator=gen) * 0.02).bfloat16(), (torch.randn(s, device="cuda", generator=gen) * 1e-3).bfloat16())
              for s in shapes]
    runs = []
    for n in (3, len(shapes)):
        params = [torch.nn.Parameter(v.clone()) for v, _ in values[:n]]
        for p, (_, g) in zip(params, values):
            p.grad = g.clone()
        opt = getattr(kaon_b200, name)(params, lr=1e-3, **kw)
        opt.sr_seed = 5
        for _ in range(2):
            opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        runs.append([t for p in params[:3] for t in (p.detach().view(torch.int16), opt.state[p]["row"], opt.state[p]["col"])])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
