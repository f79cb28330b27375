"""The cautious mask where update times gradient is subnormal: kept by its sign like any other, as the oracle does.  The
gradients are so small (the weights start at zero, so that the update shows) that every product lies between 1e-43 and
2^-126; the second step turns the sign of half of them, so that momentum and gradient disagree there."""
import numpy as np
import pytest
import torch

import kaon_oracle as ko

pytestmark = pytest.mark.gpu

# one CTA a tensor; warp units; rows that are no multiple of eight
SHAPES = [(64, 256), (96, 512), (60, 333)]


@pytest.mark.parametrize("name,size,kw", [
    ("Adakaon", 2e-27, dict(lr=0.05, momentum_dtype="float32")),
    ("Adakaon", 2e-27, dict(lr=0.05, momentum_dtype="int8")),
    ("AdaPNM", 3e-21, dict(lr=0.05, momentum_dtype="float32")),
    ("KProdigy", 2e-21, dict(momentum_dtype="float32", cautious=True, d0=1e-4, growth_rate=1.0)),
    ("AdaMuon", 1e-30, dict(lr=0.05, momentum_dtype="float32")),
])
def test_subnormal_products_are_masked_by_their_sign(name, size, kw):
    import kaon_b200
    from _gpu import to_bits
    kw = dict(kw, bf16_method="none")
    gen = torch.Generator().manual_seed(23)
    host = [torch.zeros(s) for s in SHAPES]
    params = [torch.nn.Parameter(h.clone().cuda()) for h in host]
    opt = getattr(kaon_b200, name)(params, **kw)
    orc = getattr(ko, "Oracle" + name)([to_bits(h) for h in host], SHAPES, **kw)
    for step in range(2):
        grads = [(0.5 + 0.5 * torch.rand(s, generator=gen)) * torch.randn(s, generator=gen).sign() * size for s in SHAPES]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        extra = {}
        if name == "AdaMuon":
            extra["ns_override"] = [opt.orthogonalised(p).float().cpu().numpy() for p in params]
        orc.step([to_bits(g) for g in grads], **extra)
        for i, p in enumerate(params):
            got, want = to_bits(p), orc.tensors[i].p
            assert np.any(want != 0.0), (step, i)
            # fp32 chains that differ by an ulp of a statistic, a rare code one step off
            bad = np.abs(got - want) > 2e-4 * np.abs(want) + 1e-6 * np.abs(want).max()
            assert bad.mean() < (1e-2 if kw["momentum_dtype"] == "int8" and step else 1e-3), (step, SHAPES[i], bad.mean())


@pytest.mark.parametrize("shape", [(96, 512), (64, 256), (60, 333)])
def test_the_kept_count_is_that_of_the_mask(shape):
    """Weights chosen so that the decay cancels the new momentum to within a rounding, m' + (lr wd) p: the sign of what is left turns
    on the last bit of m', and the count has to be taken of the very m' that is stored.  (m' does not depend on the weights, so a
    first run with weights of zero tells it; fp32 gradients, no centralization.  m' + (lr wd) p is exact in fp64: 24 + 24 bits
    beside 24 at the same magnitude.)"""
    import kaon_b200
    gen = torch.Generator().manual_seed(29)
    grad = (torch.randn(shape, generator=gen) * 1e-3).cuda()
    lr, wd = 0.05, 0.1
    lrwd = np.float64(np.float32(lr * wd))

    def run(weights):
        p = torch.nn.Parameter(weights.clone())
        p.grad = grad.clone()
        opt = kaon_b200.Adakaon([p], lr=lr, weight_decay=wd, momentum_dtype="float32", gradient_centralization=False)
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        (plan,) = opt._plans.values()
        return opt.state[p]["m"].double().cpu().numpy().reshape(-1), plan.kept_counts(torch.cuda.current_stream().cuda_stream)[0]

    m, _ = run(torch.zeros(shape, device="cuda"))
    w = (-m / lrwd).astype(np.float32)
    again, kept = run(torch.from_numpy(w).reshape(shape).cuda())
    assert np.array_equal(m, again)
    delta = m + lrwd * w.astype(np.float64)
    assert np.abs(delta).max() <= 2.0 ** -23 * np.abs(m).max()
    assert kept == int((np.sign(delta) * np.sign(grad.double().cpu().numpy().reshape(-1)) > 0).sum())
