"""The warp-unit kernels at the edges of their units: rows that end inside a vector, a tensor that ends inside one, rows of
fewer than eight elements, exactly one trip of a warp, one element more than a unit, whole-row units; Lion (one launch and,
with `big`, a launch per phase) and the other optimizers whose sweeps share the building blocks, one step from fresh state
against the CPU oracle."""
import numpy as np
import pytest
import torch

import kaon_oracle as ko

pytestmark = pytest.mark.gpu

EDGES = [(3,), (127,), (256,), (4097,), (16, 3), (50, 7), (33, 64), (9, 333), (2, 4104), (5, 640), (1, 128), (96, 8)]


@pytest.mark.parametrize("name,kw,big", [
    ("Lion", dict(momentum_dtype="4bit", bf16_method="none"), False),
    ("Lion", dict(momentum_dtype="bfloat16", weight_decay=0.1, bf16_method="none"), False),
    ("Lion", dict(momentum_dtype="4bit"), True),
    ("Adakaon", dict(momentum_dtype="int8"), False),
    ("AdaPNM", dict(momentum_dtype="4bit"), False),
    ("AdaPNM", dict(momentum_dtype="int8"), False),
    ("KProdigy", dict(momentum_dtype="bfloat16"), False),
    ("KProdigy", dict(momentum_dtype="int8"), False),
])
def test_unit_edges_vs_oracle(name, kw, big):
    import kaon_b200
    from _gpu import to_bits
    shapes = EDGES + ([(16385, 4096)] if big else [])
    gen = torch.Generator().manual_seed(31)
    host = [(torch.randn(s, generator=gen) * 0.02).bfloat16() for s in shapes]
    grads = [(torch.randn(s, generator=gen) * 1e-3).bfloat16() for s in shapes]
    params = [torch.nn.Parameter(h.clone().cuda()) for h in host]
    opt = getattr(kaon_b200, name)(params, lr=1e-3, **kw)
    opt.sr_seed = 5
    n_cmp = len(EDGES)
    orc = getattr(ko, "Oracle" + name)([to_bits(h) for h in host[:n_cmp]], shapes[:n_cmp], seed=5, lr=1e-3, **kw)
    for p, g in zip(params, grads):
        p.grad = g.cuda()
    opt.step()
    torch.cuda.synchronize()
    opt.check_device_status()
    if name == "Lion":
        assert opt.stats()["kernel_launches"] == (2 if big else 1)
    orc.step([to_bits(g) for g in grads[:n_cmp]])
    bad = total = 0
    for i, p in enumerate(params[:n_cmp]):
        got, want = to_bits(p).reshape(-1), orc.tensors[i].p.reshape(-1)
        diff = np.abs(got.astype(np.int32) - want.astype(np.int32))
        assert diff.max() <= 1, (shapes[i], diff.max())   # the other bf16 neighbour at most
        bad += int((diff != 0).sum())
        total += diff.size
    assert bad <= 5e-3 * total, (bad, total)
