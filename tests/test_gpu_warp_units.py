"""The warp-unit kernels at the edges of their units: rows that end inside a vector, a tensor that ends inside one, rows of
fewer than eight elements, exactly one trip of a warp, one element more than a unit, whole-row units; Lion (one launch and,
with `big`, a launch per phase) and the other optimizers whose sweeps share the building blocks, two steps from fresh state
(the second reads the codes of the first) against the CPU oracle: weights, momentum codes, scales and statistics."""
import numpy as np
import pytest
import torch

import kaon_oracle as ko

pytestmark = pytest.mark.gpu

EDGES = [(3,), (127,), (256,), (4097,), (16, 3), (50, 7), (33, 64), (9, 333), (2, 4104), (5, 640), (1, 128), (96, 8)]

# What may differ from the oracle, by what lies between gradient and result.  `EXACT`: nothing but row means of the gradient
# (bf16 weights: rounded to bf16, so the order of the sum does not show) and per-element fp32 arithmetic: the same bits.
# `SUMS`: statistics summed in another order, an ulp or two (2e-6 of a statistic or scale): a code differs where the quotient
# lies that close to a rounding boundary (|code| x 2 x 2e-7: 2e-5 of int8 codes on average, fewer of 4-bit ones; bound
# 2 + 1e-4 n), by one step; a bf16 weight by one neighbour where the sum lies as close to a boundary (bound 1e-3).
EXACT, SUMS = "exact", "sums"


@pytest.mark.parametrize("name,dtype,kw,how,big", [
    ("Lion", "bf16", dict(momentum_dtype="4bit", bf16_method="none"), EXACT, False),
    ("Lion", "bf16", dict(momentum_dtype="bfloat16", weight_decay=0.1, bf16_method="none"), EXACT, False),
    ("Lion", "bf16", dict(momentum_dtype="4bit"), EXACT, True),
    ("Lion", "f32", dict(momentum_dtype="4bit", weight_decay=0.1), SUMS, False),
    ("Lion", "f32", dict(momentum_dtype="float32"), SUMS, False),
    ("Adakaon", "bf16", dict(momentum_dtype="int8"), SUMS, False),
    ("Adakaon", "bf16", dict(momentum_dtype="bfloat16", bf16_method="none"), SUMS, False),
    ("Adakaon", "f32", dict(momentum_dtype="4bit", weight_decay=0.1), SUMS, False),
    ("Nekaon", "bf16", dict(), SUMS, False),
    ("Nekaon", "f32", dict(momentum_dtype="int8"), SUMS, False),
    ("AdaPNM", "bf16", dict(momentum_dtype="4bit"), SUMS, False),
    ("AdaPNM", "bf16", dict(momentum_dtype="int8"), SUMS, False),
    ("AdaPNM", "f32", dict(momentum_dtype="bfloat16"), SUMS, False),
    ("KProdigy", "bf16", dict(momentum_dtype="bfloat16"), SUMS, False),
    ("KProdigy", "bf16", dict(momentum_dtype="int8"), SUMS, False),
    ("KProdigy", "f32", dict(momentum_dtype="4bit", cautious=True), SUMS, False),
    ("AdaMuon", "bf16", dict(momentum_dtype="int8"), SUMS, False),
    ("AdaMuon", "f32", dict(momentum_dtype="4bit"), SUMS, False),
])
def test_unit_edges_vs_oracle(name, dtype, kw, how, big):
    import kaon_b200
    from _gpu import state_np, to_bits
    tdt = torch.bfloat16 if dtype == "bf16" else torch.float32
    shapes = EDGES + ([(16385, 4096)] if big else [])
    kw = dict(kw) if name == "KProdigy" else dict(kw, lr=1e-3)
    gen = torch.Generator().manual_seed(31)
    host = [(torch.randn(s, generator=gen) * 0.02).to(tdt) for s in shapes]
    params = [torch.nn.Parameter(h.clone().cuda()) for h in host]
    opt = getattr(kaon_b200, name)(params, **kw)
    opt.sr_seed = 5
    inner = getattr(opt, "base_optimizer", opt)
    orc = getattr(ko, "Oracle" + name)([to_bits(h) for h in host], shapes, seed=5, **kw)
    for step in range(2):
        grads = [(torch.randn(s, generator=gen) * 1e-3).to(tdt) for s in shapes]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        launched = opt.stats()["kernel_launches"] if step else 0
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        if name == "Lion":
            assert opt.stats()["kernel_launches"] - launched == (2 if big else 1)
        extra = {}
        if name == "AdaMuon":   # (the factor itself is bf16 matrix products; the chain around it is compared)
            extra["ns_override"] = [None if (o := opt.orthogonalised(p)) is None else o.float().cpu().numpy() for p in params]
        orc.step([to_bits(g) for g in grads], **extra)
        bad = total = bad_codes = codes = 0
        for i, p in enumerate(params):
            at = (step, shapes[i])
            for key, want in orc.tensors[i].state.items():
                got = state_np(inner.state[p], key)
                if not isinstance(want, np.ndarray) or got is None or want.size == 0:
                    continue
                got, want = got.reshape(-1), want.reshape(-1)
                if how == EXACT:
                    assert np.array_equal(got, want), (at, key)
                elif got.dtype.kind == "f":
                    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max(), (at, key)
                else:                                   # codes, packed codes, bf16 bits
                    diff = np.nonzero(got != want)[0]
                    bad_codes += diff.size
                    codes += got.size
                    for x, y in zip(got[diff].tolist(), want[diff].tolist()):
                        if got.dtype == np.uint8:       # (two 4-bit codes)
                            assert max(abs((x & 15) - (y & 15)), abs((x >> 4) - (y >> 4))) == 1, (at, key)
                        else:
                            assert abs(x - y) == 1, (at, key)
            got, want = to_bits(p), orc.tensors[i].p.reshape(-1)
            if how == EXACT:
                assert np.array_equal(got, want), at
            elif dtype == "bf16":
                diff = np.abs(got.astype(np.int32) - want.astype(np.int32))
                assert diff.max() <= 1, (at, diff.max())   # the other bf16 neighbour at most
                bad += int((diff != 0).sum())
            else:
                # an ulp of the weight, and what an ulp or two of a statistic moves the update by
                bad += int((np.abs(got - want) > 2.4e-7 * np.abs(want) + 1e-8).sum())
            total += got.size
        assert bad <= 1e-3 * total, (step, bad, total)
        assert bad_codes <= 2 + 1e-4 * codes, (step, bad_codes, codes)
