"""The native per-tensor pass of a step (csrc/host_ext.cpp) against what Python sees, on CPU tensors."""
import ctypes as C

import pytest
import torch

from kaon_b200 import _lib as L


def _list(n):
    ps = [torch.nn.Parameter(torch.randn(4, 6)) for _ in range(n)]
    for p in ps:
        p.grad = torch.randn(4, 6)
    was, grads = (C.c_int64 * n)(*[p.data_ptr() for p in ps]), (C.c_int64 * n)()
    return ps, [{"m": 1, "step": 3} for _ in ps], was, grads


def _scan(ps, st, was, grads):
    return L.host().scan(ps, st, C.addressof(was), C.addressof(grads))


@pytest.mark.parametrize("n", [1, 5])
def test_scan_follows_the_gradients(n):
    ps, st, was, grads = _list(n)
    assert _scan(ps, st, was, grads) == L.SCAN_ANY | L.SCAN_CHANGED
    assert list(grads) == [p.grad.data_ptr() for p in ps]
    assert _scan(ps, st, was, grads) == L.SCAN_ANY
    ps[-1].grad = None
    assert _scan(ps, st, was, grads) == (L.SCAN_CHANGED | (L.SCAN_ANY if n > 1 else 0))
    assert grads[n - 1] == 0
    L.host().bump(st, "step", C.addressof(grads))
    assert [s["step"] for s in st] == [4] * (n - 1) + [3]


@pytest.mark.parametrize("what", ["sparse", "strided", "dtype", "moved", "state", "subclass"])
def test_scan_leaves_the_unusual_to_python(what):
    ps, st, was, grads = _list(3)
    before = list(grads)
    if what == "sparse":
        ps[1].grad = ps[1].grad.to_sparse()
    elif what == "strided":
        ps[1].grad = torch.randn(6, 4).t()
    elif what == "dtype":
        ps[1].data = ps[1].data.bfloat16()
        was[1] = ps[1].data_ptr()
        ps[1].grad = None
        ps[1].grad = torch.randn(4, 6).bfloat16()
        ps[1].data = ps[1].data.float()
        was[1] = ps[1].data_ptr()
    elif what == "moved":
        ps[1].data = ps[1].data.clone()
    elif what == "state":
        st[1] = {}
    else:
        class P(torch.nn.Parameter):
            pass
        ps[1] = P(torch.randn(4, 6))
    assert _scan(ps, st, was, grads) == L.SCAN_UNUSUAL
    assert list(grads) == before          # nothing recorded: the Python path compares and uploads


@pytest.mark.parametrize("have,want", [((), 0), ((0,), 0), ((1, 0), 1), ((1, 1, 1), 2)])
def test_grads_present(have, want):
    ps = [torch.nn.Parameter(torch.zeros(2)) for _ in have]
    for p, h in zip(ps, have):
        p.grad = torch.zeros(2) if h else None
    assert L.host().grads_present(ps) == want


def test_a_module_compiled_for_another_torch_is_not_used(monkeypatch):
    """It reads tensor objects by torch's layout of them: built again by a build, refused by a step."""
    from kaon_b200 import _build
    assert not _build._host_stale() and L.host().abi == _build.host_abi()
    monkeypatch.setattr(torch, "__version__", "2.0.0")
    monkeypatch.setattr(L, "_host", None)
    assert _build._host_stale() and _build.needs_build()
    with pytest.raises(L.KaonError, match="build it again"):
        L.host()
