"""What a step notices between steps of an unchanged group: a state dict or a tensor of the list that is not the one of the
step before, gradients that moved (their addresses go up under the plan's device).  On CPU tensors, with plans that only record what they are given."""
import contextlib
import ctypes as C

import pytest
import torch

from kaon_b200 import Adakaon, Lion, _engine
from kaon_b200 import _lib as L


class RecordingPlan(_engine.GroupPlan):
    """The host half of a plan: no library handle, no device memory."""
    guarded = 0        # depth of the device guard

    def __init__(self, kind, params, states, ids, momentum_dtype, m_key="m"):
        self.device = params[0].device
        self.params, self.states, self.n = params, states, len(params)
        self.momentum_dtype = momentum_dtype
        self.param_ptrs = [p.data_ptr() for p in params]
        self.handle = None
        self.uploads = 0
        self._param_arr, self.grad_arr = (C.c_int64 * self.n)(*self.param_ptrs), (C.c_int64 * self.n)()
        self._param_addr, self.grad_addr = C.addressof(self._param_arr), C.addressof(self.grad_arr)

    def _upload(self, stream):
        assert RecordingPlan.guarded > 0, "gradient pointers uploaded outside the plan's device"
        self.uploads += 1


@contextlib.contextmanager
def _guard(device):
    RecordingPlan.guarded += 1
    yield
    RecordingPlan.guarded -= 1


@pytest.fixture
def stepped(monkeypatch):
    """opt -> the (tensor, state dict) pairs of each of its launches so far."""
    monkeypatch.setattr(_engine, "GroupPlan", RecordingPlan)
    monkeypatch.setattr(L, "raw_stream", lambda index: 0)
    monkeypatch.setattr(L, "on_device", _guard)
    monkeypatch.setattr(torch.cuda, "device", _guard)
    log = []

    def launch(self, plan, group, step, stream):
        log.append([(p, st) for p, st, g in zip(plan.params, plan.states, plan.grad_arr) if g])

    monkeypatch.setattr(Lion, "_launch", launch)
    monkeypatch.setattr(Adakaon, "_launch", launch)
    return log


def _make(cls, n=4):
    ps = [torch.nn.Parameter(torch.randn(6, 8)) for _ in range(n)]
    for p in ps:
        p.grad = torch.randn(6, 8)
    return ps, cls(ps, lr=1e-3)


def _is_live(opt, launch):
    return all(st is opt.state[p] and st for p, st in launch)


@pytest.mark.parametrize("cls", [Lion, Adakaon])
@pytest.mark.parametrize("how", ["empty", "other", "cleared", "deleted"])
def test_a_replaced_state_is_the_one_that_is_stepped(stepped, cls, how):
    ps, opt = _make(cls)
    for _ in range(3):
        opt.step()
    old = dict(opt.state[ps[1]])
    if how == "empty":
        opt.state[ps[1]] = {}
    elif how == "other":
        opt.state[ps[1]] = {k: v.clone() if torch.is_tensor(v) else v for k, v in old.items()}
    elif how == "cleared":
        opt.state[ps[1]].clear()
    else:
        del opt.state[ps[1]]
    for _ in range(2):
        opt.step()
        assert [id(p) for p, _ in stepped[-1]] == [id(p) for p in ps] and _is_live(opt, stepped[-1])
        assert opt.state[ps[1]]["m"] is not old["m"]


@pytest.mark.parametrize("known", [False, True])
def test_a_replaced_list_entry_is_stepped(stepped, known):
    ps, opt = _make(Lion)
    q = torch.nn.Parameter(torch.randn(6, 8))
    q.grad = torch.randn(6, 8)
    opt.step()
    if known:     # a tensor that has state already: nothing is initialised
        opt.state[q] = {k: v.clone() for k, v in opt.state[ps[2]].items()}
        opt.step()
    opt.step()
    opt.param_groups[0]["params"][2] = q
    opt.step()
    assert [id(p) for p, _ in stepped[-1]] == [id(p) for p in (ps[0], ps[1], q, ps[3])]
    assert _is_live(opt, stepped[-1])


def test_an_unchanged_group_keeps_its_plan_and_uploads_moved_gradients_on_its_device(stepped):
    ps, opt = _make(Lion)
    opt.step()
    plan, = opt._plans.values()
    opt.step()
    assert plan.uploads == 1
    ps[0].grad = torch.randn(6, 8)
    opt.step()
    assert plan.uploads == 2 and list(opt._plans.values()) == [plan]
    late = torch.nn.Parameter(torch.randn(3, 8))     # no gradient yet: not stepped, no state
    opt.param_groups[0]["params"].append(late)
    opt.step()
    assert late not in opt.state and list(opt._plans.values()) == [plan]
    late.grad = torch.randn(3, 8)
    opt.step()
    assert len(stepped[-1]) == 5 and stepped[-1][-1][0] is late


def test_a_plan_whose_tensors_changed_dtype_is_given_up(stepped):
    ps, opt = _make(Lion)
    opt.step()
    for p in ps:
        p.grad = None
        p.data = p.data.bfloat16()
        p.grad = torch.randn(6, 8).bfloat16()
    opt.step()
    assert [key[2] for key in opt._plans] == [torch.bfloat16]


def test_a_plan_that_cannot_be_built_leaves_none_behind(stepped, monkeypatch):
    ps, opt = _make(Lion)
    opt.step()
    ps[0].data = ps[0].data.clone()

    class Refused(RecordingPlan):
        def __init__(self, *args):
            raise NotImplementedError("refused")

    monkeypatch.setattr(_engine, "GroupPlan", Refused)
    with pytest.raises(NotImplementedError):
        opt.step()
    assert not opt._plans
    monkeypatch.setattr(_engine, "GroupPlan", RecordingPlan)
    opt.step()
    assert len(stepped[-1]) == len(ps) and _is_live(opt, stepped[-1])
