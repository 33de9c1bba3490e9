"""Models and core weights as Python objects: copies, pickles.  The weights lie on the CPU, nothing is launched."""
import copy
import dataclasses
import pickle

import pytest
import torch

import vmamba_b200 as vb
from tests.test_gpu_caller_state import state_dict
from vmamba_b200.backbone import AcceleratedVSSM


@pytest.fixture()
def model():
    m = vb.VSSMInfer.from_state_dict(state_dict(depths=(1, 1, 2, 1)), device="cpu")
    assert m.native is m.native and m.blocks[0][0].core.native is not None       # as after a first call
    return m


@pytest.mark.parametrize("again", [copy.copy, copy.deepcopy, lambda o: pickle.loads(pickle.dumps(o))], ids=["copy", "deepcopy", "pickle"])
def test_models_can_be_copied_after_their_first_call(model, again):
    for m in (again(model), again(AcceleratedVSSM(model, False, ())).fast):
        assert torch.equal(m.stem["w0"], model.stem["w0"]) and torch.equal(m.blocks[2][0].core.wx, model.blocks[2][0].core.wx)
        assert m.native is not None
    w = again(model.blocks[0][0].core)
    assert torch.equal(w.A, model.blocks[0][0].core.A) and w.native is not model.blocks[0][0].core.native


def test_core_weights_are_a_plain_dataclass(model):
    w = model.blocks[0][0].core
    names = [f.name for f in dataclasses.fields(w)]
    assert names[0] == "wx" and names[-1] == "eps" and set(dataclasses.asdict(w)) == set(names)
    assert dataclasses.replace(w, eps=1e-6).native is not w.native


def _replace_head(m):
    m.head["b"] = torch.ones_like(m.head["b"])


def _replace_core_field(m):
    m.blocks[1][0].core.Ds = m.blocks[1][0].core.Ds * 2


def _drop_a_block(m):
    m.blocks[2] = m.blocks[2][:-1]


CHANGES = {
    "stem": lambda m: m.stem.update(b0=m.stem["b0"] + 1),
    "block": lambda m: setattr(m.blocks[0][0], "w_in", m.blocks[0][0].w_in * 2),
    "core": _replace_core_field,
    "eps": lambda m: setattr(m.blocks[0][0].core, "eps", 1e-3),
    "blocks": _drop_a_block,
    "down": lambda m: m.down[0].update(bf=m.down[0]["bf"] + 1),
    "outnorm": lambda m: m.outnorm.update({2: (m.outnorm[2][0] * 2, m.outnorm[2][1])}),
    "head": _replace_head,
    "no head": lambda m: setattr(m, "head", None),
}


@pytest.mark.parametrize("what", CHANGES)
def test_changes_after_the_first_call_count(model, what):
    before = model.native
    CHANGES[what](model)
    after = model.native
    assert after is not before and after is model.native
    assert after.dtype == model.dtype and len(after.head) == (0 if model.head is None else 4)
    if model.head is not None:
        assert torch.equal(after.head[3], model.head["b"])


WRONG = {
    "type": lambda m: setattr(m, "dtype", torch.float16),
    "depthwise kernel": lambda m: setattr(m.blocks[0][0], "w_dw", torch.zeros(32, 1, 5, 5, dtype=m.dtype)),
    "norm": lambda m: setattr(m.blocks[1][0], "n2w", m.blocks[1][0].n2w[:8]),
    "out_proj": lambda m: setattr(m.blocks[0][0], "w_out", m.blocks[0][0].w_out[:16]),
    "layout": lambda m: setattr(m.blocks[0][0], "w_in", m.blocks[0][0].w_in.t()),
    "bias type": lambda m: setattr(m.blocks[0][0], "b1f", m.blocks[0][0].b1f.bfloat16()),
    "core": lambda m: setattr(m.blocks[0][0], "core", m.blocks[1][0].core),
    "core field": lambda m: setattr(m.blocks[0][0].core, "Ds", m.blocks[0][0].core.Ds[:8]),
    "outnorm": lambda m: m.outnorm.update({0: m.outnorm[1]}),
    "head": lambda m: m.head.update(nw=m.head["nw"][:8]),
    "stem": lambda m: m.stem.update(w0=torch.zeros(16, 3, 4, 4, dtype=m.dtype)),
}


@pytest.mark.parametrize("what", WRONG)
def test_parts_that_do_not_fit_are_refused(model, what):
    WRONG[what](model)
    with pytest.raises(RuntimeError):
        model.native


def test_core_weight_changes_count(model):
    w = model.blocks[0][0].core
    before = w.native
    w.eps = 1e-3
    assert w.native is not before and w.native is w.native


def test_a_model_refuses_host_images(model):
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        model(torch.zeros(1, 3, 64, 64))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        model.features(torch.zeros(1, 3, 64, 64))
