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
    m = vb.VSSMInfer.from_state_dict(state_dict(), device="cpu")
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
